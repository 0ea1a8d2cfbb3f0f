"""Two host threads that run the same entry points on problems of different
size, each on its own stream: every call is launched and every result is the
one of a call alone.  (A kernel's shared-memory limit is shared by all threads
of the process.)"""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CALLS = 1500  # of each thread


def _sector(n_sites, d, rows=None):
    import torch

    from edgpu.symmetries import Sector

    dims = np.full(n_sites, d)
    sec = Sector(torch.arange(rows or d ** n_sites, dtype=torch.int64, device="cuda"), dims)
    sec.lookup_table()
    return sec


def _up(a, dtype):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a, dtype=dtype)).to("cuda")


def _diag(large):
    """edg_assemble_diag with few or many terms."""
    import torch

    from edgpu._lib import lib, ptr
    from edgpu.modeling.assembly import _assembly_struct

    sec, nd, rng = _sector(4, 4), 1500 if large else 1, np.random.default_rng(1)
    a = _assembly_struct(sec, 4, False)
    site, diag = rng.integers(0, 4, nd), rng.standard_normal((nd, 4))
    keep = [_up(site, np.int32), _up(diag, np.float64), _up(np.ones(nd), np.float64)]
    a.n_terms, a.n_dterms = 0, nd
    a.dterm_site, a.dterm_diag, a.dterm_coef = (ptr(t) for t in keep)
    out = torch.empty(len(sec), dtype=torch.float64, device="cuda")
    present = torch.empty(len(sec), dtype=torch.uint8, device="cuda")
    return (lambda st: lib.edg_assemble_diag(ctypes.byref(a), None, None, 0, 0.0, 0.0, ptr(out), ptr(present), st),
            out, (sec, keep, present))


def _count(large):
    """edg_assemble_count with few or many instances."""
    import torch

    from edgpu import _lib
    from edgpu._lib import lib, ptr
    from edgpu.modeling.assembly import _assembly_struct

    sec, nt = _sector(4, 4), 600 if large else 1
    a = _assembly_struct(sec, 4, False)
    sites = np.zeros((nt, _lib.MAX_OPS))
    sites[:, 0] = np.arange(nt) % 4
    keep = [_up(np.arange(4)[None, :] % 3, np.int32), _up(np.zeros((1, 4, 4)), np.uint8),
            _up(np.ones((1, 4, 4)), np.float64), _up(np.ones(nt), np.int32), _up(sites, np.int32),
            _up(np.zeros((nt, _lib.MAX_OPS)), np.int32), _up(np.ones(nt), np.float64)]
    a.n_terms, a.n_dterms = nt, 0
    a.t_count, a.t_ket, a.t_amp = (ptr(t) for t in keep[:3])
    a.term_nops, a.term_site, a.term_table, a.term_coef = (ptr(t) for t in keep[3:])
    out = torch.empty(len(sec), dtype=torch.int64, device="cuda")
    return lambda st: lib.edg_assemble_count(ctypes.byref(a), ptr(out), st), out, (sec, keep)


def _levels(large):
    """edg_sector_levels with room for few or many prefixes."""
    import torch

    from edgpu._lib import lib, ptr
    from edgpu.symmetries import SectorSpec, _DeviceTables, get_symmetry_sector_generators

    op = np.zeros((6, 4, 4))
    op[:, np.arange(4), np.arange(4)] = np.arange(4)
    gens = get_symmetry_sector_generators([op], "global")
    spec = SectorSpec(loc_dims=np.full(6, 4), glob_op_diags=gens, glob_sectors=[9], sym_type_flag="U")
    tables = _DeviceTables(spec, "cuda")
    cap = 1 << 22 if large else 4096
    keys = [torch.empty(cap, dtype=torch.int64, device="cuda") for _ in range(2)]
    sums = [torch.empty(cap, dtype=torch.int32, device="cuda") for _ in range(2)]
    work = torch.empty(int(lib.edg_sector_levels_work_elems()), dtype=torch.int64, device="cuda")
    return (lambda st: lib.edg_sector_levels(ctypes.byref(tables.struct), ptr(keys[0]), ptr(keys[1]), ptr(sums[0]),
                                             ptr(sums[1]), cap, ptr(work), st), work[:67], (tables, keys, sums, work))


def _twobody(large):
    """edg_twobody_expval of real diagonal operators with few or many states a
    site."""
    import torch

    from edgpu._lib import lib, ptr

    n_sites, dmax = 26, 32 if large else 2
    sec, rng = _sector(n_sites, 2, 70000), np.random.default_rng(3)
    count = np.ones((2, n_sites, dmax))
    ket = np.zeros((2, n_sites, dmax, dmax))
    ket[..., 0] = np.arange(dmax)
    amp = np.zeros((2, n_sites, dmax, dmax, 2))
    amp[:, :, :2, 0, 0] = rng.standard_normal((2, n_sites, 2))
    pairs = np.array([(i, j) for i in range(n_sites) for j in range(i + 1, n_sites)])
    keep = [_up(sec.strides, np.int64), _up(sec.loc_dims, np.int32), _up(count, np.int32), _up(ket, np.uint8),
            _up(amp, np.float64), _up(pairs[:, 0], np.int32), _up(pairs[:, 1], np.int32),
            _up(rng.standard_normal(len(sec)), np.float64)]
    ns = lib.edg_twobody_scratch_elems(len(pairs))
    scratch = torch.empty(ns, dtype=torch.float64, device="cuda")
    out = torch.empty((n_sites, n_sites), dtype=torch.float64, device="cuda")
    p = [ptr(t) for t in keep]
    return (lambda st: lib.edg_twobody_expval(sec.lookup_table(), p[0], p[1], n_sites, p[2], p[3], p[4], dmax, p[5],
                                              p[6], len(pairs), p[7], 0, 1, ptr(out), ptr(scratch), ns, st),
            out, (sec, keep, scratch))


def _orth(large):
    """edg_krylov_orth against enough vectors for its coefficients to need
    more than the default shared memory."""
    import torch

    from edgpu._lib import lib, ptr

    n, m = 64, 4500 if large else 2700
    basis = torch.zeros((m + 1, n), dtype=torch.complex128, device="cuda")
    w = torch.ones(n, dtype=torch.complex128, device="cuda")
    coef = torch.ones((2, m + 1), dtype=torch.float64, device="cuda")
    wb = lib.edg_krylov_orth_bytes(m)
    work = torch.zeros(wb, dtype=torch.uint8, device="cuda")
    # against zero vectors w comes back as it is
    return (lambda st: lib.edg_krylov_orth(n, n, ptr(basis), m - 1, ptr(w), 1, ptr(coef[0]), ptr(coef[1]), m,
                                           ptr(work), wb, st), basis[m], (basis, w, coef, work))


@pytest.mark.parametrize("make", [_diag, _count, _levels, _twobody, _orth])
def test_calls_of_two_threads(make):
    import torch

    jobs = [make(False), make(True)]
    want = []
    for call, out, _ in jobs:
        assert call(None) == 0
        torch.cuda.synchronize()
        want.append(out.clone())
    start = threading.Barrier(2)
    refused = [0, 0]

    def run(i):
        call, st = jobs[i][0], torch.cuda.Stream()
        start.wait()
        for _ in range(CALLS):
            refused[i] += call(st.cuda_stream) != 0
        st.synchronize()

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert refused == [0, 0]
    for (_, out, _), w in zip(jobs, want):
        assert torch.equal(out, w)
