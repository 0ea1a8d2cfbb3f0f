"""One Krylov step exp(-i H dt) psi on synthetic Hermitian matrices against a
Taylor series of the same operator in complex128: the cooperative one-launch
form and the pass-by-pass form on both sides of their line, every
reorthogonalisation choice, matrices without off-diagonal entries (breakdown
after one vector), one row, and the largest Krylov dimension."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, cplx, seed, empty=False):
    import torch

    from edgpu.modeling.assembly import DeviceMatrix

    rng = np.random.default_rng(seed)
    if n > 1 and not empty:
        r = np.repeat(np.arange(n), 4)
        c = rng.integers(0, n, 4 * n)
        v = rng.choice([0.5, -0.25, 1.0], 4 * n).astype(np.complex128)
        if cplx:
            v = v * rng.choice([1, 1j, -1j], 4 * n)
        keep = r < c
        keys, first = np.unique(r[keep] * n + c[keep], return_index=True)
        r, c, v = keys // n, keys % n, v[keep][first]
        r, c, v = np.concatenate([r, c]), np.concatenate([c, r]), np.concatenate([v, v.conj()])
        order = np.lexsort((c, r))
        r, c, v = r[order], c[order], v[order]
    else:
        r = c = np.zeros(0, dtype=np.int64)
        v = np.zeros(0, dtype=np.complex128)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int64)
    d = rng.uniform(-2, 2, n)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    vals = up(v.view(np.float64) if cplx else v.real)
    diag = up(d.astype(np.complex128).view(np.float64) if cplx else d)
    mat = DeviceMatrix(n, up(rowptr), up(c.astype(np.int32)), vals, diag, None, cplx)
    a = torch.sparse_csr_tensor(mat.rowptr, up(c.astype(np.int64)), up(v), size=(n, n))
    return mat, (lambda x: (a @ x[:, None])[:, 0] + up(d) * x)


COOP_MAX = 1024 * 148  # rows of the one-launch form


@pytest.mark.parametrize("n,m", [(1, 30), (2, 30), (33, 30), (700, 1), (700, 64), (5000, 30), (COOP_MAX, 20),
                                 (COOP_MAX + 1, 20)])
@pytest.mark.parametrize("precision,reorth", [("c128", 0), ("c128", 1), ("c128", 2), ("c64", 0), ("c64", 1)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("empty", [False, True])
def test_step_matches_taylor(n, m, precision, reorth, cplx, empty):
    import torch

    from edgpu.dynamics import KrylovEvolver

    if empty and n > 700:
        pytest.skip("the breakdown does not depend on the size")
    mat, apply = _matrix(n, cplx, 3 * n + cplx, empty)
    ev = KrylovEvolver(mat, m=m, precision=precision, reorth_passes=reorth, matvec="auto" if n % 2 else "csr")
    gen = torch.Generator(device="cuda").manual_seed(n)
    psi = torch.randn(n, dtype=torch.complex128, device="cuda", generator=gen) * 3.0
    # one vector spans the state only to first order in dt: a short step
    dt = 1e-7 if m == 1 else 0.1
    want, term = psi.clone(), psi
    for k in range(1, 40):
        term = apply(term) * (-1j * dt / k)
        want = want + term
    got = psi.to(ev.vdtype).clone()
    ev.step(got, dt)
    ev.check_status()
    err = float(torch.linalg.vector_norm(got.to(torch.complex128) - want) / torch.linalg.vector_norm(want))
    # c64: a rounding of 2^-24 per stored entry of each basis vector and of psi
    tol = 5e-6 if precision == "c64" else (1e-5 if m == 1 else 1e-12)
    assert err < tol, err


@pytest.mark.parametrize("n", [33, 700, 5000, COOP_MAX, COOP_MAX + 1])
@pytest.mark.parametrize("precision,reorth", [("c128", 0), ("c128", 1), ("c64", 0), ("c64", 2)])
def test_step_on_a_packed_layout_alone(n, precision, reorth):
    """A problem without CSR arrays takes the packed product at every size."""
    import torch

    from edgpu._lib import ptr
    from edgpu.dynamics import KrylovEvolver
    from edgpu.solvers import PackedLayout

    mat, apply = _matrix(n, False, n)
    pk = PackedLayout.build(mat)
    ev = KrylovEvolver(mat, m=30, precision=precision, reorth_passes=reorth, matvec="csr")
    p = ev.p
    p.pk_tile_off, p.pk_words, p.pk_count, p.pk_colbits = ptr(pk.tile_off), ptr(pk.words), pk.count, pk.colbits
    p.pk_table = ptr(pk.table(0 if precision == "c128" else 1))
    p.cols = p.vals = None
    gen = torch.Generator(device="cuda").manual_seed(n)
    psi = torch.randn(n, dtype=torch.complex128, device="cuda", generator=gen)
    dt = 0.1
    want, term = psi.clone(), psi
    for k in range(1, 40):
        term = apply(term) * (-1j * dt / k)
        want = want + term
    got = psi.to(ev.vdtype).clone()
    ev.step(got, dt)
    ev.check_status()
    err = float(torch.linalg.vector_norm(got.to(torch.complex128) - want) / torch.linalg.vector_norm(want))
    assert err < (5e-6 if precision == "c64" else 1e-12), err


@pytest.mark.parametrize("n", [33, 5000])
@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("status,want_error", [(True, True), (False, True), (False, False)])
def test_step_with_and_without_a_status_word(n, precision, status, want_error):
    """The same step reports to a status word, through the error estimate's
    return, or has neither and takes the passes."""
    import torch

    from edgpu.dynamics import KrylovEvolver

    mat, apply = _matrix(n, False, n)
    gen = torch.Generator(device="cuda").manual_seed(n)
    psi = torch.randn(n, dtype=torch.complex128, device="cuda", generator=gen)
    want, term = psi.clone(), psi
    for k in range(1, 40):
        term = apply(term) * (-0.1j / k)
        want = want + term
    ev = KrylovEvolver(mat, m=30, precision=precision, matvec="csr")
    if not status:
        ev.p.status = None
    got = psi.to(ev.vdtype).clone()
    e = ev.step(got, 0.1, want_error=want_error)
    ev.check_status()
    assert e is None or 0.0 <= e < 1e-10
    err = float(torch.linalg.vector_norm(got.to(torch.complex128) - want) / torch.linalg.vector_norm(want))
    assert err < (5e-6 if precision == "c64" else 1e-12), err


@pytest.mark.parametrize("per_row", [60, 80])
@pytest.mark.parametrize("precision", ["c128", "c64"])
def test_both_sides_of_the_line_on_the_entries(per_row, precision):
    """At 700 rows a step of up to 162,000 entries is one launch."""
    import ctypes

    import torch

    from edgpu._lib import lib
    from edgpu.dynamics import KrylovEvolver
    from edgpu.modeling.assembly import DeviceMatrix

    n, rng = 700, np.random.default_rng(per_row)
    h = np.triu(np.where(rng.random((n, n)) < 3.6 * per_row / n, rng.choice([0.5, -0.25, 0.125], (n, n)), 0.0), 1)
    h = h + h.T
    r, c = np.nonzero(h)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d = rng.uniform(-2, 2, n)
    mat = DeviceMatrix(n, up(np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))])), up(c.astype(np.int32)),
                       up(h[r, c]), up(d), None, False)
    ev = KrylovEvolver(mat, m=60, precision=precision, matvec="csr")
    assert lib.edg_krylov_one_launch(ctypes.byref(ev.p)) == (len(r) <= 6 * 27000) == (per_row == 60)
    psi = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    e, u = np.linalg.eigh(h + np.diag(d))
    dt = 10.0 / np.abs(e).max()
    want = u @ (np.exp(-1j * dt * e) * (u.T @ psi))
    got = up(psi).to(ev.vdtype)
    ev.step(got, dt)
    ev.check_status()
    err = np.linalg.norm(got.cpu().numpy() - want) / np.linalg.norm(want)
    assert err < (5e-6 if precision == "c64" else 1e-12), err
