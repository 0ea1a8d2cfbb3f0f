"""Gauge phases of the real form on the device (``edg_gauge_apply``) against
the exponents summed on the host over the decoded configurations."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one-word keys inside and past 32 bits, more than 16 sites, two-word keys
SECTORS = {
    "su2_L8": ("su2", dict(spin=0.5, pure_theory=False, lvals=[8], has_obc=[True], sectors=[8])),
    "su2_L14": ("su2", dict(spin=0.5, pure_theory=False, lvals=[14], has_obc=[True], sectors=[14])),
    "qed_L18": ("qed", dict(spin=1, pure_theory=False, lvals=[18], has_obc=[True])),
    "qed_4x4_wide": ("qed", dict(spin=1, pure_theory=True, lvals=[4, 4], has_obc=[False, False])),
}


def _sector(name):
    from edgpu.models import QED_Model, SU2_Model

    kind, kw = SECTORS[name]
    return (SU2_Model if kind == "su2" else QED_Model)(**kw, device="cuda")


@pytest.mark.parametrize("name", list(SECTORS))
@pytest.mark.parametrize("dtype,stride", [(None, 1), ("float64", 1), ("float32", 3), ("complex128", 2),
                                          ("complex64", 1)])
def test_phases_match_decoded_configurations(name, dtype, stride):
    import torch

    from edgpu import _lib
    from edgpu._lib import check, lib, ptr, stream_handle

    sec = _sector(name).sector
    n, ns = len(sec), sec.n_sites
    dmax = int(sec.loc_dims.max())
    rng = np.random.default_rng(3)
    w = rng.integers(0, 4, (ns, dmax)).astype(np.uint8)
    e = w[np.arange(ns)[None, :], sec.configs].astype(np.int64).sum(axis=1) % 4
    phase = np.array([1, 1j, -1, -1j])[e]
    dims = _lib.SiteDims()
    for s in range(ns):
        dims.d[s] = int(sec.loc_dims[s])
    psi, want = None, phase
    if dtype is not None:
        h = rng.standard_normal((n, stride)) + (1j * rng.standard_normal((n, stride)) if "complex" in dtype else 0)
        psi = torch.from_numpy(h).to(getattr(torch, dtype)).cuda()
        want = psi[:, 0].to(torch.complex128).cpu().numpy()
    codes = {None: 0, "float64": 0, "float32": 1, "complex128": 2, "complex64": 3}
    wt = torch.from_numpy(w).cuda()
    for conj in (0, 1):
        out = torch.empty(n, dtype=torch.complex128, device="cuda")
        check(lib.edg_gauge_apply(ptr(sec.keys), n, sec.key_words, sec.n_hi, ctypes.byref(dims), ns, ptr(wt), dmax,
                                  conj, ptr(psi), codes[dtype], stride, ptr(out), stream_handle()))
        ph = np.conj(phase) if conj else phase
        ref = ph if psi is None else ph * want
        assert np.array_equal(out.cpu().numpy(), ref)  # a swap and a sign: exact


@pytest.mark.parametrize("shape", ["vector", "column", "stack", "host_dtype"])
def test_basis_maps_agree_with_the_phases(shape):
    """to/from_original_basis equal the product with the phases for every
    form of operand they take."""
    import torch

    model = _sector("su2_L8")
    model.build_Hamiltonian(1.0, 0.5)
    n = len(model.sector)
    ph = model.H._row_phase()
    assert ph is not None
    gen = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen)
    psi = {"vector": x[:, 0].contiguous(), "column": x[:, 1], "stack": x.T.contiguous(),
           "host_dtype": (x[:, 2] * 4).to(torch.int32)}[shape]
    assert torch.equal(model.H.to_original_basis(psi), ph * psi.to(torch.complex128))
    assert torch.equal(model.H.from_original_basis(psi), torch.conj(ph) * psi.to(torch.complex128))
