"""Diagonal observables on random sectors (sorted random keys, mixed local
dimensions): local expectation values and two-body correlators against sums
over the decoded configurations, across the site counts where the register
and tensor-block sizes change, ragged row counts and every state type."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sector(n_sites, n, seed, d_hi=4):
    import torch

    from edgpu.symmetries import Sector

    rng = np.random.default_rng(seed)
    dims = rng.integers(2, d_hi + 1, n_sites)
    cfg = np.unique(rng.integers(0, dims, (n, n_sites)), axis=0)  # lexicographic = key order
    sec = Sector(torch.zeros((1, 2) if np.log2(dims.astype(float)).sum() >= 63 else 1, dtype=torch.int64,
                             device="cuda"), dims)
    return Sector(sec.encode(cfg), dims), cfg, dims, rng


def _state(n, dtype, rng):
    import torch

    x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if "complex" in dtype else 0)
    psi = torch.from_numpy(x / np.linalg.norm(x)).to(getattr(torch, dtype)).cuda()
    return psi, np.abs(psi.cpu().numpy().astype(np.complex128)) ** 2


def _operator(n_sites, dims, rng):
    op = np.zeros((n_sites, int(dims.max()), int(dims.max())), dtype=np.complex128)
    for s in range(n_sites):
        op[s, np.arange(dims[s]), np.arange(dims[s])] = rng.standard_normal(dims[s])
    return op


@pytest.mark.parametrize("n_sites", [1, 2, 15, 16, 17, 32, 33, 45])
@pytest.mark.parametrize("n", [1, 255, 5000])
@pytest.mark.parametrize("dtype", ["float64", "float32", "complex128", "complex64"])
def test_local_expectation_values(n_sites, n, dtype):
    from edgpu.models.quantum_model import site_expval_device

    sec, cfg, dims, rng = _sector(n_sites, n, 100 * n_sites + n)
    op = _operator(n_sites, dims, rng)
    psi, p = _state(len(cfg), dtype, rng)
    got = site_expval_device(sec, op, psi).cpu().numpy()
    ref = [np.sum(p * np.real(op[s, cfg[:, s], cfg[:, s]])) for s in range(n_sites)]
    assert np.max(np.abs(got - ref)) < 1e-12


@pytest.mark.parametrize("n_sites", [2, 7, 8, 9, 16, 17, 24, 25, 32, 33])
@pytest.mark.parametrize("n", [1, 31, 33, 5000])
@pytest.mark.parametrize("dtype", ["float64", "complex64"])
@pytest.mark.parametrize("subset", [False, True])
def test_two_body_correlators(n_sites, n, dtype, subset):
    from edgpu.models.quantum_model import twobody_corr_device

    sec, cfg, dims, rng = _sector(n_sites, n, 200 * n_sites + n, d_hi=3)
    a, b = _operator(n_sites, dims, rng), _operator(n_sites, dims, rng)
    psi, p = _state(len(cfg), dtype, rng)
    pairs = [(0, n_sites - 1), (n_sites - 1, n_sites // 2)] if subset and n_sites > 2 else None
    got = twobody_corr_device(sec, a, b, psi, pairs).cpu().numpy()
    va = np.stack([np.real(a[s, cfg[:, s], cfg[:, s]]) for s in range(n_sites)])
    vb = np.stack([np.real(b[s, cfg[:, s], cfg[:, s]]) for s in range(n_sites)])
    full = (va * p) @ vb.T
    ref = np.zeros((n_sites, n_sites))
    for i, j in pairs or [(i, j) for i in range(n_sites) for j in range(i + 1, n_sites)]:
        ref[i, j] = ref[j, i] = full[i, j]
    assert np.max(np.abs(got - ref)) < 1e-12


@pytest.mark.parametrize("n_sites", [16, 17, 24, 25, 32, 33])
@pytest.mark.parametrize("n", [65535, 65536, 70001])
@pytest.mark.parametrize("dtype", ["float64", "float32", "complex128", "complex64"])
def test_two_body_correlators_on_both_sides_of_the_row_line(n_sites, n, dtype):
    """Sectors just below and above the rows from which real diagonal operators
    go to the tensor instruction, with a pair listed either way round."""
    from edgpu.models.quantum_model import twobody_corr_device
    from edgpu.symmetries import Sector

    sec, cfg, dims, rng = _sector(n_sites, 100000, 300 * n_sites, d_hi=3)
    assert len(cfg) >= n
    sec, cfg = Sector(sec.keys[:n].clone(), dims), cfg[:n]
    a, b = _operator(n_sites, dims, rng), _operator(n_sites, dims, rng)
    psi, p = _state(n, dtype, rng)
    pairs = [(i, j) for i in range(n_sites) for j in range(i + 1, n_sites) if (i, j) != (1, n_sites - 1)]
    pairs.append((n_sites - 1, 1))
    got = twobody_corr_device(sec, a, b, psi, pairs).cpu().numpy()
    va = np.stack([np.real(a[s, cfg[:, s], cfg[:, s]]) for s in range(n_sites)])
    vb = np.stack([np.real(b[s, cfg[:, s], cfg[:, s]]) for s in range(n_sites)])
    full = (va * p) @ vb.T
    ref = np.zeros((n_sites, n_sites))
    for i, j in pairs:
        ref[i, j] = ref[j, i] = full[i, j]
    assert np.max(np.abs(got - ref)) < 1e-12
