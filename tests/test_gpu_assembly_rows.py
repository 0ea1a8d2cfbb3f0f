"""Assembly of random operator products on random sectors against triplets
summed on the host: duplicates and entries on the diagonal (the rows that
need the compaction), rows longer than a warp's windows, one to four factors,
more than 32 and more than 1,000 instances, complex values, one- and two-word
keys, and the diagonal with its constant."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_free,d,density,nops,instances", [
    (1, 3, 1.0, 1, 1), (5, 3, 0.4, 2, 7), (5, 3, 0.5, 3, 33), (4, 4, 0.9, 2, 40), (3, 6, 1.0, 3, 6), (4, 3, 1.0, 4, 3),
    (5, 3, 0.3, 2, 1100)])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("wide", [False, True])
def test_random_products(n_free, d, density, nops, instances, cplx, wide):
    import torch

    from edgpu.modeling.assembly import assemble_blocks
    from edgpu.modeling.terms import TermBlock
    from edgpu.symmetries import Sector

    rng = np.random.default_rng(97 * n_free + 13 * d + instances)
    n_frozen = 42 if wide else 0  # frozen sites push the key space past 63 bits
    dims = np.array([3] * n_frozen + [d] * n_free)
    ns = len(dims)
    dmax = int(dims.max())
    free = np.stack(np.unravel_index(np.arange(d ** n_free), (d,) * n_free), axis=1)
    cfg = np.concatenate([np.ones((len(free), n_frozen), dtype=free.dtype), free], axis=1)
    probe = Sector(torch.zeros((1, 2) if wide else 1, dtype=torch.int64, device="cuda"), dims)
    sec = Sector(probe.encode(cfg), dims)
    n = len(cfg)
    blocks, dense = [], np.zeros((n, n), dtype=np.complex128)
    index = {tuple(c): i for i, c in enumerate(free)}
    for _ in range(instances):
        sites = rng.permutation(n_free)[:nops]
        ops = []
        for s in sites:
            m = np.where(rng.random((d, d)) < density, rng.integers(1, 4, (d, d)), 0).astype(np.complex128)
            if cplx:
                m = m * np.exp(1j * rng.uniform(0, 6, (d, d)))
            ops.append(m)
        full = []
        for m in ops:
            op = np.zeros((ns, dmax, dmax), dtype=np.complex128)
            op[:, :d, :d] = m
            full.append(op)
        blocks.append(TermBlock(ops=full, sites=np.array([[n_frozen + s for s in sites]]), strength=0.5,
                                diagonal=False, add_dagger=False))
        for i, c in enumerate(free):
            stack = [(0.5 + 0j, list(c))]
            for s, m in zip(sites, ops):
                stack = [(v * m[k[s], t], k[:s] + [t] + k[s + 1:]) for v, k in stack for t in range(d) if m[k[s], t]]
            for v, k in stack:
                dense[i, index[tuple(k)]] += v
    dop = np.zeros((ns, dmax, dmax), dtype=np.complex128)
    dop[n_frozen:, np.arange(d), np.arange(d)] = rng.standard_normal((n_free, d))
    blocks.append(TermBlock(ops=[dop], sites=np.array([[n_frozen + s] for s in range(n_free)]), strength=2.0,
                            diagonal=True, add_dagger=False))
    mat = assemble_blocks(sec, blocks, force_complex=cplx, extra_diag=0.25)
    got = mat.to_scipy().toarray()
    for i, c in enumerate(free):
        dense[i, i] += 0.25 + 2.0 * sum(np.real(dop[n_frozen + s, c[s], c[s]]) for s in range(n_free))
    cols, rp = mat.cols.cpu().numpy(), mat.rowptr.cpu().numpy()
    for r in range(n):
        w = cols[rp[r]:rp[r + 1]]
        assert np.all(np.diff(w) > 0) and r not in w
    # a column is stored when any product reaches it, even where they cancel
    scale = max(1.0, float(np.abs(dense).max()))
    assert np.max(np.abs(got - dense)) < 1e-13 * scale * max(1, instances)
