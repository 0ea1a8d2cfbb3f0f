"""One-launch Lanczos of a single small problem on synthetic symmetric
matrices: sizes around one, two and the most rows of a CTA, the line to the
pass-by-pass solver, one row, exhausted Krylov spaces (more than 256
tridiagonal rows), start vectors, several eigenpairs, f32 with a window;
against a dense solve, or the residual where the matrix is too large."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COOP_MAX = 1024 * 148  # rows of the one-launch form


def _matrix(n, seed, per_row=4):
    import torch

    rng = np.random.default_rng(seed)
    r, c = np.repeat(np.arange(n), per_row), rng.integers(0, n, per_row * n)
    keep = r < c
    keys, first = np.unique(r[keep] * n + c[keep], return_index=True)
    v = rng.choice([0.5, -0.25, 1.0], per_row * n)[keep][first]
    r, c = keys // n, keys % n
    r, c, v = np.concatenate([r, c]), np.concatenate([c, r]), np.concatenate([v, v])
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order], v[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int64)
    # a low level well below the rest: quick convergence at any size
    d = rng.uniform(0, 4, n)
    d[rng.integers(0, n, 3)] -= np.array([12.0, 9.0, 6.0])
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return up(rowptr), up(c.astype(np.int32)), up(v), up(d), (r, c, v, d)


def _solve(n, arrays, dtype, **kw):
    import torch

    from edgpu.solvers import run_lanczos

    rowptr, cols, vals, diag = arrays[:4]
    t = torch.float32 if dtype else torch.float64
    return run_lanczos(dtype, n, int(cols.numel()), rowptr, cols, vals.to(t), diag.to(t)[:, None].contiguous(),
                       **kw)


@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 511, 3000])
@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("v0", [False, True])
def test_eigenpairs_match_a_dense_solve(n, k, v0):
    import torch

    if k > n:
        pytest.skip("fewer rows than eigenpairs")
    arrays = _matrix(n, n)
    r, c, v, d = arrays[4]
    h = np.diag(d)
    h[r, c] += v
    e, x = np.linalg.eigh(h)
    start = None
    if v0:
        start = torch.from_numpy(np.random.default_rng(1).standard_normal((n, 1))).cuda()
    got = _solve(n, arrays, 0, k=k, max_iter=300, tol=1e-12, v0=start)
    assert np.max(np.abs(got.evals[0] - e[:k])) < 1e-12 * max(1.0, np.abs(e).max())
    vec = got.evecs[:, :, 0].cpu().numpy()
    for q in range(k):
        assert abs(np.linalg.norm(vec[q]) - 1) < 1e-13
        assert np.linalg.norm(h @ vec[q] - e[q] * vec[q]) < 1e-10


def test_exhausted_krylov_space():
    """tol that is never met: the space is exhausted at 300 rows and every
    Ritz value of it is exact."""
    n = 300
    arrays = _matrix(n, 7)
    r, c, v, d = arrays[4]
    h = np.diag(d)
    h[r, c] += v
    got = _solve(n, arrays, 0, k=4, max_iter=n, tol=1e-300, allow_unconverged=True)
    assert np.max(np.abs(got.evals[0] - np.linalg.eigvalsh(h)[:4])) < 1e-11


@pytest.mark.parametrize("n", [257, 40000, COOP_MAX - 3, COOP_MAX, COOP_MAX + 1])
@pytest.mark.parametrize("dtype,window", [(0, 0), (1, 0), (1, 4)])
def test_residuals_on_both_sides_of_the_line(n, dtype, window):
    import torch

    arrays = _matrix(n, n)
    rowptr, cols, vals, diag = arrays[:4]
    got = _solve(n, arrays, dtype, k=1, max_iter=200, tol=1e-5 if dtype else 1e-11, window=window)
    x = got.evecs[0, :, 0].double()
    a = torch.sparse_csr_tensor(rowptr, cols.to(torch.int64), vals, size=(n, n))
    res = (a @ x[:, None])[:, 0] + diag * x - float(got.evals[0, 0]) * x
    # f32: the vector's own rounding (2^-24) times |H| beside the tolerance
    assert float(torch.linalg.vector_norm(res)) < (1e-4 if dtype else 1e-9)
    assert abs(float(torch.linalg.vector_norm(x)) - 1) < (1e-6 if dtype else 1e-13)


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("kept", ["none", "vals", "cols"])
def test_packed_layout_alone(dtype, kept):
    """A single problem whose CSR arrays are not all given takes the packed
    product below the one-launch form's line too."""
    import torch

    from edgpu.modeling.assembly import DeviceMatrix
    from edgpu.solvers import PackedLayout, run_lanczos

    n = 3000
    rowptr, cols, vals, diag, (r, c, v, d) = _matrix(n, n)
    pk = PackedLayout.build(DeviceMatrix(n, rowptr, cols, vals, diag, None, False))
    t = torch.float32 if dtype else torch.float64
    got = run_lanczos(dtype, n, int(cols.numel()), rowptr, cols if kept == "cols" else None,
                      vals.to(t) if kept == "vals" else None, diag.to(t)[:, None].contiguous(), packed=pk,
                      max_iter=300, tol=1e-5 if dtype else 1e-12)
    h = np.diag(d)
    h[r, c] += v
    e = np.linalg.eigvalsh(h)
    # f32: the error is quadratic in the residual bound, beside the rounding
    # (2^-24) of the vectors times |H|
    assert abs(got.evals[0, 0] - e[0]) < (2e-6 if dtype else 1e-12) * np.abs(e).max()
