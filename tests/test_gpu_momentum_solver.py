"""Kernels of the momentum-sector solver against dense complex128 algebra."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 31, 257, 40000])
@pytest.mark.parametrize("steps", [1, 9, 33])
def test_orth_steps(n, steps):
    """Bases and coefficients of a run on a diagonal operator: v_i orthonormal,
    <v_i, H v_j> tridiagonal with the returned alpha and beta.  n terms of
    relative error 2^-53 each in two-pass Gram-Schmidt leave both below 1e-12."""
    from edgpu._lib import check, lib, ptr, stream_handle

    steps = min(steps, n)
    rng = np.random.default_rng(n + steps)
    h = torch.from_numpy(rng.uniform(-1, 1, n)).cuda()
    q = torch.from_numpy(rng.normal(size=n) + 1j * rng.normal(size=n)).cuda()
    V = torch.empty((steps + 1, n), dtype=torch.complex128, device="cuda")
    V[0] = q / torch.linalg.vector_norm(q)
    coef = torch.zeros((2, steps + 1), dtype=torch.float64, device="cuda")
    coef[1, 0] = 1.0
    wb = lib.edg_krylov_orth_bytes(steps)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    for j in range(steps):
        w = h * V[j]
        check(lib.edg_krylov_orth(n, n, ptr(V), j, ptr(w), 2, ptr(coef[0]), ptr(coef[1]), steps, ptr(work), wb,
                                  stream_handle()), "edg_krylov_orth")
    alpha, beta = coef.cpu().numpy()
    v = V[:steps].cpu().numpy() / beta[:steps, None]
    assert np.max(np.abs(v.conj() @ v.T - np.eye(steps))) <= 1e-12
    t = v.conj() @ (h.cpu().numpy()[:, None] * v.T)
    ref = np.diag(alpha[:steps]) + np.diag(beta[1:steps], 1) + np.diag(beta[1:steps], -1)
    assert np.max(np.abs(t - ref)) <= 1e-12


@pytest.mark.parametrize("ucs,k", [([1], [0]), ([1], [3]), ([2], [1])])
@pytest.mark.parametrize("real_form", [True, False])
def test_dense_matrix_is_the_matvec(ucs, k, real_form):
    """H_k as a matrix against its product with every unit vector: the same
    terms in another order, a hundred per entry at most (1e-13 of the norm)."""
    from edgpu.models import SU2_Model

    model = SU2_Model(spin=0.5, pure_theory=False, lvals=[6], has_obc=[False], sectors=[6], device="cuda")
    model.build_Hamiltonian(1.0, 0.5)
    if not real_form:
        model.H.build(force_complex=True)
    assert model.H.mat.is_complex != real_form
    model.set_momentum_sector(ucs, k)
    mom = model._momentum
    mom.bind(model.H)
    h = mom.dense()
    eye = torch.eye(mom.n_cols, dtype=torch.complex128, device="cuda")
    ref = torch.stack([mom.matvec(eye[c]) for c in range(mom.n_cols)], dim=1)
    assert float((h - ref).abs().max()) <= 1e-13 * float(ref.abs().max())


@pytest.mark.parametrize("n_cols", [1, 63, 64, 65, 3000])
def test_reduce_column_lengths(n_cols):
    """B^dagger w for columns of 0 to 33 entries: sums of at most 33 products
    of order one in another order (1e-13 each)."""
    from edgpu._lib import check, lib, ptr, stream_handle

    rng = np.random.default_rng(n_cols)
    lengths = rng.choice([0, 1, 3, 4, 5, 15, 16, 17, 33], n_cols)
    col_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    nnz, n_rows = int(col_ptr[-1]), 500
    rows = rng.integers(0, n_rows, nnz).astype(np.int32)
    data = rng.uniform(-1, 1, nnz) + 1j * rng.uniform(-1, 1, nnz)
    w = rng.uniform(-1, 1, n_rows) + 1j * rng.uniform(-1, 1, n_rows)
    up = lambda a: torch.from_numpy(np.concatenate([a, np.zeros(1, a.dtype)])).cuda()  # noqa: E731
    cp, ri, dv, wv = torch.from_numpy(col_ptr).cuda(), up(rows), up(data), up(w)
    y = torch.full((n_cols + 1,), 7.0, dtype=torch.complex128, device="cuda")
    check(lib.edg_momentum_reduce(n_cols, ptr(cp), ptr(ri), ptr(dv), ptr(wv), ptr(y), stream_handle()),
          "edg_momentum_reduce")
    ref = np.array([np.sum(data[a:b].conj() * w[rows[a:b]]) for a, b in zip(col_ptr[:-1], col_ptr[1:])])
    out = y.cpu().numpy()
    assert np.max(np.abs(out[:n_cols] - ref)) <= 1e-13 * 33 and out[n_cols] == 7.0


@pytest.mark.parametrize("name", ["su2_1d_L6_pbc", "su2_1d_L8_pbc_uc2", "qed1d_L6_pbc_uc2", "su2_1d_L8_pbc_tc"])
def test_host_arrays_narrowed_on_either_side(name, monkeypatch):
    """The projector's host arrays are the same, types included, whichever side
    narrows them."""
    from cases import build_momentum_case
    from edgpu import momentum

    model, g, m, ucs, ks = build_momentum_case(name, device="cuda")
    for k in ks:
        got = []
        for rows in (0, 1 << 30):
            monkeypatch.setattr(momentum, "HOST_ROWS", rows)
            model.set_momentum_sector(ucs, k, TC_symmetry=name.endswith("_tc"))
            got.append(model.momentum_basis)
        assert got[0].keys() == got[1].keys()
        for key, a in got[0].items():
            b = got[1][key]
            assert np.array_equal(a, b)
            if isinstance(a, np.ndarray):
                assert a.dtype == b.dtype and a.flags["C_CONTIGUOUS"] and b.flags["C_CONTIGUOUS"], key
