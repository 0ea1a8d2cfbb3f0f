"""The maps between the real-form basis and the original one under torch's
transformations (CPU only: the phase kernel is a stand-in that reads the
values of the tensor it is given and knows of nothing else)."""

import numpy as np
import pytest
import torch

from edgpu.modeling.hamiltonian import QMB_hamiltonian

N = 6


class _Sector:
    keys = torch.arange(N)
    device = keys.device

    def __len__(self):
        return N


@pytest.fixture
def maps(monkeypatch):
    ham = QMB_hamiltonian([N], N, sector=_Sector())
    phase = torch.tensor([1, 1j, -1, -1j, 1, 1j], dtype=torch.complex128)
    raw = []

    def apply(tab, psi, conj):
        ph = phase.conj().resolve_conj() if conj else phase
        if psi is None:
            return ph.clone()
        raw.append(psi)
        return torch.from_numpy(ph.numpy() * psi.detach().numpy())

    monkeypatch.setattr(ham, "_phase_table", lambda: torch.zeros(1))
    monkeypatch.setattr(ham, "_apply_phase", apply)
    return [(ham.to_original_basis, phase, raw), (ham.from_original_basis, phase.conj().resolve_conj(), raw)]


def _vec(seed, dtype=torch.complex128, *shape):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*(shape or (N,)), dtype=dtype, generator=g)


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_a_plain_vector_goes_to_the_kernel(maps, dtype):
    for f, phase, raw in maps:
        x = _vec(1, dtype)
        assert torch.equal(f(x), phase * x) and raw[-1] is x


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_forward_mode(maps, dtype):
    import torch.autograd.forward_ad as fw

    x, t = _vec(2, dtype), _vec(3, dtype)
    for f, phase, _ in maps:
        with fw.dual_level():
            out = fw.unpack_dual(f(fw.make_dual(x, t)))
        assert torch.equal(out.primal, phase * x) and torch.equal(out.tangent, phase * t)
        y, dy = torch.func.jvp(f, (x,), (t,))
        assert torch.equal(y, phase * x) and torch.equal(dy, phase * t)


def test_vmap(maps):
    x = _vec(4, torch.complex128, 3, N)
    for f, phase, _ in maps:
        assert torch.equal(torch.func.vmap(f)(x), phase * x)
        assert torch.equal(torch.func.vmap(f, in_dims=1)(x.T.contiguous()), phase * x)


def test_reverse_mode(maps):
    for f, phase, _ in maps:
        x = _vec(5).requires_grad_()
        f(x).real.sum().backward()
        assert torch.allclose(x.grad, phase.conj() * torch.ones(N, dtype=torch.complex128))
        g = torch.func.grad(lambda v: (f(v).abs() ** 2).sum())(x.detach())
        assert torch.allclose(g, 2 * x.detach())


def test_trace(maps):
    from torch.fx.experimental.proxy_tensor import make_fx

    x, z = _vec(6), _vec(7)
    for f, phase, _ in maps:
        assert np.allclose(make_fx(lambda v: f(v))(x)(z), phase * z)  # noqa: B023


def test_lazy_conjugation_and_sign(maps):
    x = _vec(8)
    for f, phase, _ in maps:
        assert torch.equal(f(x.conj()), phase * x.conj())
        y = x.conj().imag  # a lazy sign
        assert y.is_neg() and torch.equal(f(y), phase * y)


def test_phase_table_follows_the_matrix():
    """Exponents that are replaced or changed in place after a first use."""
    from types import SimpleNamespace

    ham = QMB_hamiltonian([N], N, sector=_Sector())
    w = np.arange(12).reshape(4, 3)
    ham.mat = SimpleNamespace(phase_weights=w)
    assert np.array_equal(ham._phase_table().numpy(), w % 4)
    assert ham._phase_table() is ham._phase_table()
    w[2, 1] += 1
    assert np.array_equal(ham._phase_table().numpy(), w % 4)
    ham.mat.phase_weights = w[:, ::-1] + 2
    assert np.array_equal(ham._phase_table().numpy(), (w[:, ::-1] + 2) % 4)
    ham.mat.phase_weights = None
    assert ham._phase_table() is None
