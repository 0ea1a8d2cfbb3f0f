"""Which matrices share a packed layout (CPU only: the layout's builder is a
stand-in that records the arrays it was given)."""

import pytest
import torch

from edgpu import solvers
from edgpu.modeling.assembly import DeviceMatrix


class _Layout:
    def __init__(self, mat):
        self.vals = mat.vals.clone()


@pytest.fixture
def builds(monkeypatch):
    made = []

    def build(mat):
        made.append(_Layout(mat))
        return made[-1]

    monkeypatch.setattr(solvers.PackedLayout, "build", build)
    return made


def _arrays():
    return (torch.tensor([0, 1, 2]), torch.tensor([1, 0], dtype=torch.int32), torch.tensor([0.5, 0.5],
                                                                                          dtype=torch.float64))


def _matrix(arrays, home=None):
    mat = DeviceMatrix(2, *arrays, torch.zeros(2, dtype=torch.float64), None, False)
    if home is not None:
        mat._shared = home
    return mat


def _home(arrays):
    return {"arrays": arrays}


def test_matrices_of_one_off_diagonal_part_share_the_layout(builds):
    arrays = _arrays()
    home = _home(arrays)
    a, b = _matrix(arrays, home), _matrix(arrays, home)
    lay = solvers.packed_layout(a)
    assert solvers.packed_layout(b) is lay and solvers.packed_layout(a) is lay and len(builds) == 1
    assert solvers.packed_layout(_matrix(arrays)) is not lay  # not of that part


@pytest.mark.parametrize("name", ["rowptr", "cols", "vals"])
@pytest.mark.parametrize("first", ["own", "shared"])
def test_other_arrays_have_a_layout_of_their_own(name, first, builds):
    arrays = _arrays()
    home = _home(arrays)
    a, b = _matrix(arrays, home), _matrix(arrays, home)
    setattr(b, name, getattr(b, name).clone())
    if name == "vals":
        b.vals[:] = 2.0
    for mat in ((b, a) if first == "own" else (a, b)):
        assert torch.equal(solvers.packed_layout(mat).vals, mat.vals)
    assert solvers.packed_layout(a) is not solvers.packed_layout(b) and len(builds) == 2
    assert solvers.packed_layout(_matrix(arrays, home)) is solvers.packed_layout(a)


def test_arrays_given_after_the_layout_was_built(builds):
    arrays = _arrays()
    a = _matrix(arrays, _home(arrays))
    lay = solvers.packed_layout(a)
    a.vals = torch.full((2,), 3.0, dtype=torch.float64)
    assert torch.equal(solvers.packed_layout(a).vals, a.vals)
    a.vals = arrays[2]
    assert solvers.packed_layout(a) is lay  # still the part's


def test_values_changed_in_place(builds):
    arrays = _arrays()
    home = _home(arrays)
    a, b = _matrix(arrays, home), _matrix(arrays, home)
    solvers.packed_layout(a)
    arrays[2].mul_(4.0)
    assert torch.equal(solvers.packed_layout(b).vals, arrays[2])
    assert torch.equal(solvers.packed_layout(a).vals, arrays[2]) and len(builds) == 2


def test_a_matrix_that_does_not_pack_is_asked_once(monkeypatch):
    calls = []
    monkeypatch.setattr(solvers.PackedLayout, "build", lambda mat: calls.append(mat))
    arrays = _arrays()
    home = _home(arrays)
    assert solvers.packed_layout(_matrix(arrays, home)) is None
    assert solvers.packed_layout(_matrix(arrays, home)) is None and len(calls) == 1
