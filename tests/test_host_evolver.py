"""What a KrylovEvolver prepares (CPU only: host arrays, no step is taken)."""

import pytest
import torch

from edgpu import solvers
from edgpu.dynamics import KrylovEvolver
from edgpu.modeling.assembly import DeviceMatrix

COOP_MAX = 1024 * 148  # rows of the one-launch step


class _Layout:
    tile_off = words = torch.zeros(4, dtype=torch.int32)
    count, colbits = 2, 18

    def table(self, dtype):
        return self.words


@pytest.fixture
def asked(monkeypatch):
    calls = []

    def packed(mat):
        calls.append("pack")
        return _Layout() if mat.packs else None

    monkeypatch.setattr(solvers, "packed_layout", packed)
    monkeypatch.setattr(solvers, "tune_spmv_group", lambda *a, **k: calls.append("tune") or 8)
    return calls


def _matrix(n, packs=True, cplx=False):
    rowptr = torch.zeros(n + 1, dtype=torch.int64)
    rowptr[n:] = 1
    w = 2 if cplx else 1
    mat = DeviceMatrix(n, rowptr, torch.zeros(1, dtype=torch.int32), torch.ones(w, dtype=torch.float64),
                       torch.zeros(n * w, dtype=torch.float64), None, cplx)
    mat.packs = packs
    return mat


@pytest.mark.parametrize("n", [40, COOP_MAX])
@pytest.mark.parametrize("precision", ["c128", "c64"])
@pytest.mark.parametrize("matvec", ["auto", "csr"])
@pytest.mark.parametrize("cplx", [False, True])
def test_a_one_launch_step_packs_and_tunes_nothing(n, precision, matvec, cplx, asked):
    ev = KrylovEvolver(_matrix(n, cplx=cplx), precision=precision, matvec=matvec)
    assert asked == [] and not ev.p.pk_words and ev.p.cols and ev.p.vals and ev.p.spmv_group == 0
    assert (ev.packed is not None) == (matvec == "auto" and not cplx)  # built when asked for
    assert ev.packed is ev.packed
    assert KrylovEvolver(_matrix(n), spmv_group=4).p.spmv_group == 4


@pytest.mark.parametrize("matvec,packs,cplx,want", [("auto", True, False, ["pack"]), ("auto", False, False,
                                                                                      ["pack", "tune"]),
                                                    ("csr", True, False, ["tune"]), ("auto", True, True, [])])
def test_larger_sectors_choose_their_product(matvec, packs, cplx, want, asked):
    ev = KrylovEvolver(_matrix(COOP_MAX + 1, packs, cplx), m=4, matvec=matvec)
    assert asked == want
    assert bool(ev.p.pk_words) == (want == ["pack"]) == (ev.packed is not None)
    assert ev.p.spmv_group == (8 if "tune" in want else 0)
