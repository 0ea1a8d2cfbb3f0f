"""One-launch sector enumeration against a host filter of the product space
and against the level-by-level path it hands over to: local dimensions on
both sides of the mask widths (8, 16, 32 states), U(1) and Z2 globals, link
pairs, n-body constraints, forbidden states, empty sectors, two-word keys, and
every hand-over point (the cap on a level's prefixes)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(dims, glob, links, nbody, strings, seed, frozen=0):
    from edgpu.symmetries import SectorSpec

    rng = np.random.default_rng(seed)
    n, dm = len(dims), int(max(dims))
    kw = dict(loc_dims=np.array(dims))
    if glob == "U":
        g = rng.integers(-1, 2, (2, n, dm)).astype(float)
        kw.update(glob_op_diags=g, glob_sectors=[0, 1], sym_type_flag="U")
    elif glob == "Z":
        kw.update(glob_op_diags=rng.choice([1.0, -1.0], (1, n, dm)), glob_sectors=[-1], sym_type_flag="Z")
    if links:
        kw.update(link_op_diags=rng.integers(-1, 2, (1, 2, n, dm)).astype(float), link_sectors=[0],
                  pair_list=[np.array([[n - 1, 0], [0, 1], [n - 3, n - 2]])])
    if nbody:
        kw.update(nbody_op_diags=rng.integers(0, 2, (2, n, dm)).astype(float), nbody_sectors=[1, 2],
                  nbody_sites_list=[np.array([0, n - 1, 1]), np.array([n - 2, 0, n - 3])], nbody_sym_type="U")
    if strings or frozen:
        sd = rng.integers(0, 2, (1, n, dm)).astype(float)
        st = np.zeros((1, n))
        if frozen:  # the leading sites keep one state each
            sd[0, :frozen] = np.arange(dm)
            sd[0, frozen:] = 0
        kw.update(string_op_diags=sd, string_sectors=st)
    return SectorSpec(**kw), kw


def _brute(kw, frozen):
    dims = kw["loc_dims"]
    n = len(dims)
    free = tuple(int(d) for d in dims[frozen:])
    cfg = np.stack(np.unravel_index(np.arange(int(np.prod(free))), free), axis=1)
    cfg = np.concatenate([np.zeros((len(cfg), frozen), dtype=cfg.dtype), cfg], axis=1)
    s_ = np.arange(n)
    ok = np.ones(len(cfg), dtype=bool)
    if "glob_op_diags" in kw:
        for g, t in zip(kw["glob_op_diags"], kw["glob_sectors"]):
            v = g[s_[None, :], cfg]
            ok &= (v.sum(axis=1) if kw["sym_type_flag"] == "U" else v.prod(axis=1)) == t
    if "link_op_diags" in kw:
        lv = kw["link_op_diags"][0]
        for a, b in kw["pair_list"][0]:
            ok &= lv[0, a, cfg[:, a]] + lv[1, b, cfg[:, b]] == 0
    if "nbody_op_diags" in kw:
        for v, t, sites in zip(kw["nbody_op_diags"], kw["nbody_sectors"], kw["nbody_sites_list"]):
            ok &= sum(v[s, cfg[:, s]] for s in sites) == t
    if "string_op_diags" in kw:
        ok &= np.all(kw["string_op_diags"][0][s_[None, :], cfg] == 0, axis=1)
    return cfg[ok]


@pytest.mark.parametrize("dims,frozen", [([3] * 9, 0), ([2, 1, 8, 3, 8, 2, 4], 0), ([4, 9, 3, 16, 5], 0),
                                         ([3, 17, 32, 4, 2], 0), ([2, 33, 3, 5, 4], 0), ([3] * 46, 38)])
@pytest.mark.parametrize("glob", ["U", "Z", None])
@pytest.mark.parametrize("links,nbody,strings", [(True, False, False), (False, True, False), (True, True, True),
                                                 (False, False, False)])
def test_levels_match_the_filtered_product_space(dims, frozen, glob, links, nbody, strings, monkeypatch):
    from edgpu import symmetries

    spec, kw = _spec(dims, glob, links, nbody, strings, 11 * len(dims) + links + 2 * nbody, frozen)
    ref = _brute(kw, frozen)
    sizes = None
    for cap in (1 << 22, 5000, 300, 20, 1):
        monkeypatch.setattr(symmetries, "LEVELS_CAP", cap)
        sec = symmetries.enumerate_sector(spec)
        assert len(sec) == len(ref), cap
        if len(ref):
            assert np.array_equal(sec.configs, ref), cap
        assert sizes is None or sec.level_sizes == sizes
        sizes = sec.level_sizes


def test_little_free_memory():
    """With 60 MB left the enumeration works with fewer prefixes a level."""
    import torch

    from edgpu.symmetries import SectorSpec, enumerate_sector, get_symmetry_sector_generators

    op = np.zeros((14, 4, 4))
    op[:, np.arange(4), np.arange(4)] = np.arange(4)
    op[6:, 1:, 1:] = 9.0  # the last sites keep their first state: 4^6 states pass
    gens = get_symmetry_sector_generators([op], "global")
    spec = SectorSpec(loc_dims=np.full(14, 4), glob_op_diags=gens, glob_sectors=[9], sym_type_flag="U")
    want = enumerate_sector(spec)
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    room = torch.cuda.memory_reserved() + 60 * 2**20
    torch.cuda.set_per_process_memory_fraction(room / total)
    try:
        got = enumerate_sector(spec)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert len(want) > 100 and torch.equal(got.keys, want.keys) and got.level_sizes == want.level_sizes
