"""Timed cases of the engine: what its users have it do, through the model API.

Each case is one pass of a path as a user's program calls it: building a
sector and its Hamiltonian, ground states (single and coupling sweeps, plain
and mixed precision), batches of small instances, time evolution, observables,
momentum sectors and the matrix-free Z_n engine.  Couplings, states and
vectors come from the seed; lattices, precisions and options from the case.

``exact`` recomputes the floating-point results in 64 bits with plain torch
and numpy from the inputs in hand (the sector's keys, the assembled matrix,
the operators): a fully reorthogonalised Lanczos or a dense solve, a Taylor
series of exp(-iHt), sums over decoded configurations, and an explicit
translation-by-translation Z_n Hamiltonian.
"""

import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ed-lgt_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from edgpu.batch import TiledBatch  # noqa: E402
from edgpu.models import QED_Model, SU2_Model  # noqa: E402
from edgpu.models.zn_model import ZnModel  # noqa: E402
from edgpu.solvers import lanczos_mixed  # noqa: E402


# --------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest solve: the 1D QED chain of the test configurations, its
        # two lowest eigenvalues, where launches and host work count
        {"name": "ground_qed_8", "path": "ground", "model": "qed", "lx": 8, "ly": 1, "pbc": False, "k": 2,
         "precision": "fp64", "g": 1.0, "m": 1.0},
        # an ordinary plain f64 ground state (73,789 rows, full reorthogonalisation)
        {"name": "ground_su2_12", "path": "ground", "model": "su2", "lx": 12, "ly": 1, "pbc": False, "k": 1,
         "precision": "fp64", "g": 1.0, "m": 0.5},
        # the headline coupling sweep: three ground states of the periodic
        # L = 14 chain (1,232,454 rows), mixed precision, one batched solve
        {"name": "sweep_su2_14", "path": "sweep", "lx": 14, "pbc": True, "couplings": 3, "g": 1.0, "m": 0.5},
        # sector enumeration and assembly from nothing, large 1D sector
        {"name": "setup_su2_14", "path": "setup", "model": "su2", "lx": 14, "ly": 1, "pbc": True, "g": 1.0, "m": 0.5},
        # the same in 2D with plaquettes and two-word keys (197,547 rows)
        {"name": "setup_qed_4x4", "path": "setup", "model": "qed_pure", "lx": 4, "ly": 4, "pbc": True, "g": 1.0,
         "m": 0.0},
        # string-breaking quench of a static pair: complex64 Krylov steps with
        # observables at every step (7,133,222 rows)
        {"name": "quench_su2_16", "path": "quench", "lx": 16, "first": 5, "second": 10, "precision": "c64",
         "krylov": 30, "reorth": 0, "steps": 2, "dt": 0.05, "keep": False, "g": 1.0, "m": 1.0},
        # a small quench with the default options, states kept at every time
        {"name": "quench_su2_10", "path": "quench", "lx": 10, "first": 3, "second": 6, "precision": "c128",
         "krylov": 30, "reorth": 1, "steps": 10, "dt": 0.05, "keep": True, "g": 1.0, "m": 1.0},
        # local densities and two-body correlators of a large state
        {"name": "observe_su2_16", "path": "observe", "lx": 16, "first": 5, "second": 10, "dtype": "complex128"},
        # couplings and charge sectors of the 3x2 lattice beside larger
        # chains, in one batched solve
        {"name": "batch_qed_3x2", "path": "batch", "instances": 64, "charges": True, "chain": 10,
         "precision": "mixed"},
        # the largest lattice: one batched application of the matrix-free Z3
        # Hamiltonian on 4x3 (245,518,920 rows, eight couplings)
        {"name": "zn_apply_4x3", "path": "zn_apply", "lx": 4, "ly": 3, "zn": 3, "nvec": 8, "dtype": "float32"},
        # ground states of a smaller Z3 lattice at four couplings
        {"name": "zn_ground_4x2", "path": "zn_ground", "lx": 4, "ly": 2, "zn": 3, "nvec": 4, "precision": "mixed"},
        # a momentum sector: projector and ground state
        {"name": "momentum_su2_12", "path": "momentum", "lx": 12, "kx": 0, "g": 1.0, "m": 0.5},
    ]


def draw(rng):
    path = rng.choice(["ground", "ground", "sweep", "setup", "setup", "quench", "quench", "observe", "batch",
                       "zn_apply", "zn_ground", "momentum"])
    g, m = round(rng.uniform(0.6, 1.6), 3), round(rng.uniform(0.3, 1.2), 3)
    if path in ("ground", "setup"):
        model = rng.choice(["su2", "su2", "qed"] + (["qed_pure"] if path == "setup" else []))
        if model == "su2":
            lx, ly, pbc = rng.choice([6, 8, 10, 12] + ([14] if path == "setup" else [])), 1, rng.random() < 0.5
        elif model == "qed":
            lx, ly = rng.choice([(6, 1), (8, 1), (10, 1), (12, 1), (14, 1), (3, 2), (4, 2)])
            pbc = ly == 1 and rng.random() < 0.5
        else:
            lx, ly = rng.choice([(2, 2), (3, 2), (3, 3), (4, 3), (4, 4)])
            pbc, m = True, 0.0
        c = {"path": path, "model": model, "lx": lx, "ly": ly, "pbc": pbc, "g": g, "m": m}
        if path == "ground":
            c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
            # rings have degenerate pairs above the ground state
            c["k"] = 1 if c["precision"] == "mixed" or pbc else rng.choice([1, 2, 3])
        return c
    if path == "sweep":
        return {"path": path, "lx": rng.choice([8, 10, 12, 14]), "pbc": rng.random() < 0.5,
                "couplings": rng.choice([1, 2, 3]), "g": g, "m": m}
    if path in ("quench", "observe"):
        lx = rng.choice([8, 10, 12, 14] + ([16] if path == "observe" else []))
        first = rng.randrange(1, lx // 2)
        c = {"path": path, "lx": lx, "first": first, "second": rng.randrange(first + 1, lx - 1)}
        if path == "observe":
            c["dtype"] = rng.choice(["float64", "float32", "complex128", "complex64"])
            return c
        return {**c, "precision": rng.choice(["c64", "c128"]), "krylov": rng.randrange(12, 37),
                "reorth": rng.choice([0, 1]), "steps": rng.randrange(1, 6), "dt": round(rng.uniform(0.02, 0.06), 3),
                "keep": rng.random() < 0.5, "g": g, "m": m}
    if path == "batch":
        return {"path": path, "instances": int(round(math.exp(rng.uniform(math.log(3), math.log(64))))),
                "charges": rng.random() < 0.5, "chain": rng.choice([0, 6, 8, 10]),
                "precision": rng.choice(["mixed", "fp64"])}
    if path == "momentum":
        lx = rng.choice([6, 8, 10, 12])
        return {"path": path, "lx": lx, "kx": rng.randrange(lx), "g": g, "m": m}
    lx, ly, zn = rng.choice([(2, 2, 4), (2, 3, 3), (4, 2, 2), (4, 2, 3), (2, 4, 3)]
                            + ([(2, 5, 3), (6, 2, 2), (4, 3, 2)] if path == "zn_apply" else []))
    c = {"path": path, "lx": lx, "ly": ly, "zn": zn, "nvec": rng.choice([1, 2, 4, 8])}
    if path == "zn_apply":
        c["dtype"] = rng.choice(["float32", "float64"])
        c["scale"] = round(rng.uniform(0.5, 2.0), 3)
    else:
        c["precision"] = rng.choice(["mixed", "fp64"])
        c["scale"] = round(rng.uniform(0.9, 1.1), 3)
    return c


# ---------------------------------------------------------------- the models
def _model_kwargs(c):
    name = c.get("model", "su2")
    lvals = [c["lx"]] if c.get("ly", 1) == 1 else [c["lx"], c["ly"]]
    obc = [not c.get("pbc", False)] * len(lvals)
    if name == "su2":
        kw = dict(spin=0.5, pure_theory=False, lvals=lvals, has_obc=obc, sectors=[c["lx"]])
        if "first" in c:  # two static j = 1/2 charges
            kw["bg_list"] = [0.5 if s in (c["first"], c["second"]) else 0 for s in range(c["lx"])]
        return SU2_Model, kw
    return QED_Model, dict(spin=1, pure_theory=name == "qed_pure", lvals=lvals, has_obc=obc)


def _model(c):
    cls, kw = _model_kwargs(c)
    return cls(**kw, device="cuda")


def _couplings(c, seed, n=1):
    """n coupling pairs within 5 % of the case's centre."""
    r = np.random.default_rng([int(seed), 17])
    return [(float(c["g"] * r.uniform(0.95, 1.05)), float(c["m"] * r.uniform(0.95, 1.05))) for _ in range(n)]


def _build(model, c, g, m):
    model.build_Hamiltonian(g) if c.get("model") == "qed_pure" else model.build_Hamiltonian(g, m)
    return model.H.mat


def _sweep_couplings(c, seed):
    f = {1: (1.0,), 2: (0.5, 2.0), 3: (0.5, 1.0, 2.0)}[c["couplings"]]
    return [(a * g, m) for a, (g, m) in zip(f, _couplings(c, seed, len(f)))]


def _batch_matrices(c, seed):
    """g log-uniform in [0.1, 5] and m uniform in [0, 2] in the zero-charge
    sector of the 3x2 lattice, the charged sectors, and an open chain."""
    r = np.random.default_rng([int(seed), 23])
    base = QED_Model(spin=1, pure_theory=False, lvals=[3, 2], has_obc=[True, True], device="cuda")
    mats = []
    for _ in range(c["instances"]):
        mats.append(_build(base, c, float(np.exp(r.uniform(np.log(0.1), np.log(5.0)))), float(r.uniform(0.0, 2.0))))
    if c["charges"]:
        for q, bg in {-2: [1, 0, 0, 0, 0, 1], -1: [1, 0, 0, 0, 0, 0], 1: [-1, 0, 0, 0, 0, 0],
                      2: [-1, 0, 0, 0, 0, -1]}.items():
            mq = QED_Model(spin=1, pure_theory=False, lvals=[3, 2], has_obc=[True, True], bg_list=bg, charge=q,
                           device="cuda")
            mats.append(_build(mq, c, float(r.uniform(0.9, 1.1)), 1.0))
    if c["chain"]:
        chain = SU2_Model(spin=0.5, pure_theory=False, lvals=[c["chain"]], has_obc=[True], sectors=[c["chain"]],
                          device="cuda")
        mats.append(_build(chain, c, float(r.uniform(0.9, 1.1)), 0.5))
    return mats


def _zn_couplings(c, seed):
    r = np.random.default_rng([int(seed), 29])
    g = np.geomspace(0.7, 1.6, c["nvec"]) * c.get("scale", 1.0) * r.uniform(0.97, 1.03, c["nvec"])
    return g, float(r.uniform(0.45, 0.55))


def _random_state(n, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    wide = torch.complex128 if dtype.startswith("complex") else torch.float64
    psi = torch.randn(n, dtype=wide, device="cuda", generator=gen)
    return (psi / torch.linalg.vector_norm(psi)).to(getattr(torch, dtype))


_LOCAL = ("E_square", "T2_px", "N_tot", "N_pair")
_TWOBODY = (("N_pair", "N_pair"), ("T2_px", "T2_px"), ("N_tot", "T2_px"))


# ------------------------------------------------------------------ the paths
def prepare(case, seed):
    c, path = case, case["path"]
    s = {"case": c}
    if path == "setup":
        # nothing is in hand but the parameters
        s["coupling"] = _couplings(c, seed)[0]
    elif path == "ground":
        s["model"] = _model(c)
        s["coupling"] = _couplings(c, seed)[0]
        # the bare vacuum, whose amplitude fixes the phase of the state
        s["vacuum"] = _vacuum(_build(s["model"], c, *s["coupling"]))
    elif path == "sweep":
        s["model"] = _model(c)
        s["couplings"] = _sweep_couplings(c, seed)
        s["vacuum"] = torch.stack([_vacuum(_build(s["model"], c, *p)) for p in s["couplings"]])
    elif path == "quench":
        s["model"] = model = _model(c)
        g, m = _couplings(c, seed)[0]
        _build(model, c, g, m)
        # a string state: the configuration of lowest diagonal energy
        psi = np.zeros(model.sector_dim, dtype=np.complex128)
        psi[int(_vacuum(model.H.mat))] = 1.0
        s["psi"] = psi
        s["times"] = np.arange(c["steps"] + 1) * c["dt"]
        s["obs"] = None if c["keep"] else {k: model.ops[k] for k in ("T2_px", "N_pair")}
    elif path == "observe":
        s["model"] = model = _model(c)
        s["psi"] = _random_state(model.sector_dim, c["dtype"], seed)
    elif path == "batch":
        s["mats"] = _batch_matrices(c, seed)
        s["batch"] = TiledBatch(s["mats"], k=1, precision=c["precision"])
        s["batch"].capture()
    elif path == "zn_apply":
        s["model"] = model = ZnModel((c["lx"], c["ly"]), c["zn"], device="cuda")
        g, m = _zn_couplings(c, seed)
        s["couplings"] = torch.from_numpy(np.ascontiguousarray(model.build_Hamiltonian(g, m))).cuda()
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        s["x"] = torch.randn((model.sector_dim, c["nvec"]), dtype=getattr(torch, c["dtype"]), device="cuda",
                             generator=gen)
        s["y"] = torch.empty_like(s["x"])
    elif path == "zn_ground":
        s["model"] = model = ZnModel((c["lx"], c["ly"]), c["zn"], device="cuda")
        s["g"], s["m"] = _zn_couplings(c, seed)
        model.build_Hamiltonian(s["g"], s["m"])
        s["vacuum"] = _zn_vacuum(model)
    elif path == "momentum":
        s["model"] = _model({**c, "pbc": True})
        s["coupling"] = _couplings(c, seed)[0]
    else:
        raise ValueError(f"unknown path {path}")
    return s


def run(state):
    s, c, path = state, state["case"], state["case"]["path"]
    if path == "setup":
        model = _model(c)
        mat = _build(model, c, *s["coupling"])
        return {"keys": model.sector.keys, "rowptr": mat.rowptr, "cols": mat.cols, "vals": mat.vals,
                "diag": mat.diag, "present": mat.diag_present}
    if path == "ground":
        model = s["model"]
        _build(model, c, *s["coupling"])
        model.diagonalize_Hamiltonian(c["k"], precision=c["precision"])
        psi = _phase_fixed(model.H.GSpsi.device(), s["vacuum"])
        # the state of a mixed-precision solve is kept in single precision
        return {"energy": model.H.Nenergies,
                "psi": psi.to(torch.complex64 if psi.is_complex() else torch.float32)
                if c["precision"] == "mixed" else psi}
    if path == "sweep":
        model = s["model"]
        mats = [_build(model, c, *p) for p in s["couplings"]]
        r64, _ = lanczos_mixed(mats[0], diags=[mt.diag for mt in mats])
        psi = r64.evecs[0]  # (rows, couplings)
        sign = torch.sign(psi.gather(0, s["vacuum"][None, :]))
        return {"energies": r64.evals[:, 0], "psi": (psi * sign).to(torch.float32)}
    if path == "quench":
        model = s["model"]
        model.time_evolution_Hamiltonian(s["psi"], s["times"], m_krylov=c["krylov"], precision=c["precision"],
                                         observables=s["obs"], reorth_passes=c["reorth"])
        single = c["precision"] == "c64"  # results of a complex64 evolution are kept in single precision
        if c["keep"]:
            states = torch.stack([p.device() for p in model.H.psi_time])
            return {"states": states.to(torch.complex64) if single else states}
        return {k: v.astype(np.float32) if single else v for k, v in model.H.obs_time.items()}
    if path == "observe":
        model, psi = s["model"], s["psi"]
        out = {k: model.local_expval(model.ops[k], psi) for k in _LOCAL}
        for a, b in _TWOBODY:
            out[f"{a}_{b}"] = model.twobody_expval(model.ops[a], model.ops[b], psi)
        return out
    if path == "batch":
        return {"energies": s["batch"].solve().clone()}
    if path == "zn_apply":
        s["model"].engine.matvec(s["x"], s["y"], s["couplings"], c["nvec"])
        return {"y": s["y"]}
    if path == "zn_ground":
        model = s["model"]
        res = model.diagonalize_Hamiltonian(1, precision=c["precision"])
        psi = res.evecs.view(-1, c["nvec"])[: model.sector_dim]
        # the refinement stops at a relative residual of 1e-8: single precision
        return {"energies": res.evals[:, 0], "psi": (psi * torch.sign(psi[s["vacuum"]])).to(torch.float32)}
    model = s["model"]  # momentum
    _build(model, c, *s["coupling"])
    model.set_momentum_sector([1], [c["kx"]])
    model.diagonalize_Hamiltonian(1)
    b = model.momentum_basis
    return {"energy": model.H.Nenergies, "col_ptr": b["L_col_ptr"], "row_idx": b["L_row_idx"], "data": b["L_data"]}


def _vacuum(mat):
    """Row of the lowest diagonal element (device index)."""
    d = mat.diag.view(torch.complex128).real if mat.is_complex else mat.diag
    return torch.argmin(d)


def _phase_fixed(psi, row):
    """psi times the phase that makes its amplitude on ``row`` positive."""
    a = psi[row]
    return psi * (a.conj() / a.abs())


def _zn_vacuum(model):
    """Row of the lowest diagonal energy at the first coupling."""
    L = model.lattice
    keys = model.engine.keys[: model.sector_dim]
    d = torch.zeros(len(keys), dtype=torch.float64, device="cuda")
    for l in range(L.n_links):
        f = (keys >> (L.link_bits * l)) & ((1 << L.link_bits) - 1)
        d += model.couplings[0][2] * torch.where(f > L.n // 2, f - L.n, f) ** 2
    for s in range(L.n_sites):
        d += model.couplings[0][1] * (1 - 2 * (s % L.lx % 2)) * ((keys >> (L.field_bits + s)) & 1)
    return int(torch.argmin(d))


# ------------------------------------------------------------------ the work
@lru_cache(maxsize=None)
def _shape(items):
    """(rows, off-diagonal entries) of a case's sector matrix."""
    c = dict(items)
    model = _model(c)
    mat = _build(model, c, 1.0, 0.5)
    return mat.n, mat.nnz


def _shape_of(c, **more):
    c = {k: v for k, v in {**c, **more}.items() if k in ("model", "lx", "ly", "pbc", "first", "second")}
    return _shape(tuple(sorted(c.items())))


@lru_cache(maxsize=None)
def _zn_rows(lx, ly, zn):
    return ZnModel((lx, ly), zn, device="cuda").sector_dim


def work(case):
    """Every input once, every output once; a Krylov method cannot do with
    less than one product with the matrix (4-byte columns and its values)."""
    c, path = case, case["path"]
    if path == "setup":
        n, nnz = _shape_of(c)
        return {"bytes": 8 * n + 8 * (n + 1) + 12 * nnz + 9 * n, "flops": 2 * nnz}
    if path == "ground":
        n, nnz = _shape_of(c)
        return {"bytes": 12 * nnz + 8 * (n + 1) + 8 * n + 16 * n, "flops": 2 * nnz}
    if path == "sweep":
        n, nnz = _shape_of(c)
        v = c["couplings"]
        return {"bytes": 8 * nnz + 8 * (n + 1) + 8 * n * v + 4 * n * v, "flops": 2 * nnz * v}
    if path == "quench":
        n, nnz = _shape_of(c)
        s = 8 if c["precision"] == "c64" else 16
        out = c["steps"] * n * s if c["keep"] else 0
        # every step multiplies by the matrix krylov times and reads each Krylov vector once more
        return {"bytes": c["steps"] * c["krylov"] * (4 * nnz + 3 * n * s) + out,
                "flops": c["steps"] * c["krylov"] * 4 * nnz}
    if path == "observe":
        n, _ = _shape_of(c)
        pairs = c["lx"] * (c["lx"] - 1) // 2
        s = {"float64": 8, "float32": 4, "complex128": 16, "complex64": 8}[c["dtype"]]
        return {"bytes": n * (8 + s), "flops": n * (2 * c["lx"] * len(_LOCAL) + 2 * pairs * len(_TWOBODY))}
    if path == "batch":
        n = 90 * c["instances"] + (171 if c["charges"] else 0)
        nnz = 4 * n
        if c["chain"]:
            cn, cz = _shape_of({"lx": c["chain"]})
            n, nnz = n + cn, nnz + cz
        return {"bytes": 12 * nnz + 16 * n, "flops": 2 * nnz}
    if path in ("zn_apply", "zn_ground"):
        n, v = _zn_rows(c["lx"], c["ly"], c["zn"]), c["nvec"]
        e = 4 if c.get("dtype") == "float32" else 8
        return {"bytes": n * (8 + 2 * e * v), "flops": 2 * n * v * 3 * c["lx"] * c["ly"]}
    n, nnz = _shape_of(c, pbc=True)
    return {"bytes": 8 * n + 12 * nnz + 20 * n, "flops": 2 * nnz}


# ------------------------------------------------------- the results in 64 bits
def exact(case, seed):
    path = case["path"]
    if path == "setup":
        return None  # keys and pattern are whole numbers; the values are the operators' own elements
    if path == "zn_apply":
        return _exact_zn_apply(case, seed)
    return {"ground": _exact_ground, "sweep": _exact_sweep, "quench": _exact_quench, "observe": _exact_observe,
            "batch": _exact_batch, "zn_ground": _exact_zn_ground, "momentum": _exact_momentum}[path](case, seed)


def _matrix(mat):
    """x -> H x for (rows, columns) operands, from the assembled arrays."""
    kind = torch.complex128 if mat.is_complex else torch.float64
    vals = mat.vals.view(kind) if mat.is_complex else mat.vals
    diag = mat.diag.view(kind) if mat.is_complex else mat.diag
    a = torch.sparse_csr_tensor(mat.rowptr, mat.cols.to(torch.int64), vals, size=(mat.n, mat.n))

    def apply(x):
        if x.is_complex() and not mat.is_complex:
            r = torch.view_as_real(x)
            return torch.view_as_complex((a @ r + diag[:, None] * r).contiguous())
        y = x.reshape(mat.n, -1).to(kind)
        return (a @ y + diag[:, None] * y).reshape(x.shape)

    return apply, kind


def _lowest(apply, n, k, kind=torch.float64, start=None, most=500):
    """The k lowest eigenpairs by Lanczos with two Gram-Schmidt passes."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    if start is None:
        start = torch.randn(n, dtype=kind, device="cuda", generator=gen)
    most = min(most, n)
    q = torch.empty((most + 1, n), dtype=kind, device="cuda")
    q[0] = start / torch.linalg.vector_norm(start)
    a, b = [], []
    for j in range(most):
        w = apply(q[j])
        a.append(float(torch.vdot(q[j], w).real))
        for _ in range(2):
            w = w - q[: j + 1].T @ (q[: j + 1].conj() @ w)
        b.append(float(torch.linalg.vector_norm(w)))
        last = b[-1] <= 1e-11 * max(1.0, abs(a[-1])) or j + 1 == most
        if j + 1 >= k and (last or j % 10 == 9):
            t = np.diag(a) + np.diag(b[:-1], 1) + np.diag(b[:-1], -1)
            e, v = np.linalg.eigh(t)
            if last or np.max(np.abs(b[-1] * v[-1, :k])) < 1e-13 * max(1.0, abs(e[0])):
                break
        q[j + 1] = w / b[-1]
    coef = torch.from_numpy(v[:, :k].astype(np.complex128 if kind.is_complex else np.float64)).cuda()
    return e[:k], (q[: len(a)].T @ coef)


def _eigen(mat, k):
    apply, kind = _matrix(mat)
    if mat.n <= 3000:
        h = apply(torch.eye(mat.n, dtype=kind, device="cuda"))
        e, v = torch.linalg.eigh(h)
        return e[:k].cpu().numpy(), v[:, :k]
    return _lowest(apply, mat.n, k, kind)


def _digits(model):
    """Local state of every site and row, decoded from one-word keys."""
    k = model.sector.keys.clone()
    out = [None] * len(model.loc_dims)
    for s in range(len(model.loc_dims) - 1, -1, -1):
        d = int(model.loc_dims[s])
        out[s] = k % d
        k = torch.div(k, d, rounding_mode="floor")
    return out


def _gauge(model):
    """i**e(row) that maps a real-form vector to the model's basis, or None."""
    w = model.H.mat.phase_weights
    if w is None:
        return None
    w = torch.from_numpy(np.asarray(w, dtype=np.int64)).cuda()
    e = sum(w[s][d] for s, d in enumerate(_digits(model))) % 4
    return torch.tensor([1, 1j, -1, -1j], dtype=torch.complex128, device="cuda")[e]


def _exact_ground(c, seed):
    s = prepare(c, seed)
    model = s["model"]
    e, v = _eigen(model.H.mat, c["k"])
    psi = v[:, 0]
    ph = _gauge(model)
    psi = psi if ph is None else ph * psi
    return {"energy": e / model.n_sites, "psi": _phase_fixed(psi, s["vacuum"])}


def _exact_sweep(c, seed):
    s = prepare(c, seed)
    es, vs = [], []
    for p, row in zip(s["couplings"], s["vacuum"]):
        e, v = _eigen(_build(s["model"], c, *p), 1)
        es.append(e[0])
        vs.append(v[:, 0] * torch.sign(v[row, 0]))
    return {"energies": np.array(es), "psi": torch.stack(vs, dim=1)}


def _evolved(apply, psi, t, norm):
    """exp(-i H t) psi by a Taylor series over substeps of norm * h <= 1."""
    n = max(1, math.ceil(abs(t) * norm))
    for _ in range(n):
        term = psi
        for j in range(1, 26):
            term = apply(term) * (-1j * t / n / j)
            psi = psi + term
    return psi


def _exact_quench(c, seed):
    s = prepare(c, seed)
    model = s["model"]
    mat = model.H.mat
    apply, _ = _matrix(mat)
    rows = torch.repeat_interleave(torch.arange(mat.n, device="cuda"), mat.rowptr[1:] - mat.rowptr[:-1])
    mod = mat.vals.view(torch.complex128).abs() if mat.is_complex else mat.vals.abs()
    norm = torch.zeros(mat.n, dtype=torch.float64, device="cuda").index_add_(0, rows, mod)
    shift = _vacuum_energy(mat)
    dg = (mat.diag.view(torch.complex128).real if mat.is_complex else mat.diag) - shift
    norm = float((norm + dg.abs()).max())
    del rows, mod, dg
    # exp(-iHt) = exp(-i shift t) exp(-i (H - shift) t)
    moved = lambda x: apply(x) - shift * x  # noqa: E731
    ph = _gauge(model)
    x = torch.from_numpy(s["psi"]).cuda()
    x = x if ph is None else ph.conj() * x
    states = [x]
    for k in range(1, len(s["times"])):
        dt = float(s["times"][k] - s["times"][k - 1])
        states.append(_evolved(moved, states[-1], dt, norm) * complex(math.cos(shift * dt), -math.sin(shift * dt)))
    if c["keep"]:
        return {"states": torch.stack([y if ph is None else ph * y for y in states])}
    digits = _digits(model)
    out = {}
    for name, op in s["obs"].items():
        out[name] = np.array([_site_sums(y.abs() ** 2, op, digits) for y in states])
    return out


def _vacuum_energy(mat):
    d = mat.diag.view(torch.complex128).real if mat.is_complex else mat.diag
    return float(d.median())


def _site_values(op, digits):
    d = torch.from_numpy(np.real(np.array([np.diagonal(o) for o in op])).copy()).cuda()
    return [d[s][digits[s]] for s in range(len(digits))]


def _site_sums(p, op, digits):
    return np.array([float((p * v).sum()) for v in _site_values(op, digits)])


def _exact_observe(c, seed):
    s = prepare(c, seed)
    model, digits = s["model"], _digits(s["model"])
    p = s["psi"].to(torch.complex128).abs() ** 2
    out = {k: _site_sums(p, model.ops[k], digits) for k in _LOCAL}
    n = len(digits)
    for a, b in _TWOBODY:
        va, vb = _site_values(model.ops[a], digits), _site_values(model.ops[b], digits)
        corr = np.zeros((n, n))
        for i in range(n):
            pi = p * va[i]
            for j in range(i + 1, n):
                corr[i, j] = corr[j, i] = float((pi * vb[j]).sum())
        out[f"{a}_{b}"] = corr
    return out


def _exact_batch(c, seed):
    return {"energies": np.array([_eigen(m, 1)[0] for m in _batch_matrices(c, seed)])}


def _exact_momentum(c, seed):
    """The lowest energy of H on the vectors with T psi = exp(i 2 pi k / L)
    psi: Lanczos in the whole sector from a projected start vector, projected
    again after every product."""
    s = prepare(c, seed)
    model, lx = s["model"], c["lx"]
    mat = _build(model, c, *s["coupling"])
    apply, _ = _matrix(mat)
    ph = _gauge(model)
    digits = _digits(model)
    d = [int(x) for x in model.loc_dims]
    moved = torch.zeros_like(model.sector.keys)
    for site in range(lx):
        moved = moved * d[site] + digits[site - 1]
    image = torch.searchsorted(model.sector.keys, moved)

    def project(x):
        y, z = x.clone(), x
        for t in range(1, lx):
            shifted = torch.empty_like(z)
            shifted[image] = z
            z = shifted
            y = y + z * complex(np.exp(-2j * np.pi * c["kx"] * t / lx))
        return y / lx

    def h(x):
        y = apply(x if ph is None else ph.conj() * x)
        return project(y if ph is None else ph * y)

    gen = torch.Generator(device="cuda").manual_seed(7)
    start = project(torch.randn(mat.n, dtype=torch.complex128, device="cuda", generator=gen))
    e, _ = _lowest(h, mat.n, 1, torch.complex128, start, most=300)
    return {"energy": e / model.n_sites, "col_ptr": None, "row_idx": None, "data": None}


# ------------------------------------------- a plain Z_n Hamiltonian (exact)
class _PlainZn:
    """H of the Z_n model on zero-momentum representatives: every image is
    translated through the group, the smallest key found among the
    representatives by a search, amplitudes sqrt(|Stab r'| / |Stab r|)."""

    def __init__(self, lx, ly, zn, lb, keys):
        self.lx, self.ly, self.zn, self.lb, self.keys = lx, ly, zn, lb, keys
        self.n = lx * ly
        self.bits = 2 * lb * self.n
        self.sorted, self.order = torch.sort(keys)
        occ = np.arange(1 << self.n)
        bit = [(occ >> s) & 1 for s in range(self.n)]
        lane = 2 * lb * lx
        lanes = np.arange(1 << lane)
        self.group = []
        for a in range(0, lx, 2):
            turned = np.zeros_like(lanes)
            for x in range(lx):
                field = (lanes >> (2 * lb * x)) & ((1 << (2 * lb)) - 1)
                turned |= field << (2 * lb * ((x + a) % lx))
            for b in range(ly):
                to = [(s % lx + a) % lx + lx * ((s // lx + b) % ly) for s in range(self.n)]
                new = sum(bit[s] << to[s] for s in range(self.n))
                sign = np.zeros_like(occ)
                for s in range(self.n):
                    for t in range(s + 1, self.n):
                        if to[s] > to[t]:
                            sign ^= bit[s] & bit[t]
                self.group.append((torch.from_numpy(turned).cuda(), b, torch.from_numpy(new).cuda(),
                                   torch.from_numpy(sign).cuda()))
        self.stab = self._reduced(keys)[2]

    def _reduced(self, k):
        """(smallest key of the orbit, sign of the translation to it, size of
        the stabiliser, whether a translation maps the state to minus itself)."""
        lane = 2 * self.lb * self.lx
        occ = k >> self.bits
        best, sign = k.clone(), torch.zeros_like(k)
        stab, odd = torch.zeros_like(k), torch.zeros_like(k, dtype=torch.bool)
        for turned, b, new, sg in self.group:
            im = new[occ] << self.bits
            for y in range(self.ly):
                im |= turned[(k >> (lane * y)) & ((1 << lane) - 1)] << (lane * ((y + b) % self.ly))
            s = sg[occ]
            less = im < best
            sign = torch.where(less, s, sign)
            best = torch.where(less, im, best)
            same = im == k
            stab += same
            odd |= same & (s != 0)
        return best, sign, stab, odd

    def _field(self, k, l):
        return (k >> (self.lb * l)) & ((1 << self.lb) - 1)

    def _step(self, k, l, up):
        f = self._field(k, l)
        return k + ((torch.remainder(f + up, self.zn) - f) << (self.lb * l))

    def apply(self, x, coup, chunk=1 << 24):
        """coup: (t, m, g^2/2, -1/(2 g^2)) of every column of x."""
        y = torch.empty(x.shape, dtype=torch.float64, device="cuda")
        for r0 in range(0, len(self.keys), chunk):
            y[r0:r0 + chunk] = self._rows(x, coup, slice(r0, min(r0 + chunk, len(self.keys))))
        return y

    def _image(self, x, k2, live, amp, rows):
        best, sign, _, odd = self._reduced(k2)
        at = torch.searchsorted(self.sorted, best).clamp_(max=len(self.sorted) - 1)
        live = live & ~odd & (self.sorted[at] == best)
        at = self.order[at]
        f = torch.sqrt(self.stab[at].double() / self.stab[rows].double())
        f = torch.where(live, f * amp * (1 - 2 * sign), torch.zeros_like(f))
        return f[:, None] * x[at].double()

    def _rows(self, x, coup, rows):
        k = self.keys[rows]
        occ = k >> self.bits
        hop = torch.zeros((len(k), x.shape[1]), dtype=torch.float64, device="cuda")
        plaq = torch.zeros_like(hop)
        esq = torch.zeros(len(k), dtype=torch.float64, device="cuda")
        mass = torch.zeros_like(esq)
        sites = [(s % self.lx, s // self.lx) for s in range(self.n)]
        at = lambda px, py: px % self.lx + self.lx * (py % self.ly)  # noqa: E731
        for s, (px, py) in enumerate(sites):
            mass += (1 - 2 * (px % 2)) * ((occ >> s) & 1)
            for mu in (0, 1):
                l, t = 2 * s + mu, at(px + 1 - mu, py + mu)
                f = self._field(k, l).double()
                esq += torch.where(f > self.zn // 2, f - self.zn, f) ** 2
                # c^dag_s U c_t where s is empty, its conjugate where t is
                ns, nt = (occ >> s) & 1, (occ >> t) & 1
                k2 = torch.where(ns == 0, self._step(k, l, 1), self._step(k, l, -1))
                k2 = k2 ^ (((1 << s) | (1 << t)) << self.bits)
                between = sum(((occ >> q) & 1) for q in range(min(s, t) + 1, max(s, t))) if abs(s - t) > 1 else 0
                eta = 1 if mu == 0 or px % 2 == 0 else -1
                amp = eta * (1.0 - 2.0 * ((torch.zeros_like(k) + between) % 2))
                hop += self._image(x, k2, ns != nt, amp, rows)
            loop = [2 * s, 2 * at(px + 1, py) + 1, 2 * at(px, py + 1), 2 * s + 1]
            for up in (1, -1):
                k2 = k
                for l, w in zip(loop, (up, up, -up, -up)):
                    k2 = self._step(k2, l, w)
                plaq += self._image(x, k2, torch.ones_like(k, dtype=torch.bool), 1.0, rows)
        d = esq[:, None] * coup[:, 2] + mass[:, None] * coup[:, 1]
        return d * x[rows].double() - coup[:, 0] * hop + coup[:, 3] * plaq


def _plain_zn(model):
    L = model.lattice
    return _PlainZn(L.lx, L.ly, L.n, L.link_bits, model.engine.keys[: model.sector_dim])


def _exact_zn_apply(c, seed):
    s = prepare(c, seed)
    return {"y": _plain_zn(s["model"]).apply(s["x"], s["couplings"])}


def _exact_zn_ground(c, seed):
    s = prepare(c, seed)
    model = s["model"]
    h = _plain_zn(model)
    n = model.sector_dim
    es, vs = [], []
    for row in np.asarray(model.couplings):
        cp = torch.from_numpy(row[None, :].copy()).cuda()
        e, v = _lowest(lambda x: h.apply(x[:, None], cp)[:, 0], n, 1, most=min(300, n))
        es.append(e[0])
        vs.append(v[:, 0] * torch.sign(v[s["vacuum"], 0]))
    return {"energies": np.array(es), "psi": torch.stack(vs, dim=1)}
