"""Device assembly of the sector Hamiltonian from term blocks.

Host side: the term blocks are flattened into local transition tables (the
nonzero entries, ``|op| > 1e-10``, of every site operator used, as
``_prepare_local_transition_data`` does, edlgt/symmetries/
sym_qmb_operations.py:32-92) plus one record per term instance.  The device
builds the canonical matrix (duplicates summed, columns ascending) in three
kernels: per-row entry bounds, generation + per-row merge, compaction.

Real form.  The gauge models' hoppings carry factors ``-i t``; a diagonal
unitary ``D = prod_s phi_s(c_s)`` with ``phi_s(c) = i**(w_s(c))`` (``w`` a
per-site integer weight, typically x-coordinate times matter number) maps
``H`` to ``D^dagger H D``, applied here factor by factor to the site
operators.  When every transformed site table has a single common phase and
every instance's total phase is real, the matrix is assembled real; otherwise
the faithful complex matrix is assembled.  Eigenvalues are unchanged and
eigenvectors map back by ``psi = D psi'``.
"""

from __future__ import annotations

import hashlib

import numpy as np
import torch

from .. import _lib
from .._lib import check, lib, ptr, stream_handle, upload_arrays
from .terms import TermBlock

__all__ = ["DeviceMatrix", "assemble_blocks", "OP_TOL"]

OP_TOL = 1e-10


class DeviceMatrix:
    """Canonical sector matrix: off-diagonal CSR + dense diagonal, on the device.

    ``vals``/``diag`` are float64 tensors (interleaved re/im when ``is_complex``).
    ``diag_present`` marks rows whose (r, r) entry exists in the reference's
    triplet set (a local term with ``|op_cc| >= 1e-10`` or a diagonal hit).
    ``phase_weights`` (n_sites, dmax) integer exponents of ``i`` of the real
    form's gauge transform, or None.
    """

    def __init__(self, n, rowptr, cols, vals, diag, diag_present, is_complex, phase_weights=None):
        self.n = int(n)
        self.rowptr = rowptr
        self.cols = cols
        self.vals = vals
        self.diag = diag
        self.diag_present = diag_present
        self.is_complex = bool(is_complex)
        self.phase_weights = phase_weights
        self.nnz = int(cols.shape[0]) if cols is not None else 0

    @property
    def shape(self):
        return (self.n, self.n)

    def dtype_code(self):
        return 2 if self.is_complex else 0

    def to_scipy(self, include_diag=True):
        """Host canonical CSR (pattern of the reference after summing duplicates)."""
        from scipy.sparse import csr_matrix

        rp = self.rowptr.cpu().numpy()
        cols = self.cols.cpu().numpy()[: self.nnz].astype(np.int64)
        v = self.vals.cpu().numpy()
        d = self.diag.cpu().numpy()
        if self.is_complex:
            v = v.view(np.complex128)[: self.nnz]
            d = d.view(np.complex128)
        else:
            v = v[: self.nnz]
        rows = np.repeat(np.arange(self.n), np.diff(rp))
        if include_diag:
            pres = self.diag_present.cpu().numpy().astype(bool)
            r = np.nonzero(pres)[0]
            rows = np.concatenate([rows, r])
            cols = np.concatenate([cols, r])
            v = np.concatenate([v, d[r]])
            order = np.lexsort((cols, rows))
            rows, cols, v = rows[order], cols[order], v[order]
        indptr = np.zeros(self.n + 1, dtype=np.int64)
        np.add.at(indptr, rows + 1, 1)
        indptr = np.cumsum(indptr)
        return csr_matrix((v, cols, indptr), shape=self.shape)

    def matvec(self, x: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
        """y = H x on the device (x: float64 or complex128 tensor of length n)."""
        if self.is_complex:
            x = x.to(torch.complex128)
            code = 2
        else:
            if x.is_complex():
                raise TypeError("real matrix: use a real vector (or apply to real and imaginary parts)")
            x = x.to(torch.float64)
            code = 0
        y = torch.empty_like(x) if out is None else out
        check(lib.edg_spmv(code, self.n, self.nnz, ptr(self.rowptr), ptr(self.cols) if self.nnz else None,
                           ptr(self.vals) if self.nnz else None, ptr(self.diag), 1, ptr(x), ptr(y), stream_handle()),
              "edg_spmv")
        return y


def _uniform_phase(mat, tol=1e-12):
    """Common phase e^{i theta} of all entries above OP_TOL, or None."""
    nz = mat[np.abs(mat) > OP_TOL]
    if nz.size == 0:
        return 1.0 + 0.0j
    ph = nz[np.argmax(np.abs(nz))]
    ph = ph / abs(ph)
    rot = nz / ph
    if np.all(np.abs(rot.imag) <= tol * np.maximum(1.0, np.abs(rot))):
        return ph
    return None


def _phase_vec(weights_row):
    return np.power(1j, np.asarray(weights_row, dtype=np.int64) % 4)


def _nonzero(m):
    """np.nonzero of a complex array (several times faster than testing the
    complex values)."""
    return np.nonzero((m.real != 0) | (m.imag != 0))


def _offdiag_signature(blocks, phase_weights, force_complex, dmax):
    """Content hash of everything the off-diagonal part of the matrix depends
    on: the off-diagonal blocks' operators, instances, strengths and h.c.
    flags, the real form's phase weights and the form request."""
    h = hashlib.sha256(repr((bool(force_complex), int(dmax))).encode())
    if phase_weights is not None:
        h.update(np.ascontiguousarray(np.asarray(phase_weights, dtype=np.int64)).tobytes())
    for b in blocks:
        if b.diagonal:
            continue
        h.update(repr((b.strength, b.add_dagger, len(b.ops))).encode())
        h.update(np.ascontiguousarray(b.sites).tobytes())
        for o in b.ops:
            o = np.ascontiguousarray(o)
            h.update(repr((str(o.dtype), o.shape)).encode())
            h.update(o.tobytes())
    return h.hexdigest()


def _offdiag_tables(blocks, phase_weights, force_complex, dmax):
    """Local transition tables and instance records of the off-diagonal
    blocks, and whether they admit the real form (every gauge-transformed
    table has one common phase and every instance's total phase is real)."""
    keys = []  # (block, factor, site, conjugated) of every table
    index = {}
    terms = []  # (sites tuple, tables tuple, coef)
    for bi, b in enumerate(blocks):
        if b.diagonal:
            continue
        sites = b.sites.tolist()
        for dag in ([False, True] if b.add_dagger else [False]):
            coef = complex(np.conj(b.strength) if dag else b.strength)
            for inst in sites:
                tabs = []
                for j, s in enumerate(inst):
                    key = (bi, j, s, dag)
                    t = index.get(key)
                    if t is None:
                        t = index[key] = len(keys)
                        keys.append(key)
                    tabs.append(t)
                if len(set(inst)) != len(inst):
                    raise ValueError("a term instance acts twice on the same site")
                terms.append((tuple(inst), tuple(tabs), coef))
    table_site = [k[2] for k in keys]
    raw_tables = np.zeros((len(keys),) + (() if not keys else blocks[keys[0][0]].ops[0].shape[-2:]),
                          dtype=np.complex128)
    same = {}  # tables that come from one operator: one gather
    for t, (bi, j, s, dag) in enumerate(keys):
        same.setdefault((bi, j, dag), ([], []))
        same[bi, j, dag][0].append(t)
        same[bi, j, dag][1].append(s)
    for (bi, j, dag), (ts, ss) in same.items():
        m = np.asarray(blocks[bi].ops[j])[ss]
        raw_tables[ts] = m.conj().transpose(0, 2, 1) if dag else m
    real_ok, tables_real, coefs_real = False, None, None
    if not force_complex and len(raw_tables):
        # every table at once, on its nonzero entries: gauge-transform, then the
        # table's common phase (the phase of its largest entry above OP_TOL,
        # the first in row-major order), as _uniform_phase does table by table
        nt, d = raw_tables.shape[:2]
        ti, bi, ki = _nonzero(raw_tables)
        v = raw_tables[ti, bi, ki]
        if phase_weights is not None:
            phi = _phase_vec(np.asarray(phase_weights)[np.asarray(table_site)])  # (nt, d)
            v = np.conj(phi)[ti, bi] * v * phi[ti, ki]
        mag = np.abs(v)
        keep = mag > OP_TOL
        big_at = np.zeros((nt, d * d))
        big_at[ti, bi * d + ki] = np.where(keep, mag, 0.0)
        first = big_at.argmax(axis=1)
        full = np.zeros((nt, d * d), dtype=np.complex128)
        full[ti, bi * d + ki] = v
        big = np.where(big_at[np.arange(nt), first] > 0.0, full[np.arange(nt), first], 0.0)
        ph = np.where(big == 0, 1.0 + 0.0j, big / np.where(big == 0, 1.0, np.abs(big)))
        v = v / ph[ti]
        bad = keep & (np.abs(v.imag) > 1e-12 * np.maximum(1.0, np.abs(v)))
        ok = not bad.any()
        if ok:
            tabs_t = np.zeros((nt, d, d))
            tabs_t[ti, bi, ki] = v.real
            phases = ph.tolist()
        if ok:
            cr = []
            for sites, tabs, coef in terms:
                z = coef
                for t in tabs:
                    z *= phases[t]
                if abs(z.imag) > 1e-12 * max(1.0, abs(z)):
                    ok = False
                    break
                cr.append(z.real)
        if ok:
            real_ok, tables_real, coefs_real = True, tabs_t, cr
    return raw_tables, terms, real_ok, tables_real, coefs_real


def _table_arrays(raw_tables, terms, dmax, is_complex, tables_real, coefs_real):
    """Device table arrays: per table and bra the kets whose |amplitude| >
    OP_TOL in ascending order (t_count, t_ket, t_amp, zero beyond the
    count), and the instance records (term_nops, term_site, term_table,
    term_coef).  Vectorised over all tables at once."""
    nt = max(len(raw_tables), 1)
    t_count = np.zeros((nt, dmax), dtype=np.int32)
    t_ket = np.zeros((nt, dmax, dmax), dtype=np.uint8)
    t_amp = np.zeros((nt, dmax, dmax, 2 if is_complex else 1), dtype=np.float64)
    if len(raw_tables):
        raw = np.asarray(raw_tables)[:, :dmax, :dmax]
        ti, bi, ki = _nonzero(raw)
        on = np.abs(raw[ti, bi, ki]) > OP_TOL
        ti, bi, ki = ti[on], bi[on], ki[on]
        v = raw[ti, bi, ki] if is_complex else np.asarray(tables_real)[ti, bi, ki]
        # kets of a bra are neighbours and ascending: their positions count up
        # from the bra's first one
        row = ti * dmax + bi
        cnt = np.bincount(row, minlength=nt * dmax)
        pos = np.arange(len(row)) - (np.cumsum(cnt) - cnt)[row]
        t_count[:] = cnt.reshape(nt, dmax)
        t_ket[ti, bi, pos] = ki
        t_amp[ti, bi, pos, 0] = v.real
        if is_complex:
            t_amp[ti, bi, pos, 1] = v.imag
    n_terms = len(terms)
    term_nops = np.zeros(max(n_terms, 1), dtype=np.int32)
    term_site = np.zeros((max(n_terms, 1), _lib.MAX_OPS), dtype=np.int32)
    term_table = np.zeros((max(n_terms, 1), _lib.MAX_OPS), dtype=np.int32)
    term_coef = np.zeros((max(n_terms, 1), 2 if is_complex else 1), dtype=np.float64)
    by_nops = {}  # instances with the same number of factors: one assignment
    for k_, (sites, _, _) in enumerate(terms):
        by_nops.setdefault(len(sites), []).append(k_)
    for nops, rows in by_nops.items():
        if nops > _lib.MAX_OPS:
            raise ValueError(f"at most {_lib.MAX_OPS} operator factors per term instance")
        term_nops[rows] = nops
        term_site[rows, :nops] = [terms[k_][0] for k_ in rows]
        term_table[rows, :nops] = [terms[k_][1] for k_ in rows]
    if n_terms:
        if is_complex:
            c = np.array([t[2] for t in terms], dtype=np.complex128)
            term_coef[:n_terms, 0], term_coef[:n_terms, 1] = c.real, c.imag
        else:
            term_coef[:n_terms, 0] = coefs_real
    return [t_count, t_ket, t_amp, term_nops, term_site, term_table, term_coef]


def assemble_blocks(sector, blocks, phase_weights=None, force_complex=False, extra_diag=None):
    """Assemble the canonical matrix of ``sum(blocks)`` in ``sector``.

    ``extra_diag``: optional constant added to every diagonal element (identity
    terms).  Returns a :class:`DeviceMatrix`.

    The off-diagonal part (CSR plus the diagonal contributions of instances
    that map a state to itself) depends only on the off-diagonal blocks, the
    phase weights and the form; the sector keeps the last one built, and a
    build whose off-diagonal blocks hash to the same content (a coupling
    sweep that changes diagonal terms only) reuses it and computes only the
    diagonal.
    """
    import ctypes

    loc_dims = sector.loc_dims
    dmax = None
    for b in blocks:
        dmax = b.ops[0].shape[-1] if dmax is None else dmax
    if dmax is None:
        dmax = int(loc_dims.max())
    dev = sector.device
    st = stream_handle()
    n = len(sector)

    # diagonal terms: sites, their operators' diagonals, strengths
    dblocks = [b for b in blocks if b.diagonal and len(b.sites)]
    dsite = np.concatenate([b.sites[:, 0] for b in dblocks]) if dblocks else np.zeros(0, dtype=np.int64)
    ddiag = [np.diagonal(np.asarray(b.ops[0]), axis1=-2, axis2=-1)[b.sites[:, 0]] for b in dblocks]
    dterms_real = all(not np.any(np.abs(v.imag) > 1e-12) and abs(b.strength.imag) <= 1e-12
                      for v, b in zip(ddiag, dblocks))

    # ---- off-diagonal part: reused or built ----
    sig = _offdiag_signature(blocks, phase_weights, force_complex, dmax)
    off = getattr(sector, "_offdiag_cache", None)
    reused = off is not None and off["sig"] == sig and off["use_real"] == (off["real_ok"] and dterms_real)
    keep = []
    if not reused:
        raw_tables, terms, real_ok, tables_real, coefs_real = _offdiag_tables(blocks, phase_weights, force_complex,
                                                                              dmax)
        # instances in the order of their leading sites (stable): a row's
        # columns then come out almost sorted (the fill kernel's insertion)
        order = sorted(range(len(terms)), key=lambda i: min(terms[i][0]))
        terms = [terms[i] for i in order]
        coefs_real = [coefs_real[i] for i in order] if coefs_real is not None else None
        use_real = real_ok and dterms_real
        arrays = _table_arrays(raw_tables, terms, dmax, not use_real, tables_real, coefs_real)
        keep = list(upload_arrays(dev, {k: (a, a.dtype) for k, a in enumerate(arrays)}).values())
        n_tables = arrays[0].shape[0]
        off = _assemble_offdiag(sector, dev, st, n, 1 if use_real else 2, dmax, not use_real, len(terms), n_tables, keep)
        off.update(sig=sig, real_ok=real_ok, use_real=use_real,
                   layouts={"arrays": (off["rowptr"], off["cols"], off["vals"])})
        sector._offdiag_cache = off
    is_complex = not off["use_real"]
    w = 2 if is_complex else 1

    # ---- diagonal terms: one pass over the rows, on top of the off-diagonal
    # part's own diagonal ----
    n_d = len(dsite)
    extra = complex(extra_diag) if extra_diag is not None and extra_diag != 0 else None
    if n == 0 or (n_d == 0 and extra is None):
        diag, present = off["diag"].clone(), off["present"].clone()
    else:
        diag = torch.empty(n * w, dtype=torch.float64, device=dev)
        present = torch.empty(n, dtype=torch.uint8, device=dev)
        a = _assembly_struct(sector, dmax, is_complex)
        a.n_terms = 0
        a.n_dterms = n_d
        if n_d:
            vals = np.zeros((n_d, dmax, w), dtype=np.float64)
            coef = np.zeros((n_d, w), dtype=np.float64)
            at = 0
            for v, b in zip(ddiag, dblocks):
                rows = slice(at, at + len(v))
                vals[rows, : v.shape[1], 0] = v.real
                coef[rows, 0] = b.strength.real
                if is_complex:
                    vals[rows, : v.shape[1], 1] = v.imag
                    coef[rows, 1] = b.strength.imag
                at += len(v)
            dk = upload_arrays(dev, {"site": (dsite, np.int32), "diag": (vals, np.float64),
                                     "coef": (coef, np.float64)})
            keep += dk.values()
            a.dterm_site, a.dterm_diag, a.dterm_coef = ptr(dk["site"]), ptr(dk["diag"]), ptr(dk["coef"])
        ex = extra if extra is not None else 0j
        check(lib.edg_assemble_diag(ctypes.byref(a), ptr(off["diag"]), ptr(off["present"]),
                                    0 if extra is None else 1, ex.real, ex.imag, ptr(diag), ptr(present), st),
              "edg_assemble_diag")
    mat = DeviceMatrix(n, off["rowptr"], off["cols"], off["vals"], diag, present, is_complex,
                       phase_weights if (not is_complex and phase_weights is not None) else None)
    mat._keep = keep  # device tables uploaded by this build
    mat.raw_entries = off["raw_entries"]  # generated entries before the per-row merge
    mat.offdiag_reused = reused  # off-diagonal part shared with an earlier build
    # that part's arrays and their layout, for the matrices that share them
    mat._shared = off["layouts"]
    return mat


def _assembly_struct(sector, dmax, is_complex):
    a = _lib.Assembly()
    a.n_sites = sector.n_sites
    a.dmax = dmax
    for s in range(sector.n_sites):
        a.loc_dims[s] = int(sector.loc_dims[s])
        a.strides[s] = int(sector.strides[s])
    a.sector = sector.lookup_table()
    a.complex_values = 1 if is_complex else 0
    return a


def _assemble_offdiag(sector, dev, st, n, w, dmax, is_complex, n_terms, n_tables, tabs):
    """Off-diagonal instances only: count, scan, fill (with per-row merge)
    and compaction; returns the CSR, the diagonal contributions of
    instances whose ket is the bra, and their presence flags."""
    import ctypes

    a = _assembly_struct(sector, dmax, is_complex)
    a.t_count, a.t_ket, a.t_amp = ptr(tabs[0]), ptr(tabs[1]), ptr(tabs[2])
    a.n_terms = n_terms
    a.term_nops, a.term_site, a.term_table, a.term_coef = ptr(tabs[3]), ptr(tabs[4]), ptr(tabs[5]), ptr(tabs[6])
    a.n_dterms = 0
    bound = torch.empty(max(n, 1), dtype=torch.int64, device=dev)
    check(lib.edg_assemble_count(ctypes.byref(a), ptr(bound), st), "edg_assemble_count")
    offsets = torch.empty(n + 1, dtype=torch.int64, device=dev)
    scratch = torch.empty(lib.edg_scan_scratch_elems(n), dtype=torch.int64, device=dev)
    check(lib.edg_scan_i64(ptr(bound), ptr(offsets), n, ptr(scratch), st), "edg_scan_i64")
    total = int(offsets[n].item())
    cols = torch.empty(max(total, 1), dtype=torch.int32, device=dev)
    vals = torch.empty(max(total, 1) * w, dtype=torch.float64, device=dev)
    row_nnz = torch.empty(max(n, 1), dtype=torch.int64, device=dev)
    diag = torch.empty(max(n, 1) * w, dtype=torch.float64, device=dev)
    present = torch.empty(max(n, 1), dtype=torch.uint8, device=dev)
    flags = torch.zeros(2, dtype=torch.int32, device=dev)
    check(lib.edg_assemble_rows(ctypes.byref(a), n_tables, ptr(offsets), ptr(cols), ptr(vals),
                                ptr(row_nnz), ptr(diag), ptr(present), ptr(flags), st), "edg_assemble_rows")
    e, merged = flags.tolist()
    if e != 0:
        raise _lib.EdgError(e, "an operator maps a sector configuration outside the sector")
    rowptr, nnz = offsets, total
    if merged:  # some rows are shorter than their bound: close the gaps
        tmp_cols, tmp_vals = cols, vals
        rowptr = torch.empty(n + 1, dtype=torch.int64, device=dev)
        check(lib.edg_scan_i64(ptr(row_nnz), ptr(rowptr), n, ptr(scratch), st), "edg_scan_i64")
        nnz = int(rowptr[n].item())
        cols = torch.empty(max(nnz, 1), dtype=torch.int32, device=dev)
        vals = torch.empty(max(nnz, 1) * w, dtype=torch.float64, device=dev)
        check(lib.edg_assemble_compact(n, 1 if is_complex else 0, ptr(offsets), ptr(tmp_cols), ptr(tmp_vals),
                                       ptr(rowptr), ptr(cols), ptr(vals), st), "edg_assemble_compact")
        del tmp_cols, tmp_vals
    return {"rowptr": rowptr, "cols": cols[:nnz], "vals": vals[: nnz * w], "diag": diag[: n * w],
            "present": present[:n], "raw_entries": total, "keep": tabs}
