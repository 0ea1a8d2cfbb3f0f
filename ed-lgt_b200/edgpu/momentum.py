"""Momentum (translation) sectors on the device.

Mirrors ``QuantumModel.set_momentum_sector`` (edlgt/models/quantum_model.py:
213-276) with ``get_momentum_basis`` and its zero-k / finite-k projectors
(edlgt/symmetries/translational_sym.py:508-949, 1307-1358).  The projector B
(sector rows x momentum states) is built by ``edg_momentum_translations``,
``edg_momentum_references``, ``edg_momentum_columns`` and
``edg_momentum_rowmap``; the reference then assembles B^dagger O B term by
term (``nbody_data_momentum*``, :1394-1969), here H_k = B^dagger H B is
applied without being formed: ``edg_momentum_expand``, the sector matvec,
``edg_momentum_reduce``.  Spectra come from a dense Hermitian solve of H_k
(one kernel) up to ``DENSE_MAX`` momentum states and from
a fully reorthogonalised Lanczos above that.
"""

from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _lib
from ._lib import check, lib, ptr, stream_handle

__all__ = ["MomentumBasis", "translation_sources", "krylov_evolve", "DENSE_MAX"]

DENSE_MAX = 4096
# Sector rows up to which the projector's host arrays are narrowed on the host: a
# small basis pays more for a few device operations than for its bytes (host_arrays
# at 282 rows 0.10 ms so, 0.18 to 0.27 with them; 2,214 rows 0.13, 0.19 to 0.25;
# 17,906 rows 0.29 to 0.32, 0.23 to 0.32; 147,578 rows 1.6 to 1.9, 0.53 to 0.74)
HOST_ROWS = 1 << 14


def translation_sources(lvals, unit_cell):
    """source[s, dest] = site whose local state lands on ``dest`` under the
    block shift s; shifts and sites both enumerated row-major (first axis
    slowest), as _prepare_translation_source_sites
    (translational_sym.py:508-560)."""
    lvals = np.asarray(lvals, dtype=np.int64)
    ucs = np.asarray(unit_cell, dtype=np.int64)
    if lvals.shape != ucs.shape or np.any(ucs < 1) or np.any(lvals % ucs):
        raise ValueError("unit cell sizes must divide the lattice lengths, one per axis")
    R = lvals // ucs
    n_sites = int(np.prod(lvals))
    coords = np.stack(np.unravel_index(np.arange(n_sites), tuple(lvals)), axis=1)
    n_shifts = int(np.prod(R))
    src = np.empty((n_shifts, n_sites), dtype=np.int32)
    for s in range(n_shifts):
        t = np.array(np.unravel_index(s, tuple(R)))
        dest = np.ravel_multi_index(tuple(((coords + t * ucs) % lvals).T), tuple(lvals))
        src[s, dest] = np.arange(n_sites)
    return src, R.astype(np.int32)


def _phase_table(k_vals, R):
    """exp(-2 pi i k_d t / R_d) by repeated products, [dim][max R]
    (_prepare_phase_table, translational_sym.py:344-365)."""
    D, max_r = len(R), int(np.max(R))
    tab = np.zeros((D, max_r), dtype=np.complex128)
    for d in range(D):
        tab[d, 0] = 1.0
        if R[d] <= 1:
            continue
        step = np.exp(-1j * 2.0 * np.pi * (int(k_vals[d]) % int(R[d])) / float(R[d]))
        for t in range(1, int(R[d])):
            tab[d, t] = tab[d, t - 1] * step
    return tab


class MomentumBasis:
    """The projector B of one momentum sector, on the device."""

    def __init__(self, sector, lvals, unit_cell, k_vals, local_map=None, label_sign=None):
        """``local_map`` / ``label_sign``: the translation-charge variant (1D,
        unit cell 1): the local map applied with every unit shift and the
        per-state signs whose product twists the odd shifts."""
        sector.require_narrow("momentum basis")
        dev = sector.device
        self.sector = sector
        self.device = dev
        n = len(sector)
        src, R = translation_sources(lvals, unit_cell)
        tc = local_map is not None
        if tc and (len(R) != 1 or src.shape[0] != src.shape[1]):
            raise ValueError("the translation-charge basis is defined on a 1D ring with a one-site unit cell")
        k_vals = np.asarray(k_vals, dtype=np.int64).reshape(-1)
        if len(k_vals) != len(R):
            raise ValueError(f"expected {len(R)} momentum labels, got {len(k_vals)}")
        if len(R) > 3:
            raise ValueError("momentum sectors support 1 to 3 lattice dimensions")
        n_shifts = src.shape[0]
        self.n_rows = n
        self.zero_k = not np.any(k_vals != 0)
        g = _lib.MomentumGroup()
        g.lattice_dim = len(R)
        g.n_shifts = n_shifts
        stride = 1
        for d in range(len(R) - 1, -1, -1):
            g.shifts_per_dir[d] = int(R[d])
            g.shift_strides[d] = stride
            g.k_vals[d] = int(k_vals[d])
            stride *= int(R[d])
        self.group = g
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        src_d = up(src)
        strides = up(sector.strides.astype(np.int64))
        loc = up(sector.loc_dims.astype(np.int32))
        flag = torch.zeros(1, dtype=torch.int32, device=dev)
        trans = torch.empty((max(n, 1), n_shifts), dtype=torch.int32, device=dev)
        if tc:
            cmap = up(np.asarray(local_map, dtype=np.int32))
            lsign = up(np.asarray(label_sign, dtype=np.float64))
            row_sign = torch.empty(max(n, 1), dtype=torch.float64, device=dev)
            map_args = (ptr(cmap), int(cmap.shape[0]), ptr(lsign), ptr(row_sign))
        else:
            row_sign = None
            map_args = (None, 0, None, None)
        check(lib.edg_momentum_translations(sector.lookup_table(), ptr(strides), ptr(loc), int(sector.n_sites),
                                            ptr(src_d), n_shifts, *map_args, ptr(trans), ptr(flag), stream_handle()),
              "edg_momentum_translations")
        rs = ptr(row_sign) if tc else None
        ns = lib.edg_momentum_scratch_elems(n)
        scratch = torch.empty(max(ns, 1), dtype=torch.int64, device=dev)
        pvec = torch.empty((max(n, 1), len(R)), dtype=torch.int32, device=dev)
        refs = torch.empty(max(n, 1), dtype=torch.int64, device=dev)
        n_cols = ctypes.c_int64(0)
        check(lib.edg_momentum_references(ptr(trans), n, ctypes.byref(g), ptr(pvec), ptr(refs), ctypes.byref(n_cols),
                                          ptr(scratch), ns, stream_handle()), "edg_momentum_references")
        m = int(n_cols.value)
        self.n_cols = m
        tab = up(_phase_table(k_vals, R))
        col_ptr = torch.empty(m + 1, dtype=torch.int64, device=dev)
        nnz = ctypes.c_int64(0)
        cs = lib.edg_scan_scratch_elems(m)
        cscratch = torch.empty(max(cs, 1), dtype=torch.int64, device=dev)
        zk = 1 if self.zero_k else 0
        check(lib.edg_momentum_columns(ptr(trans), ptr(refs), m, ptr(pvec), ctypes.byref(g), ptr(tab), tab.shape[1],
                                       zk, rs, ptr(col_ptr), ctypes.byref(nnz), None, None, ptr(cscratch), cs,
                                       stream_handle()), "edg_momentum_columns")
        self.nnz = int(nnz.value)
        row_idx = torch.empty(max(self.nnz, 1), dtype=torch.int32, device=dev)
        data = torch.empty(max(self.nnz, 1), dtype=torch.complex128, device=dev)
        check(lib.edg_momentum_columns(ptr(trans), ptr(refs), m, ptr(pvec), ctypes.byref(g), ptr(tab), tab.shape[1],
                                       zk, rs, ptr(col_ptr), ctypes.byref(nnz), ptr(row_idx), ptr(data),
                                       ptr(cscratch), cs, stream_handle()), "edg_momentum_columns")
        row_col = torch.empty(max(n, 1), dtype=torch.int64, device=dev)
        row_val = torch.empty(max(n, 1), dtype=torch.complex128, device=dev)
        check(lib.edg_momentum_rowmap(ptr(col_ptr), ptr(row_idx), ptr(data), m, n, ptr(row_col), ptr(row_val),
                                      ptr(flag), stream_handle()), "edg_momentum_rowmap")
        self.col_ptr, self.row_idx, self.data = col_ptr, row_idx, data
        self.row_col, self.row_val = row_col, row_val
        self.refs = refs[:m]
        self._bound = None

    # ------------------------------------------------------------ host view
    def host_arrays(self) -> dict:
        """The reference's momentum_basis dict (CSC and CSR of B, host)."""
        cp, ri = self.col_ptr, self.row_idx[: self.nnz]
        dv, rv, rc = self.data[: self.nnz], self.row_val[: self.n_rows], self.row_col[: self.n_rows]
        if self.n_rows <= HOST_ROWS:
            cp, ri, dv, rv, rc = (x.cpu().numpy() for x in (cp, ri, dv, rv, rc))
            has = rc >= 0
            r_ptr = np.zeros(self.n_rows + 1, dtype=np.int32)
            np.cumsum(has, out=r_ptr[1:])
            rv, rc = rv[has], rc[has].astype(np.int32)
            if self.zero_k:
                dv, rv = dv.real.copy(), rv.real.copy()
            cp, ri = cp.astype(np.int32), ri.astype(np.int32, copy=False)
        else:
            # narrowed on the device: half the bytes to copy, no pass over them here
            has = rc >= 0
            r_ptr = torch.zeros(self.n_rows + 1, dtype=torch.int32, device=self.device)
            torch.cumsum(has, 0, dtype=torch.int32, out=r_ptr[1:])
            if self.nnz < self.n_rows:
                rv, rc = rv[has], rc[has]
            if self.zero_k:
                dv, rv = dv.real, rv.real
            cp, ri, dv, r_ptr, rc, rv = (x.cpu().numpy() for x in (
                cp.to(torch.int32), ri, dv.contiguous(), r_ptr, rc.to(torch.int32), rv.contiguous()))
        return {"pair_mode": False, "n_rows": self.n_rows, "n_cols": self.n_cols, "L_col_ptr": cp,
                "L_row_idx": ri, "L_data": dv, "R_row_ptr": r_ptr, "R_col_idx": rc, "R_data": rv}

    # ------------------------------------------------------------ operator
    def bind(self, ham):
        """Attach the sector Hamiltonian (``QMB_hamiltonian`` with a built
        matrix); a real-form matrix gets its gauge phases folded into B."""
        mat = ham.mat
        ph = ham._row_phase()
        if ph is None:
            rv, dv = self.row_val, self.data
        else:
            rv = torch.conj(ph) * self.row_val[: self.n_rows]
            rows = self.row_idx[: self.nnz].to(torch.int64)
            dv = torch.conj(ph[rows]) * self.data[: self.nnz] if self.nnz else self.data
        # a complex vector on a real matrix runs as two interleaved real
        # right-hand sides, whose diagonals the batched matvec reads per side
        diag = mat.diag if mat.is_complex else mat.diag.repeat_interleave(2).contiguous()
        self._bound = (mat, rv.contiguous(), dv.contiguous(), diag)

    def matvec(self, x: torch.Tensor) -> torch.Tensor:
        """y = B^dagger H B x for a complex128 momentum-space vector."""
        x = x.to(torch.complex128).contiguous()
        return self._product()(ptr(x))

    def _product(self):
        """A function of a vector's address that returns H_k times it, on this
        stream, in buffers made once: each call overwrites the result of the
        one before."""
        mat, rv, dv, diag = self._bound
        v = torch.empty(self.n_rows, dtype=torch.complex128, device=self.device)
        w = torch.empty_like(v)
        y = torch.empty(self.n_cols, dtype=torch.complex128, device=self.device)
        # on a real matrix a complex vector is two interleaved real ones
        code, nvec = (2, 1) if mat.is_complex else (0, 2)
        st = stream_handle()
        expand = (self.n_rows, ptr(self.row_col), ptr(rv))
        spmv = (code, mat.n, mat.nnz, ptr(mat.rowptr), ptr(mat.cols) if mat.nnz else None,
                ptr(mat.vals) if mat.nnz else None, ptr(diag), nvec, ptr(v), ptr(w), st)
        reduce = (self.n_cols, ptr(self.col_ptr), ptr(self.row_idx), ptr(dv), ptr(w), ptr(y), st)

        def apply(x, _alive=(mat, rv, dv, diag, v, w)):  # the tensors behind the addresses
            check(lib.edg_momentum_expand(*expand, x, spmv[8], st), "edg_momentum_expand")
            check(lib.edg_spmv(*spmv), "edg_spmv")
            check(lib.edg_momentum_reduce(*reduce), "edg_momentum_reduce")
            return y

        return apply

    def dense(self) -> torch.Tensor:
        """H_k as a dense (n_cols, n_cols) complex128 matrix
        (``edg_momentum_dense``)."""
        mat, rv, dv, _ = self._bound
        m = self.n_cols
        out = torch.empty((m, m), dtype=torch.complex128, device=self.device)
        check(lib.edg_momentum_dense(m, ptr(self.col_ptr), ptr(self.row_idx), ptr(dv), ptr(self.row_col), ptr(rv),
                                     1 if mat.is_complex else 0, ptr(mat.rowptr), ptr(mat.cols) if mat.nnz else None,
                                     ptr(mat.vals) if mat.nnz else None, ptr(mat.diag), ptr(out), stream_handle()),
              "edg_momentum_dense")
        return out

    def lowest(self, k, tol=1e-12, max_iter=None, seed=0):
        """(energies, vectors [n_cols, k]) of H_k, ascending."""
        m = self.n_cols
        if m == 0:
            raise ValueError("the momentum sector is empty")
        if k > m:
            raise ValueError(f"n_eigs must be <= {m}")
        if m <= DENSE_MAX:
            h = self.dense()
            h = 0.5 * (h + h.conj().T)
            w, v = torch.linalg.eigh(h)
            self.last_matvecs = m
            return w[:k].cpu().numpy(), v[:, :k]
        w, v, its = _lanczos(self._product(), m, k, tol, max_iter or min(m, 400), self.device, seed)
        self.last_matvecs = its
        return w, v


def krylov_evolve(apply, psi0, time_line, m_krylov=40, tol=1e-12):
    """psi(t) = exp(-i H t) psi0 at every (absolute) time of ``time_line``, the
    role of expm_multiply in QMB_hamiltonian.time_evolution
    (edlgt/modeling/qmb_hamiltonian.py:370-384): each interval is covered by
    Lanczos-exponential steps whose size halves until the a-posteriori error
    estimate beta_m |[exp(-i T dt)]_{m-1,0}| is at most ``tol``."""
    from scipy.linalg import expm

    time_line = np.asarray(time_line, dtype=np.float64)
    if len(time_line) == 0 or time_line[0] < 0 or np.any(np.diff(time_line) < 0):
        raise ValueError("time_line must be ascending and start at t >= 0")
    psi = psi0.to(torch.complex128).clone()
    n = psi.shape[0]
    m_k = max(1, min(m_krylov, n))
    out = []
    t_prev = 0.0  # expm_multiply returns exp(-i H t) psi0 at the absolute times
    dt_try = None
    for t in time_line:
        remaining = float(t) - t_prev
        while remaining > 0:
            nrm = float(torch.linalg.vector_norm(psi))
            if nrm == 0.0:
                break
            V = torch.empty((m_k + 1, n), dtype=torch.complex128, device=psi.device)
            V[0] = psi / nrm
            a, b = [], []
            j_used = m_k
            for j in range(m_k):
                w = apply(V[j])
                a.append(float(torch.vdot(V[j], w).real))
                for _ in range(2):
                    w = w - V[: j + 1].T @ (V[: j + 1].conj() @ w)
                bj = float(torch.linalg.vector_norm(w))
                b.append(bj)
                if bj <= 1e-14 * max(1.0, abs(a[-1])):
                    j_used = j + 1
                    break
                V[j + 1] = w / bj
            T = np.diag(a[:j_used]) + np.diag(b[: j_used - 1], 1) + np.diag(b[: j_used - 1], -1)
            dt = remaining if dt_try is None else min(remaining, dt_try)
            while True:
                E = expm(-1j * dt * T)
                err = (b[j_used - 1] if j_used == m_k else 0.0) * abs(E[j_used - 1, 0]) * nrm
                if err <= tol or dt < 1e-12:
                    break
                dt *= 0.5
            coef = torch.from_numpy(np.ascontiguousarray(E[:, 0] * nrm)).to(psi.device)
            psi = V[:j_used].T @ coef
            remaining -= dt
            dt_try = 2 * dt
        t_prev = float(t)
        out.append(psi.clone())
    return out


def _lanczos(apply, m, k, tol, max_iter, device, seed):
    """Lanczos with two classical Gram-Schmidt passes against the whole basis
    on complex128 vectors (``edg_krylov_orth``); converged when every wanted
    Ritz pair has |beta_j s_jk| <= tol max(1, |theta_k|).  The host reads the
    coefficients when it tests for convergence, every fifth to twentieth step."""
    from scipy.linalg import eigh_tridiagonal

    max_iter = min(max_iter, 14000)  # the most basis vectors edg_krylov_orth takes
    gen = torch.Generator(device=device).manual_seed(seed)
    q = torch.randn(m, dtype=torch.complex128, device=device, generator=gen)
    Q = torch.empty((max_iter + 1, m), dtype=torch.complex128, device=device)  # unnormalised: |Q[i]| = beta[i]
    torch.div(q, torch.linalg.vector_norm(q), out=Q[0])
    coef = torch.zeros((2, max_iter + 1), dtype=torch.float64, device=device)  # alpha, beta
    coef[1, 0] = 1.0
    wb = lib.edg_krylov_orth_bytes(max_iter)
    work = torch.empty(wb, dtype=torch.uint8, device=device)
    step = (ptr(coef[0]), ptr(coef[1]), max_iter, ptr(work), wb, stream_handle())
    q0 = Q.data_ptr()
    theta = s = None
    next_check, last = 5 * ((k + 4) // 5), None
    for j in range(max_iter):
        w = apply(q0 + 16 * m * j)
        check(lib.edg_krylov_orth(m, m, q0, j, ptr(w), 2, *step), "edg_krylov_orth")
        done = j + 1 == max_iter
        if j + 1 >= k and (done or j + 1 >= next_check):
            alpha, beta = coef[:, : j + 2].cpu().numpy()
            n = j + 1
            # a breakdown, once k steps are taken, ends the recurrence at its step
            ends = np.nonzero(beta[k: n + 1] <= 1e-14 * np.maximum(1.0, np.abs(alpha[k - 1: n])))[0]
            if len(ends):
                n, done = k + int(ends[0]), True
            if not np.all(beta[:n] > 0):
                raise ValueError(f"the start vector spans fewer than {k} states of the momentum sector")
            theta, s = eigh_tridiagonal(alpha[:n], beta[1:n], select="i", select_range=(0, k - 1))
            res = np.abs(beta[n] * s[-1, :])
            if done or np.all(res <= tol * np.maximum(1.0, np.abs(theta))):
                break
            # the next check where the contraction so far reaches the tolerance,
            # less a fifth: a read stops the device for about 0.1 ms
            worst, wait = float(np.max(res / np.maximum(1.0, np.abs(theta)))), 5
            if last is not None and 0.0 < worst < last[1] and tol > 0.0:
                need = np.log(tol / worst) * (n - last[0]) / np.log(worst / last[1])
                wait = 5 * int(min(4, max(1, 0.8 * need // 5)))
            next_check, last = n + wait, (n, worst)
    n = s.shape[0]
    vecs = Q[:n].T @ torch.from_numpy((s / beta[:n, None]).astype(np.complex128)).to(device)
    return theta, vecs, n
