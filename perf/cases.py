"""Performance cases of the tensor-product-basis Davidson path.

A case names one call of the package's public entry points on a seeded
synthetic system: its orbital number, electrons and strings per spin, and what
is done with it.  Systems, string sets and workload sizes are those of
`sbd_b200.synth` and of the benchmark.

    sigma     one sigma = H C on device vectors (Context.sigma_device), the step
              that every Davidson iteration repeats
    davidson  one cycle of the restarted Davidson (Context.davidson)
    batch     one cycle for several small problems at once (davidson_batch)
    rdm       the 1- and 2-particle RDMs of a state (Context.rdm)
    genmult   the same Hamiltonian as a second-quantised operator applied to a
              device vector (GenOp.mult_device)
    genexpand the expanded basis of a state (GenOp.expand)

`exact` evaluates the same quantities in 64 bits with torch alone, from string
occupations and one-spin operator matrices.
"""
import math
import os
import tempfile

import numpy as np
import torch

import sbd_b200
from sbd_b200 import synth

PRECISION = {"fp64": sbd_b200.FP64, "mixed": sbd_b200.MIXED, "mixed_tc": sbd_b200.MIXED_TC}


def _sigma(name, norb, nea, neb, na, nb, precision="fp64"):
    return {"name": name, "kind": "sigma", "norb": norb, "nea": nea, "neb": neb, "na": na, "nb": nb,
            "precision": precision}


def listed():
    return [
        # the smallest calls: launches and waits are all that counts (the smoke system, a full string space)
        _sigma("sigma_56x56", 8, 3, 3, 56, 56),
        # a full CI space of a small active space, 245,025 determinants
        _sigma("sigma_495x495", 12, 4, 4, 495, 495),
        # an open-shell selected basis: different, odd string counts per spin
        _sigma("sigma_1501x803", 20, 6, 5, 1501, 803),
        # the middle of the range: 16M determinants
        _sigma("sigma_4000x4000", 26, 6, 6, 4000, 4000),
        # the benchmark's headline: 144M determinants
        _sigma("sigma_12000x12000", 36, 8, 8, 12000, 12000),
        # the FP32 sigma of the mixed-precision Davidson at the headline size
        _sigma("sigma_mixed_12000x12000", 36, 8, 8, 12000, 12000, "mixed"),
        # the tensor-core sigma of the mixed-precision Davidson's first steps
        _sigma("sigma_mixed_tc_4000x4000", 26, 6, 6, 4000, 4000, "mixed_tc"),
        # one whole cycle (10 steps, the reference's block) on a selected basis of a small system
        {"name": "davidson_700x700", "kind": "davidson", "norb": 16, "nea": 5, "neb": 5, "na": 700, "nb": 700,
         "block": 10, "precision": "fp64"},
        # many small problems of the batching workload (norb 10-20, 3-6 electrons and hundreds of strings per spin)
        {"name": "batch_8", "kind": "batch", "problems": 8, "lo": 200, "hi": 1000, "block": 10},
        # density matrices at the end of a run, 1M determinants
        {"name": "rdm_1000x1000", "kind": "rdm", "norb": 20, "nea": 5, "neb": 5, "na": 1000, "nb": 1000},
        # the generic operator path on the 245,025-state full space (24 sites)
        {"name": "genmult_495x495", "kind": "genmult", "norb": 12, "nea": 4, "neb": 4, "na": 495, "nb": 495},
        # every configuration that the operator reaches from a small active space's state when orbitals are added
        {"name": "genexpand_70x70", "kind": "genexpand", "norb": 12, "nea": 4, "neb": 4, "active": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _spin_counts(rng, norb, lo, hi):
    """Electrons and strings per spin: equal spins half of the time."""
    nea = rng.randint(3, min(8, norb // 2))
    neb = nea if rng.random() < 0.5 else rng.randint(max(2, nea - 2), nea)
    na = min(_log_int(rng, lo, hi), math.comb(norb, nea))
    nb = na if neb == nea and rng.random() < 0.5 else min(_log_int(rng, lo, hi), math.comb(norb, neb))
    return nea, neb, na, nb


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "sigma_mixed", "sigma_tc", "davidson", "batch", "rdm", "genmult",
                       "genexpand"])
    if kind.startswith("sigma"):
        norb = rng.randint(8, 36)
        nea, neb, na, nb = _spin_counts(rng, norb, 56, 12000)
        precision = {"sigma": "fp64", "sigma_mixed": "mixed", "sigma_tc": "mixed_tc"}[kind]
        return {"kind": "sigma", "norb": norb, "nea": nea, "neb": neb, "na": na, "nb": nb, "precision": precision}
    if kind == "davidson":
        norb = rng.randint(10, 26)
        nea, neb, na, nb = _spin_counts(rng, norb, 100, 3000)
        return {"kind": kind, "norb": norb, "nea": nea, "neb": neb, "na": na, "nb": nb,
                "block": rng.randint(6, 12), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "batch":
        lo = _log_int(rng, 60, 500)
        return {"kind": kind, "problems": rng.randint(2, 16), "lo": lo, "hi": rng.randint(lo + 100, 1500),
                "block": rng.randint(6, 10)}
    if kind == "rdm":
        norb = rng.randint(8, 26)
        nea, neb, na, nb = _spin_counts(rng, norb, 56, 2500)
        return {"kind": kind, "norb": norb, "nea": nea, "neb": neb, "na": na, "nb": nb}
    if kind == "genmult":
        norb = rng.randint(7, 14)
        nea, neb, na, nb = _spin_counts(rng, norb, 20, 700)
        return {"kind": kind, "norb": norb, "nea": nea, "neb": neb, "na": na, "nb": nb}
    active = rng.randint(5, 9)
    return {"kind": kind, "norb": active + rng.randint(1, 5), "nea": rng.randint(2, active // 2),
            "neb": rng.randint(1, active // 2), "active": active}


# ------------------------------------------------------------------ inputs

def _strings(norb, ne, count, h_diag, seed):
    """Selected strings of one spin, ascending (all of them when the request covers the string space)."""
    total = math.comb(norb, ne)
    if count >= total:
        return synth.full_strings(norb, ne)
    if 4 * count >= total:  # a large share of the space: the lightest strings by their orbitals' one-body energy
        full = synth.full_strings(norb, ne)
        e = np.array([sum(h_diag[p] for p in range(norb) if (int(s) >> p) & 1) for s in full])
        return np.sort(full[np.argsort(e, kind="stable")[:count]])
    return synth.selected_strings(norb, ne, count, h_diag, seed)


def _system(case, seed):
    ints = synth.make_integrals(case["norb"], seed)
    if case.get("active"):  # every string of some of the orbitals, which ones from the seed
        orbs = np.sort(np.random.default_rng(seed).choice(case["norb"], case["active"], replace=False))
        spread = [np.array([sum(1 << int(orbs[k]) for k in range(case["active"]) if (int(s) >> k) & 1)
                            for s in synth.full_strings(case["active"], ne)], dtype=np.uint64)
                  for ne in (case["nea"], case["neb"])]
        return ints, spread[0], spread[1]
    h = np.diag(ints.h)
    a = _strings(case["norb"], case["nea"], case["na"], h, seed + 1)
    if (case["neb"], case["nb"]) == (case["nea"], case["na"]):
        return ints, a, a.copy()
    return ints, a, _strings(case["norb"], case["neb"], case["nb"], h, seed + 2)


def _ranks(strs, ne):
    aufbau = np.uint64((1 << ne) - 1)
    return np.array([bin(int(s)).count("1") for s in strs & ~aufbau], dtype=np.float64)


def _vector(case, a, b, seed, device):
    """A normalised state: random signs and sizes that fall off with the excitation rank, as a CI vector's do."""
    g = torch.Generator(device=device).manual_seed(seed)
    c = torch.randn(len(a), len(b), dtype=torch.float64, device=device, generator=g)
    c *= torch.from_numpy(np.exp(-0.7 * _ranks(a, case["nea"]))).to(device)[:, None]
    c *= torch.from_numpy(np.exp(-0.7 * _ranks(b, case["neb"]))).to(device)[None, :]
    return c / torch.linalg.norm(c)


def _start_vector(hd, seed):
    """A guess from the diagonal: the lowest determinant plus ten per cent of random signs that fall off with it.
    (Its Rayleigh quotient is soon below every diagonal element, so that the diagonal correction's denominators
    stay away from zero and two runs follow the same steps.)"""
    low = hd.min()
    w = np.exp(low - hd) * np.sign(np.random.default_rng(seed).normal(size=len(hd)))
    w *= 0.1 / np.linalg.norm(w)
    w[np.flatnonzero(hd <= low + 1e-9)[0]] += 1.0
    return w / np.linalg.norm(w)


def _batch_cases(case, seed):
    """The batch's systems: sizes from the case, integrals and strings from the seed."""
    rng = np.random.default_rng([case["problems"], case["lo"], case["hi"]])
    out = []
    for k in range(case["problems"]):
        norb, ne = int(rng.integers(10, 21)), int(rng.integers(3, 7))
        n = min(int(rng.integers(case["lo"], case["hi"] + 1)), math.comb(norb, ne))
        out.append(({"norb": norb, "nea": ne, "neb": ne, "na": n, "nb": n}, 1000 * (seed % 1000003) + k))
    return out


def _states(a, b, norb):
    return (a[:, None] | (b[None, :] << np.uint64(norb))).ravel()


def _genop(ints, ne, states):
    g = sbd_b200.GenOp(states, sign=True, device=0)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "FCIDUMP")
        synth.write_fcidump(path, ints, ne)
        g.set_fcidump(path)
    return g


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ctxs, starts = [], []
        for k, (sub, s) in enumerate(_batch_cases(case, seed)):
            ints, a, b = _system(sub, s)
            ctxs.append(sbd_b200.context_from_integrals(ints, a, b, device=0))
            starts.append(_start_vector(ctxs[-1].hii(), seed + k))
        return {"case": case, "ctxs": ctxs, "starts": starts}
    ints, a, b = _system(case, seed)
    if kind in ("genmult", "genexpand"):
        g = _genop(ints, case["nea"] + case["neb"], _states(a, b, case["norb"]))
        c = _vector(case, a, b, seed, "cuda").reshape(-1)
        if kind == "genexpand":
            return {"case": case, "op": g, "w": c.cpu().numpy()}
        torch.cuda.synchronize()
        return {"case": case, "op": g, "c": c, "w": torch.zeros_like(c)}
    ctx = sbd_b200.context_from_integrals(ints, a, b, device=0)
    if kind == "sigma":
        c = _vector(case, a, b, seed, "cuda")
        s = torch.empty_like(c)
        torch.cuda.synchronize()
        return {"case": case, "ctx": ctx, "c": c, "s": s}
    if kind == "davidson":
        return {"case": case, "ctx": ctx, "w": _start_vector(ctx.hii(), seed)}
    return {"case": case, "ctx": ctx, "w": _vector(case, a, b, seed, "cuda").cpu().numpy()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sigma":
        state["ctx"].sigma_device(state["c"].data_ptr(), state["s"].data_ptr(), PRECISION[case["precision"]])
        return state["s"]
    if kind == "davidson":
        e, w, te, tt = state["ctx"].davidson(state["w"], 1, case["block"], 1e-12,
                                             precision=PRECISION[case["precision"]], max_trace=case["block"])
        return {"energy": e, "vector": w, "trace": te, "residuals": tt}
    if kind == "batch":
        e, ws, _ = sbd_b200.davidson_batch(state["ctxs"], state["starts"], 1, case["block"], 1e-12)
        return {"energies": e, "vectors": ws}
    if kind == "rdm":
        one, two = state["ctx"].rdm(state["w"])
        return {"one": one, "two": two}
    if kind == "genmult":
        state["w"].zero_()
        torch.cuda.current_stream().synchronize()  # the operator works on a stream of its own
        state["op"].mult_device(state["c"].data_ptr(), state["w"].data_ptr())
        return state["w"]
    return state["op"].expand(state["w"], 0.0).view(np.int64)


# ------------------------------------------------------------------ what a pass cannot do without

def _occ(strs, norb):
    return ((strs[:, None] >> np.arange(norb, dtype=np.uint64)) & np.uint64(1)).astype(np.float32)


def _pair_counts(strs, norb):
    """Singles and doubles entries of one spin's strings (both directions)."""
    o = torch.from_numpy(_occ(strs, norb))
    ne = int(o[0].sum())
    s = d = 0
    for k in range(0, len(strs), 2000):
        m = o[k:k + 2000] @ o.T
        s += int((m == ne - 1).sum())
        d += int((m == ne - 2).sum())
    return s, d


def _elements(case):
    """Determinants and Hamiltonian elements (diagonal included) of one system."""
    _, a, b = _system(case, 0)
    na, nb = len(a), len(b)
    sa, da = _pair_counts(a, case["norb"])
    sb, db = (sa, da) if na == nb and np.array_equal(a, b) else _pair_counts(b, case["norb"])
    return na * nb, na * nb + nb * (sa + da) + na * (sb + db) + sa * sb


def work(case):
    """Bytes and operations of one pass: vectors once in and once out, two operations per Hamiltonian element."""
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for sub, _ in _batch_cases(case, 0):
            n, nnz = _elements(sub)
            total["bytes"] += 16.0 * n
            total["flops"] += 2.0 * nnz * (case["block"] + 1) + 2.0 * n * case["block"] ** 2
        return total
    n, nnz = _elements(case)
    if case["kind"] == "davidson":
        return {"bytes": 16.0 * n, "flops": 2.0 * nnz * (case["block"] + 1) + 2.0 * n * case["block"] ** 2}
    if case["kind"] == "rdm":
        return {"bytes": 8.0 * n + 8.0 * (2 * case["norb"] ** 2 + 4 * case["norb"] ** 4), "flops": 2.0 * nnz}
    if case["kind"] == "genmult":
        return {"bytes": 8.0 * n + 24.0 * n, "flops": 2.0 * nnz}
    if case["kind"] == "genexpand":
        return {"bytes": 32.0 * n, "flops": 2.0 * nnz}
    return {"bytes": 16.0 * n, "flops": 2.0 * nnz}


# ------------------------------------------------------------------ 64-bit evaluation with torch alone
#
# Everything below is in the alpha-strings-then-beta-strings order of the
# creation operators.  H = H_a (x) 1 + 1 (x) H_b + sum over folded pairs
# (pq|rs) A_pq (x) B_rs with A_pq = E_pq + E_qp (A_pp = n_p) on one spin's
# strings.  The package's vectors are in the interleaved order, which differs
# by the sign of `_phase`.

def _pair(p, q):
    hi, lo = torch.maximum(p, q), torch.minimum(p, q)
    return hi * (hi + 1) // 2 + lo


def _lowest_pair(m):
    """Lowest eigenvalue of a small symmetric matrix and its vector, by cyclic Jacobi rotations from the identity
    (which also settle the vector's sign)."""
    m, n = m.copy(), len(m)
    v = np.eye(n)
    for _ in range(100):
        if (np.triu(m, 1) ** 2).sum() < 1e-300:
            break
        for p in range(n):
            for q in range(p + 1, n):
                if abs(m[p, q]) < 1e-300:
                    continue
                theta = 0.5 * (m[q, q] - m[p, p]) / m[p, q]
                t = (1.0 if theta >= 0 else -1.0) / (abs(theta) + math.hypot(theta, 1.0))
                c = 1.0 / math.sqrt(t * t + 1.0)
                r = np.array([[c, c * t], [-c * t, c]])
                m[:, [p, q]] = m[:, [p, q]] @ r
                m[[p, q], :] = r.T @ m[[p, q], :]
                v[:, [p, q]] = v[:, [p, q]] @ r
    k = int(np.argmin(np.diag(m)))
    return float(m[k, k]), v[:, k]


class _Spin:
    """One spin's strings: occupations, single and double excitations with signs."""

    def __init__(self, strs, norb, device):
        o = torch.from_numpy(_occ(strs, norb)).to(device)
        self.occ, self.norb, self.n = o, norb, len(strs)
        self.below = torch.cumsum(o, 1) - o  # occupied orbitals below each
        ne = int(o[0].sum())
        m = o @ o.T
        self.si, self.sj = torch.nonzero(m == ne - 1, as_tuple=True)
        self.di, self.dj = torch.nonzero(m == ne - 2, as_tuple=True)
        del m
        d = o[self.si] - o[self.sj]
        self.p, self.q = d.argmax(1), d.argmin(1)  # created in the bra, annihilated in the ket
        cnt = self._at(self.sj, self.q) + self._at(self.sj, self.p) - (self.q < self.p).float()
        self.ssign = 1.0 - 2.0 * (cnt % 2).double()

    def _at(self, row, col):
        return self.below[row, col]

    def doubles(self, lo, hi):
        """(bra, ket, p1 < p2 created, q1 < q2 annihilated, sign of p1+ p2+ q2 q1) of double entries lo..hi."""
        i, j = self.di[lo:hi], self.dj[lo:hi]
        d = (self.occ[i] - self.occ[j]).to(torch.int8)
        p1, q1 = d.argmax(1), d.argmin(1)
        rev = torch.flip(d, (1,))
        p2, q2 = self.norb - 1 - rev.argmax(1), self.norb - 1 - rev.argmin(1)
        cnt = self._at(j, q1) + self._at(j, q2) - 1
        for x in (p1, p2):
            cnt = cnt + self._at(j, x) - (q1 < x).float() - (q2 < x).float()
        return i, j, p1, p2, q1, q2, 1.0 - 2.0 * (cnt.long() % 2).double()

    def chunks(self, size=1 << 21):
        return [(k, min(k + size, len(self.di))) for k in range(0, len(self.di), size)]

    def one_spin(self, h, eri):
        """The one-spin Hamiltonian, dense."""
        o = self.occ.double()
        diag_j = torch.einsum("ppqq->pq", eri) - torch.einsum("pqqp->pq", eri)
        m = torch.diag(o @ torch.diagonal(h) + 0.5 * ((o @ diag_j) * o).sum(1))
        x = torch.einsum("pqrr->pqr", eri) - torch.einsum("prrq->pqr", eri)
        for k in range(0, len(self.si), 1 << 20):
            s = slice(k, k + (1 << 20))
            p, q = self.p[s], self.q[s]
            m[self.si[s], self.sj[s]] = self.ssign[s] * (h[p, q] + (x[p, q] * o[self.sj[s]]).sum(1))
        for lo, hi in self.chunks():
            i, j, p1, p2, q1, q2, sg = self.doubles(lo, hi)
            m[i, j] = sg * (eri[p1, q1, p2, q2] - eri[p1, q2, p2, q1])
        return m

    def folded(self):
        """(bra, ket, folded pair, sign) of every A_pq entry, the occupations A_pp included."""
        i, p = torch.nonzero(self.occ, as_tuple=True)
        return (torch.cat([self.si, i]), torch.cat([self.sj, i]), torch.cat([_pair(self.p, self.q), _pair(p, p)]),
                torch.cat([self.ssign, torch.ones(len(i), dtype=torch.float64, device=i.device)]))


class _Exact:
    def __init__(self, ints, a, b, device):
        self.h = torch.from_numpy(ints.h).to(device)
        self.eri = torch.from_numpy(ints.eri).to(device)
        self.a, self.b = _Spin(a, ints.norb, device), _Spin(b, ints.norb, device)
        t = torch.tril_indices(ints.norb, ints.norb, device=device)
        self.v = self.eri[t[0], t[1]][:, t[0], t[1]].contiguous()
        self.ha, self.hb = self.a.one_spin(self.h, self.eri), self.b.one_spin(self.h, self.eri)
        self.ecore = ints.ecore

    def phase(self):
        cnt = self.a.occ @ self.b.below.T
        return 1.0 - 2.0 * (cnt.long() % 2).double()

    def sigma(self, c):
        na, nb, np_ = self.a.n, self.b.n, len(self.v)
        out = self.ha @ c
        out += c @ self.hb.T
        out += self.ecore * c
        i, j, pq, sg = self.a.folded()
        order = torch.argsort(i, stable=True)
        rows = torch.zeros(na + 1, dtype=torch.int64, device=c.device)
        rows[1:] = torch.cumsum(torch.bincount(i, minlength=na), 0)
        mat = torch.sparse_csr_tensor(rows, (pq * na + j)[order], sg[order], size=(na, np_ * na))
        bi, bj, rs, bs = self.b.folded()
        border = torch.argsort(bi, stable=True)
        bi, bj, rs, bs = bi[border], bj[border], rs[border], bs[border]
        ct = c.T.contiguous()
        w = max(1, min(nb, int(4e8) // (np_ * na)))
        cuts = torch.searchsorted(bi, torch.arange(0, nb + w, w, device=c.device)).tolist()
        for k, ib0 in enumerate(range(0, nb, w)):
            e = slice(cuts[k], cuts[k + 1])
            wd = min(w, nb - ib0)
            x = torch.zeros(np_, wd, na, dtype=torch.float64, device=c.device)
            x.view(np_ * wd, na)[rs[e] * wd + bi[e] - ib0] = bs[e][:, None] * ct[bj[e]]
            y = (self.v @ x.view(np_, wd * na)).view(np_, wd, na).transpose(1, 2).reshape(np_ * na, wd)
            out[:, ib0:ib0 + wd] += mat @ y
        return out

    def diagonal(self):
        t = torch.tril_indices(self.a.norb, self.a.norb, device=self.v.device)
        d = torch.nonzero(t[0] == t[1]).squeeze(1)
        j = self.v[d][:, d]
        return (self.ecore + torch.diagonal(self.ha)[:, None] + torch.diagonal(self.hb)[None, :]
                + self.a.occ.double() @ j @ self.b.occ.double().T)

    def davidson(self, w, block):
        """One cycle of the restarted Davidson from w: energy, vector, Ritz values, residual norms."""
        hd = self.diagonal()
        cs, hcs, te, tt = [w.clone()], [], [], []
        for ib in range(block):
            hcs.append(self.sigma(cs[ib]))
            m = torch.tensor([[float((cs[i] * hcs[max(i, j)]).sum()) if i <= j else float((cs[j] * hcs[i]).sum())
                               for j in range(ib + 1)] for i in range(ib + 1)], dtype=torch.float64)
            e0, u = _lowest_pair(m.numpy())
            w = sum(float(u[k]) * cs[k] for k in range(ib + 1))
            r = e0 * w - sum(float(u[k]) * hcs[k] for k in range(ib + 1))
            w = w / torch.linalg.norm(w)
            tol = float(torch.linalg.norm(r))
            te.append(e0)
            tt.append(tol)
            if ib + 1 < block:
                den = e0 - hd
                t = torch.where(den.abs() > 1e-12, r / den, r / (den - 1e-12)) / tol
                for c in cs:
                    t = t - (c * t).sum() * c
                cs.append(t / torch.linalg.norm(t))
        return float((w * self.sigma(w)).sum()), w, te, tt

    def rdm(self, c):
        """one[2][L^2], two[4][L^4] of c (this order's signs) in the layout i + L j + L^2 k + L^3 l."""
        L, dev = self.a.norb, c.device
        one = torch.zeros(2, L * L, dtype=torch.float64, device=dev)
        two = torch.zeros(4, L ** 4, dtype=torch.float64, device=dev)
        for s, (spin, x) in enumerate(((self.a, c), (self.b, c.T.contiguous()))):
            rho = x @ x.T

            def add(cr1, cr2, an2, an1, val):  # <cr1+ cr2+ an2 an1>
                two[3 * s].index_add_(0, an1 + L * an2 + L * L * cr1 + L ** 3 * cr2, val)

            v = rho[spin.si, spin.sj] * spin.ssign
            one[s].index_add_(0, spin.p + L * spin.q, v)
            for r in range(L):
                rr = torch.full_like(spin.p, r)
                t = v * (spin.occ[spin.si, r] * spin.occ[spin.sj, r]).double()
                add(spin.p, rr, rr, spin.q, t)
                add(rr, spin.p, spin.q, rr, t)
                add(spin.p, rr, spin.q, rr, -t)
                add(rr, spin.p, rr, spin.q, -t)
            o = spin.occ.double()
            d = torch.diagonal(rho)
            p = torch.arange(L, device=dev)
            one[s].index_add_(0, p + L * p, o.T @ d)
            nn = (o * d[:, None]).T @ o
            pp, qq = torch.meshgrid(p, p, indexing="ij")
            pp, qq, nn = pp.reshape(-1), qq.reshape(-1), torch.where(pp != qq, nn, 0.0).reshape(-1)
            add(pp, qq, qq, pp, nn)
            add(pp, qq, pp, qq, -nn)
            for lo, hi in spin.chunks():
                i, j, p1, p2, q1, q2, sg = spin.doubles(lo, hi)
                t = rho[i, j] * sg
                add(p1, p2, q2, q1, t)
                add(p2, p1, q1, q2, t)
                add(p1, p2, q1, q2, -t)
                add(p2, p1, q2, q1, -t)
        # opposite spins: <E_ki E_lj> = sum over (ja, ib) of (E_ki^T c)[ja, ib] (c E_lj^T)[ja, ib]

        def entries(spin):
            i, p = torch.nonzero(spin.occ, as_tuple=True)
            return (torch.cat([spin.si, i]), torch.cat([spin.sj, i]), torch.cat([spin.p * L + spin.q, p * L + p]),
                    torch.cat([spin.ssign, torch.ones(len(i), dtype=torch.float64, device=dev)]))

        ai, aj, ak, asg = entries(self.a)
        bi, bj, bk, bsg = entries(self.b)
        g = torch.zeros(L * L, L * L, dtype=torch.float64, device=dev)
        w = max(1, int(2e8) // (L * L * self.b.n))
        ct = c.T.contiguous()
        for j0 in range(0, self.a.n, w):
            wd = min(w, self.a.n - j0)
            e = torch.nonzero((aj >= j0) & (aj < j0 + wd)).squeeze(1)
            t = torch.zeros(L * L * wd, self.b.n, dtype=torch.float64, device=dev)
            t[ak[e] * wd + aj[e] - j0] = asg[e][:, None] * c[ai[e]]
            x = torch.zeros(L * L * self.b.n, wd, dtype=torch.float64, device=dev)
            x[bk * self.b.n + bi] = bsg[:, None] * ct[bj, j0:j0 + wd]
            x = x.view(L * L, self.b.n, wd).transpose(1, 2).reshape(L * L, wd * self.b.n)
            g += t.view(L * L, wd * self.b.n) @ x.T
        g4 = g.view(L, L, L, L)  # [k][i][l][j], k and i of alpha
        # the array's two opposite-spin blocks hold double excitations by the order of the spin orbitals: one
        # whose lower created and lower annihilated spin orbitals differ in spin goes to the other block
        p = torch.arange(L, device=dev)
        le, ne = p[:, None] <= p[None, :], p[:, None] != p[None, :]
        other = (le[:, None, :, None] != le[None, :, None, :]) & ne[:, :, None, None] & ne[None, None, :, :]
        for block, part in ((2, torch.where(other, 0.0, g4)), (1, torch.where(other, g4, 0.0))):
            two[block] += part.permute(2, 0, 3, 1).reshape(-1)  # l, k, j, i: i fastest
            two[3 - block] += part.permute(0, 2, 1, 3).reshape(-1)
        return one, two


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "genexpand":
        return None  # whole numbers
    if kind == "batch":
        es, ws = [], []
        for k, (sub, s) in enumerate(_batch_cases(case, seed)):
            ints, a, b = _system(sub, s)
            x = _Exact(ints, a, b, dev)
            ph = x.phase()
            w0 = torch.from_numpy(_start_vector(x.diagonal().reshape(-1).cpu().numpy(), seed + k))
            w0 = w0.to(dev).view(len(a), len(b))
            e, w, _, _ = x.davidson(w0 * ph, case["block"])
            es.append(e)
            ws.append((w * ph).reshape(-1).cpu().numpy())
        return {"energies": np.array(es), "vectors": ws}
    ints, a, b = _system(case, seed)
    x = _Exact(ints, a, b, dev)
    if kind == "genmult":  # the site order is this order: no phase
        return x.sigma(_vector(case, a, b, seed, dev)).reshape(-1)
    ph = x.phase()
    if kind == "sigma":
        return ph * x.sigma(ph * _vector(case, a, b, seed, dev))
    if kind == "davidson":
        w0 = torch.from_numpy(_start_vector(x.diagonal().reshape(-1).cpu().numpy(), seed))
        w0 = w0.to(dev).view(len(a), len(b))
        e, w, te, tt = x.davidson(w0 * ph, case["block"])
        return {"energy": e, "vector": (w * ph).reshape(-1).cpu().numpy(), "trace": np.array(te),
                "residuals": np.array(tt)}
    one, two = x.rdm(ph * _vector(case, a, b, seed, dev))
    return {"one": one.reshape(-1).cpu().numpy(), "two": two.reshape(-1).cpu().numpy()}
