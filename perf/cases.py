"""Performance cases of the framework: what a CI program has it do, through the
Python mirror (ciflow_gb300.ciflow) and the C ABI it binds.

Kinds of case (the dict's "kind"):

* "product": y = H x on device buffers with a matrix that the program keeps, the
  call an eigensolver of its own makes per iteration. method "fci" | "doci" |
  "big" (CI_Big: a determinant list whose elements are recomputed in the call),
  type "f64" (plain matrix) | "f32" (mixed matrix, FP32 product) | "f64_mixed"
  (mixed matrix, FP64 product).
* "list_build": a determinant list's matrix (FCI_File) built from the list and
  multiplied once.
* "rdm": the 1- and 2-particle density matrices of a CI vector in host memory.
* "solve": the whole call: integrals in host memory to ground-state energy and
  vector (matrix build and eigensolve). The reference converges its eigensolver to
  machine precision (ARPACK with tol 0); the residual target here is as small as
  both methods reach, so that the vector is determined to about ten digits.

Integrals are synthetic: (pq|rs) = sum_k L^k_pq L^k_rs over `rank` symmetric
factors, which makes them positive semidefinite as a pair matrix, with orbital
energies rising along the diagonal of h. Vectors have a CI vector's shape: one
leading determinant and amplitudes that fall with the orbital energies occupied.
"""
import itertools
import math

import numpy as np
import torch

from ciflow_gb300 import _abi as A
from ciflow_gb300.ciflow import CI_Big, DOCI, FCI, FCI_File, Hamiltonian

TOL = 1e-11


def listed():
    return [
        # the mixed method's hot call at the headline size (12 orbitals, 6+6 electrons)
        {"name": "fci_f32_L12", "kind": "product", "method": "fci", "type": "f32", "L": 12, "na": 6, "nb": 6, "rank": 16},
        # the same call at the size most served requests have: a GPU that one call hardly fills
        {"name": "fci_f32_L10", "kind": "product", "method": "fci", "type": "f32", "L": 10, "na": 5, "nb": 5, "rank": 16},
        # the plain method's hot call at the headline size
        {"name": "fci_f64_L12", "kind": "product", "method": "fci", "type": "f64", "L": 12, "na": 6, "nb": 6, "rank": 16},
        # a small open-shell space with ragged string counts (126 x 84): launch latency counts
        {"name": "fci_f64_L9", "kind": "product", "method": "fci", "type": "f64", "L": 9, "na": 4, "nb": 3, "rank": 16},
        # seniority-zero CI at its largest size, the mixed method's FP32 product
        {"name": "doci_f32_L24", "kind": "product", "method": "doci", "type": "f32", "L": 24, "na": 12, "nb": 12, "rank": 24},
        # seniority-zero CI at a middle size away from half filling, the plain method's product
        {"name": "doci_f64_L20", "kind": "product", "method": "doci", "type": "f64", "L": 20, "na": 8, "nb": 8, "rank": 24},
        # a CISD list of 32 orbitals whose matrix is kept: build and first product
        {"name": "list_build_L32", "kind": "list_build", "L": 32, "na": 8, "nb": 8, "rank": 16, "keep": 1.0, "shuffle": False},
        # a selected-CI list (a random part of a CISD list, in no order) whose matrix is not kept
        {"name": "big_f64_L28", "kind": "product", "method": "big", "type": "f64", "L": 28, "na": 7, "nb": 7, "rank": 16,
         "keep": 0.7, "shuffle": True},
        # density matrices of the headline solve's state, and of the largest seniority-zero state
        {"name": "rdm_fci_L12", "kind": "rdm", "method": "fci", "L": 12, "na": 6, "nb": 6, "rank": 16},
        {"name": "rdm_doci_L24", "kind": "rdm", "method": "doci", "L": 24, "na": 12, "nb": 12, "rank": 24},
        # the whole headline call, mixed method
        {"name": "solve_fci_mixed_L12", "kind": "solve", "method": "fci", "type": "mixed", "L": 12, "na": 6, "nb": 6, "rank": 16},
        # the small solve that an orbital optimiser makes thousands of: latency alone
        {"name": "solve_doci_f64_L12", "kind": "solve", "method": "doci", "type": "f64", "L": 12, "na": 6, "nb": 6, "rank": 16},
    ]


def _fci_dim(c):
    return math.comb(c["L"], c["na"]) * math.comb(c["L"], c["nb"])


def _draw_fci(rng, lo, hi):
    """An FCI space of lo..hi determinants."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    every = [{"L": L, "na": na, "nb": nb} for L in range(6, 13) for na in range(2, L - 1) for nb in range(1, na + 1)]
    every = [c for c in every if lo <= _fci_dim(c) <= hi and abs(math.log(_fci_dim(c) / want)) < 0.7]
    return dict(rng.choice(every), rank=rng.choice([10, 14, 16, 20, 28]))


def _draw_doci(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    every = [(L, n) for L in range(10, 31) for n in range(3, L - 2) if lo <= math.comb(L, n) <= hi]
    near = [s for s in every if abs(math.log(math.comb(*s) / want)) < 0.7]
    L, n = rng.choice(near or every)
    return {"L": L, "na": n, "nb": n, "rank": rng.choice([16, 20, 24])}


def _draw_list(rng, lo, hi):
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    every = []
    for L in range(12, 41):
        for na in range(3, 11):
            for nb in range(na - 1, na + 1):
                if L > 2 * na:
                    n = _cisd_size(L, na, nb)
                    if want <= n <= 130000:
                        every.append({"L": L, "na": na, "nb": nb, "keep": round(want / n, 4)})
    c = rng.choice([e for e in every if e["keep"] > 0.15])
    return dict(c, rank=16, shuffle=rng.random() < 0.5)


def draw(rng):
    kind = rng.choice(["fci", "fci", "doci", "list", "list", "rdm_fci", "rdm_doci", "solve"])
    if kind == "fci":
        return dict(_draw_fci(rng, 2000, 853776), kind="product", method="fci", type=rng.choice(["f32", "f32", "f64", "f64_mixed"]))
    if kind == "doci":
        return dict(_draw_doci(rng, 2000, 2704156), kind="product", method="doci", type=rng.choice(["f32", "f64_mixed", "f64"]))
    if kind == "list":
        if rng.random() < 0.5:
            return dict(_draw_list(rng, 1500, 52000), kind="list_build")
        return dict(_draw_list(rng, 1500, 52000), kind="product", method="big", type="f64")
    if kind == "rdm_fci":
        return dict(_draw_fci(rng, 2000, 853776), kind="rdm", method="fci")
    if kind == "rdm_doci":
        return dict(_draw_doci(rng, 2000, 2704156), kind="rdm", method="doci")
    if rng.random() < 0.5:
        # closed shells: their lowest state stands alone, so its vector is well determined
        L, n = rng.choice([(7, 3), (8, 4), (9, 4), (10, 4), (10, 5), (11, 5)])
        return {"kind": "solve", "method": "fci", "type": rng.choice(["mixed", "f64"]), "L": L, "na": n, "nb": n, "rank": rng.choice([12, 16, 20])}
    L, n = rng.choice([(10, 4), (11, 5), (14, 6), (14, 7), (16, 8), (18, 7), (20, 10)])
    return {"kind": "solve", "method": "doci", "type": rng.choice(["mixed", "f64"]), "L": L, "na": n, "nb": n, "rank": rng.choice([16, 24])}


# ---- inputs ----

def _sym(rng, L, sigma):
    m = np.triu(rng.normal(0.0, sigma, (L, L)))
    return m + np.triu(m, 1).T


def _integrals(case, seed):
    """(h, eri chemist), the tensor exactly 8-fold symmetric."""
    L = case["L"]
    rng = np.random.default_rng(seed)
    h = _sym(rng, L, 0.05)
    h[np.diag_indices(L)] = -2.0 + 0.25 * np.arange(L)
    eri = np.zeros((L * L, L * L))
    for _ in range(case["rank"]):
        v = (_sym(rng, L, 0.1) + 0.3 * np.eye(L)).reshape(-1)
        eri += np.multiply.outer(v, v)
    return h, eri.reshape((L,) * 4)


def _strings(L, n):
    """The strings of n electrons in L orbitals, ascending (the rank order of the spaces)."""
    s = np.zeros(1, np.int64)
    by = [[s[:0]] * (n + 1) for _ in range(L + 1)]
    by[0][0] = s
    for l in range(1, L + 1):
        for k in range(min(l, n) + 1):
            low = by[l - 1][k]
            by[l][k] = np.concatenate([low, by[l - 1][k - 1] | (1 << (l - 1))]) if k else low
    return by[L][n]


def _level(strings, L):
    """Sum of the occupied orbitals' energies above the lowest string's."""
    e = np.zeros(len(strings))
    for p in range(L):
        e += 0.25 * p * ((strings >> p) & 1)
    return e - e.min()


def _cisd_size(L, na, nb):
    a, b = na * (L - na), nb * (L - nb)
    dbl = lambda n: math.comb(n, 2) * math.comb(L - n, 2)  # noqa: E731
    return 1 + a + b + dbl(na) + dbl(nb) + a * b


def _det_list(case, seed):
    """(up, down) of a CISD list: the lowest determinant first, its singles and doubles
    after it; `keep` of them at random (the first always), `shuffle`: in random order."""
    def excited(n, k):
        out = []
        for hs in itertools.combinations(range(n), k):
            for ps in itertools.combinations(range(n, case["L"]), k):
                s = (1 << n) - 1
                for o in hs + ps:
                    s ^= 1 << o
                out.append(s)
        return np.array(out, np.int64)

    na, nb = case["na"], case["nb"]
    ra, rb = np.int64((1 << na) - 1), np.int64((1 << nb) - 1)
    a1, a2, b1, b2 = excited(na, 1), excited(na, 2), excited(nb, 1), excited(nb, 2)
    up = np.concatenate([[ra], a1, np.full(len(b1), ra), a2, np.full(len(b2), ra), np.repeat(a1, len(b1))])
    dn = np.concatenate([[rb], np.full(len(a1), rb), b1, np.full(len(a2), rb), b2, np.tile(b1, len(a1))])
    rng = np.random.default_rng(seed + 1)
    n = max(2, int(round(case["keep"] * len(up))))
    at = np.concatenate([[0], 1 + np.sort(rng.choice(len(up) - 1, n - 1, replace=False))])
    if case["shuffle"]:
        at = rng.permutation(at)
    return up[at].astype(np.uint64), dn[at].astype(np.uint64)


def _vector(case, seed):
    """A CI vector of the case's space, normalised (host, float64)."""
    rng = np.random.default_rng(seed + 2)
    L = case["L"]
    if "keep" in case:
        up, dn = _det_list(case, seed)
        e = _level(up.astype(np.int64), L) + _level(dn.astype(np.int64), L)
    elif case["method"] == "doci":
        e = 2.0 * _level(_strings(L, case["na"]), L)
    else:
        e = (_level(_strings(L, case["na"]), L)[:, None] + _level(_strings(L, case["nb"]), L)[None, :]).reshape(-1)
    c = rng.standard_normal(len(e), dtype=np.float32) * np.exp(-0.5 * e)
    c[int(np.argmin(e))] = 3.0
    return c / np.linalg.norm(c)


def _hamiltonian(case, seed):
    h, eri = _integrals(case, seed)
    return Hamiltonian(case["L"], 0, case["na"], case["nb"], 0.0, h, eri)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        h, eri = _integrals(case, seed)
        return {"case": case, "h": h, "eri": eri}
    ham = _hamiltonian(case, seed)
    s = {"case": case, "ham": ham}
    c = _vector(case, seed)
    if kind == "rdm":
        s["cim"] = (FCI if case["method"] == "fci" else DOCI)(ham, A.MIXED)
        s["c"] = c
        return s
    dt = torch.float32 if case.get("type") == "f32" else torch.float64
    s["x"] = torch.from_numpy(c).cuda().to(dt)
    s["y"] = torch.empty_like(s["x"])
    if kind == "list_build":
        s["up"], s["down"] = _det_list(case, seed)
        ham.device()
    elif case["method"] == "big":
        up, dn = _det_list(case, seed)
        s["cim"] = CI_Big(ham, up=up, down=dn)
    else:
        s["cim"] = (FCI if case["method"] == "fci" else DOCI)(ham, A.FP64 if case["type"] == "f64" else A.MIXED)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "product":
        s["cim"].get_mat().mvprod_device(s["x"], s["y"])
        return s["y"]
    if kind == "list_build":
        s["cim"] = FCI_File(s["ham"], up=s["up"], down=s["down"])
        m = s["cim"].get_mat()
        m.mvprod_device(s["x"], s["y"])
        return {"y": s["y"], "elements": m.datasize()}
    if kind == "rdm":
        L = case["L"]
        n2 = L * (L - 1) // 2
        one, aa, ab, bb = np.empty((2, L, L)), np.empty((n2, n2)), np.empty((L * L, L * L)), np.empty((n2, n2))
        A.check(A.lib().cigpu_rdm(s["cim"].get_mat().handle, A.ptr(s["c"]), A.ptr(one), A.ptr(aa), A.ptr(ab), A.ptr(bb)), "cigpu_rdm")
        return {"one": one, "aa": aa, "ab": ab, "bb": bb}
    ham = Hamiltonian(case["L"], 0, case["na"], case["nb"], 0.0, s["h"], s["eri"])
    cim = (FCI if case["method"] == "fci" else DOCI)(ham, A.FP64 if case["type"] == "f64" else A.MIXED)
    cim.solve(tol=TOL)
    return {"e0": cim.get_ci_energy(), "c": _phase(cim.get_eigvec())}


def _phase(c):
    """An eigenvector's sign is free: its first component of (nearly) the largest
    magnitude is made positive, as a program that compares states does."""
    m = np.abs(c)
    return c if c[int(np.argmax(m > 0.9 * m.max()))] > 0 else -c


def work(case):
    """Products: x and y once, and a multiply and an add for each structural element of
    H (what the operator is, however it is applied). Solves: the integrals in, the
    vector out and 20 products, fewer than any Krylov method needs to reach the
    residual target. Densities: c in, the matrices out, a multiply and an add for each
    two-electron excitation of the state."""
    L, na, nb = case["L"], case["na"], case["nb"]
    sa, sb = na * (L - na), nb * (L - nb)
    dbl = lambda n: math.comb(n, 2) * math.comb(L - n, 2)  # noqa: E731
    if "keep" in case:
        dim = max(2, int(round(case["keep"] * _cisd_size(L, na, nb))))
        # a listed determinant meets about the share `keep` of the reference's excitations
        row = 1 + min(dim, 0.1 * case["keep"] * (sa + sb + dbl(na) + dbl(nb) + sa * sb))
    elif case["method"] == "doci":
        dim, row = math.comb(L, na), 1 + sa
    else:
        dim, row = _fci_dim(case), 1 + sa + sb + dbl(na) + dbl(nb) + sa * sb
    ints = 8 * (L * L + L**4)
    size = 4 if case.get("type") == "f32" else 8
    if case["kind"] == "rdm":
        n2 = L * (L - 1) // 2
        return {"bytes": 8 * dim + 8 * (2 * L * L + 2 * n2 * n2 + L**4), "flops": 2 * dim * row}
    if case["kind"] == "solve":
        return {"bytes": ints + 8 * dim, "flops": 20 * 2 * dim * row}
    lists = 16 * dim if "keep" in case else 0
    return {"bytes": 2 * size * dim + ints + lists, "flops": 2 * dim * row}


# ---- the same in 64 bits, plain torch ----

def _moves(strings, L, dev):
    """E_pq on strings: (source [L, L, D], sign [L, L, D]) with
    (E_pq c)[I] = sign[p, q, I] c[source[p, q, I]]."""
    D = len(strings)
    src, sgn = np.zeros((L, L, D), np.int64), np.zeros((L, L, D))
    pre = np.stack([_popcount(strings & ((1 << p) - 1)) for p in range(L)])
    for p in range(L):
        for q in range(L):
            has = ((strings >> p) & 1) == 1
            ok = has if p == q else has & (((strings >> q) & 1) == 0)
            J = np.where(ok, strings if p == q else (strings ^ (1 << p)) | (1 << q), strings[0])
            src[p, q] = np.searchsorted(strings, J)
            # <I| a+_p a_q |J>: electrons of I below p (p taken out), below q in the rest
            below_q = pre[q] - (1 if p < q else 0)
            sgn[p, q] = np.where(ok, 1.0 - 2.0 * ((pre[p] + below_q) % 2), 0.0) if p != q else ok
    return torch.from_numpy(src).to(dev), torch.from_numpy(sgn).to(dev)


def _popcount(v):
    n = np.zeros(np.shape(v), np.int64)
    for b in range(64):
        n += (v >> b) & 1
    return n


class _FciOperator:
    def __init__(self, case, seed, dev):
        L = self.L = case["L"]
        h, eri = _integrals(case, seed)
        self.a = _moves(_strings(L, case["na"]), L, dev)
        self.b = _moves(_strings(L, case["nb"]), L, dev)
        self.k = torch.from_numpy(h - 0.5 * np.einsum("prrq->pq", eri)).to(dev)
        self.v = torch.from_numpy(eri.reshape(L * L, L * L)).to(dev)
        self.shape = (self.a[0].shape[2], self.b[0].shape[2])

    def one(self, C, spin, p, q):
        src, sgn = (self.a, self.b)[spin]
        return sgn[p, q][:, None] * C[src[p, q]] if spin == 0 else C[:, src[p, q]] * sgn[p, q][None, :]

    def __call__(self, x):
        L, C = self.L, x.reshape(self.shape)
        D = torch.empty((L * L, C.numel()), dtype=C.dtype, device=C.device)
        for p in range(L):
            for q in range(L):
                D[p * L + q] = (self.one(C, 0, p, q) + self.one(C, 1, p, q)).reshape(-1)
        y = self.k.reshape(-1) @ D
        G = (0.5 * self.v) @ D
        del D
        y = y.reshape(self.shape)
        for p in range(L):
            for q in range(L):
                g = G[p * L + q].reshape(self.shape)
                y += self.one(g, 0, p, q) + self.one(g, 1, p, q)
        return y.reshape(-1)

    def rdm(self, c):
        L, C = self.L, c.reshape(self.shape)
        X = [torch.stack([self.one(C, s, p, q).reshape(-1) for p in range(L) for q in range(L)]) for s in (0, 1)]
        one = torch.stack([(x @ c).reshape(L, L) for x in X])
        # <a+_pA a+_qB a_sB a_rA> = <E^A_pr E^B_qs> = (E^A_rp c)(E^B_qs c)
        ab = (X[0] @ X[1].T).reshape(L, L, L, L).permute(1, 2, 0, 3).reshape(L * L, L * L)
        del X
        return {"one": one, "aa": self.same(C, 0), "ab": ab, "bb": self.same(C.T.contiguous(), 1)}

    def same(self, C, spin):
        """<a+_p a+_q a_s a_r> of one spin, C with that spin's strings first."""
        L, D = self.L, C.shape[0]
        src, sgn = (self.a, self.b)[spin]
        occ = torch.stack([sgn[p, p] for p in range(L)]) > 0
        held = sum(occ[p].long() << p for p in range(L))
        n = int(occ[:, 0].sum())
        rest, rows = torch.from_numpy(_strings(L, n - 2)).to(C.device) if n >= 2 else None, []
        for p in range(L):
            for q in range(p + 1, L):
                out = torch.zeros((len(rest) if rest is not None else 1, C.shape[1]), dtype=C.dtype, device=C.device)
                at = torch.nonzero(occ[p] & occ[q])[:, 0]
                if rest is not None and len(at):
                    between = sum((occ[m][at].long() for m in range(p + 1, q)), torch.zeros_like(at))
                    out[torch.searchsorted(rest, held[at] ^ (1 << p) ^ (1 << q))] = C[at] * (1.0 - 2.0 * (between % 2))[:, None]
                rows.append(out.reshape(-1))
        M = torch.stack(rows)
        return M @ M.T


class _DociOperator:
    def __init__(self, case, seed, dev):
        L = self.L = case["L"]
        h, eri = _integrals(case, seed)
        self.K = np.einsum("pqpq->pq", eri).copy()
        J = np.einsum("ppqq->pq", eri)
        w = _strings(L, case["na"])
        self.s = torch.from_numpy(w).to(dev)
        occ = torch.stack([((self.s >> p) & 1).double() for p in range(L)])
        self.diag = 2.0 * torch.from_numpy(np.diag(h).copy()).to(dev) @ occ
        self.diag += torch.sum(occ * (torch.from_numpy(2.0 * J - self.K).to(dev) @ occ), 0)
        self.occ = occ

    def hop(self, x, j, k):
        """x at the strings with orbitals j and k exchanged, 0 where both or neither is held."""
        J = torch.searchsorted(self.s, self.s ^ ((1 << j) | (1 << k))).clamp_(max=len(self.s) - 1)
        return torch.where(self.occ[j] != self.occ[k], x[J], torch.zeros_like(x))

    def __call__(self, x):
        y = self.diag * x
        for j in range(self.L):
            for k in range(j + 1, self.L):
                y += float(self.K[j, k]) * self.hop(x, j, k)
        return y

    def rdm(self, c):
        L = self.L
        n = (self.occ * (c * c)) @ self.occ.T
        B = torch.diag(torch.diagonal(n))
        for j in range(L):
            for k in range(j + 1, L):
                B[j, k] = B[k, j] = 0.5 * torch.dot(c, self.hop(c, j, k))
        one = torch.diag(torch.diagonal(n))
        iu = [(p, q) for p in range(L) for q in range(p + 1, L)]
        aa = torch.diag(torch.stack([n[p, q] for p, q in iu]))
        ab = torch.zeros((L, L, L, L), dtype=c.dtype, device=c.device)
        for p in range(L):
            for q in range(L):
                ab[p, q, p, q] = n[p, q]
        for p in range(L):
            for q in range(L):
                ab[p, p, q, q] = B[p, q]
        return {"one": torch.stack([one, one]), "aa": aa, "ab": ab.reshape(L * L, L * L), "bb": aa.clone()}


class _ListOperator:
    """Slater-Condon elements of every connected pair of the list, rows in chunks."""

    def __init__(self, case, seed, dev):
        L = self.L = case["L"]
        h, eri = _integrals(case, seed)
        self.h, self.g = torch.from_numpy(h).to(dev), torch.from_numpy(eri).to(dev)
        up, dn = _det_list(case, seed)
        w = torch.from_numpy(np.stack([up, dn]).astype(np.int64)).to(dev)
        self.occ = torch.stack([((w >> p) & 1) for p in range(L)], 2).double()  # [spin, det, orbital]
        self.n = w.shape[1]
        self.ne = (case["na"], case["nb"])

    def __call__(self, x):
        oa, ob = self.occ[0], self.occ[1]
        fa, fb = oa.float(), ob.float()
        y, elements = torch.zeros_like(x), 0
        jk = torch.einsum("ppqq->pq", self.g) - torch.einsum("pqqp->pq", self.g)
        tot = oa + ob
        for r0 in range(0, self.n, 2048):
            rows = slice(r0, min(r0 + 2048, self.n))
            ea = self.ne[0] - fa[rows] @ fa.T
            eb = self.ne[1] - fb[rows] @ fb.T
            for na, nb in ((0, 0), (1, 0), (0, 1), (2, 0), (0, 2), (1, 1)):
                I, J = torch.nonzero((ea == na) & (eb == nb), as_tuple=True)
                I = I + r0
                for at in range(0, len(I), 1 << 21):
                    i, j = I[at:at + (1 << 21)], J[at:at + (1 << 21)]
                    v = self.elements(i, j, na, nb, jk, tot)
                    y.index_add_(0, i, v * x[j])
                    elements += int(((v.abs() > 1e-14) & (i <= j)).sum())
        return y, elements

    def elements(self, i, j, na, nb, jk, tot):
        a, b = self.occ[0], self.occ[1]
        if na + nb == 0:
            one = tot[i] @ torch.diagonal(self.h)
            J = torch.einsum("ppqq->pq", self.g)
            K = J - jk
            return one + 0.5 * torch.sum(tot[i] * (tot[i] @ J), 1) - 0.5 * torch.sum(a[i] * (a[i] @ K) + b[i] * (b[i] @ K), 1)
        if na + nb == 1:
            o = a if na else b
            (p,), (q,), s = self.diff(o[i], o[j], 1)
            v = self.h[p, q]
            common, other = o[i] * o[j], (b if na else a)[i]
            rows = torch.zeros_like(v)
            for r in range(self.L):
                rows = rows + (common[:, r] + other[:, r]) * self.g[p, q, r, r] - common[:, r] * self.g[p, r, r, q]
            return s * (v + rows)
        if na == 1:
            (p,), (q,), s = self.diff(a[i], a[j], 1)
            (r,), (t,), u = self.diff(b[i], b[j], 1)
            return s * u * self.g[p, q, r, t]
        o = a if na else b
        (p, r), (q, t), s = self.diff(o[i], o[j], 2)
        return s * (self.g[p, q, r, t] - self.g[p, t, r, q])

    @staticmethod
    def diff(oi, oj, k):
        """Orbitals of i not in j (ascending), of j not in i, and the sign that brings
        them into line (one string's electrons in ascending order)."""
        pi, pj = oi * (1 - oj), oj * (1 - oi)
        ci, cj = torch.cumsum(oi, 1) - oi, torch.cumsum(oj, 1) - oj  # electrons below each orbital
        par = torch.sum(pi * ci + pj * cj, 1) % 2
        ps = torch.topk(pi, k, 1, sorted=False).indices.sort(1).values
        qs = torch.topk(pj, k, 1, sorted=False).indices.sort(1).values
        return tuple(ps.T), tuple(qs.T), 1.0 - 2.0 * par


def _lowest(op, n, dev):
    """The lowest eigenpair by Lanczos with full reorthogonalisation."""
    g = torch.Generator(device="cpu").manual_seed(7)
    q = torch.randn(n, generator=g, dtype=torch.float64).to(dev)
    q /= torch.linalg.norm(q)
    Q, al, be = [q], [], []
    for m in range(min(n, 260)):
        w = op(Q[-1])
        al.append(float(w @ Q[-1]))
        B = torch.stack(Q)
        for _ in range(2):
            w = w - B.T @ (B @ w)
        b = float(torch.linalg.norm(w))
        if m % 5 == 4 or b < 1e-10 or m + 1 == min(n, 260):
            T = np.diag(al) + np.diag(be, 1) + np.diag(be, -1)
            e, z = np.linalg.eigh(T)
            if abs(b * z[-1, 0]) < 1e-11 or b < 1e-10 or m + 1 == min(n, 260):
                c = (B.T @ torch.from_numpy(z[:, 0].copy()).to(dev)).cpu().numpy()
                return float(e[0]), c / np.linalg.norm(c)
        be.append(b)
        Q.append(w / b)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "solve":
        op = (_FciOperator if case["method"] == "fci" else _DociOperator)(case, seed, dev)
        n = _fci_dim(case) if case["method"] == "fci" else math.comb(case["L"], case["na"])
        e0, v = _lowest(op, n, dev)
        return {"e0": e0, "c": _phase(v)}
    c = torch.from_numpy(_vector(case, seed)).to(dev)
    if case.get("type") == "f32":
        c = c.float().double()
    if "keep" in case:
        y, elements = _ListOperator(case, seed, dev)(c)
        return {"y": y, "elements": elements} if kind == "list_build" else y
    op = (_FciOperator if case["method"] == "fci" else _DociOperator)(case, seed, dev)
    return op.rdm(c) if kind == "rdm" else op(c)
