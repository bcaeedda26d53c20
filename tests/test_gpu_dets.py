"""Determinant-list CI on the device (cigpu_build_dets), through the C ABI.

* The CRS of the reference's own determinant lists (BeH2 STO-3G, 1225
  determinants; Be cc-pVDZ, 100 GKCI determinants) is bit-identical to the
  reference's FCI_File CRS (SHA-256 of the upper triangle), and E0 matches the
  reference (1e-8 Eh plain, 1e-6 mixed) and the known answer of TestDetFile.cpp.
* The 70-orbital Be list of Testmp.cpp (128-bit strings) gives the CRS of the
  oracle's 128-bit restatement and the known answer -14.346369472944886.
* The full FCI list in the reference's determinant order gives the FCI CRS.
* CI_Big storage (no stored matrix): matvecs equal the CRS matvecs and E0 agrees.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from ciflow_gb300 import _abi as A
from ciflow_gb300.ciflow import CI_Big, FCI, FCI_File, Hamiltonian
from ciflow_gb300.synthetic import make_integrals

from .helpers import crs_sha256, dets_case

pytestmark = pytest.mark.gpu


def upper_sha(cim):
    row, col, val = cim.get_mat().upper()
    return crs_sha256(row, col, val)


@pytest.mark.parametrize("tag", ["beh2", "be_gkci", "be70"])
def test_dets_crs_and_energy(tag):
    ints, up, down, words, meta = dets_case(tag)
    ham = Hamiltonian.from_integrals(ints)
    cim = FCI_File(ham, up=up, down=down, words=words)
    assert cim.get_dim() == meta["dim"] and cim.get_mat().datasize() == meta["nnz"]
    assert upper_sha(cim) == meta["crs_sha256"]
    cim.solve(tol=1e-10)
    assert cim.get_ci_energy() == pytest.approx(meta["e0_oracle"], abs=1e-9)
    if "e0_known_answer" in meta:
        assert cim.get_ci_energy() == pytest.approx(meta["e0_known_answer"], abs=1e-9)
    mixed = FCI_File(ham, up=up, down=down, words=words, precision=A.MIXED)
    mixed.solve(tol=1e-7)
    assert mixed.get_ci_energy() == pytest.approx(meta["e0_oracle"], abs=1e-6)


def test_full_list_gives_the_fci_matrix():
    ints = make_integrals(8, 4, 3, nchol=16, seed=12)

    def strings(L, n):
        out, s = [], (1 << n) - 1
        while s < (1 << L):
            out.append(s)
            t = s | (s - 1)
            s = (t + 1) | (((~t & -~t) - 1) >> ((s & -s).bit_length()))
        return out
    ua, db = strings(8, 4), strings(8, 3)
    up = np.array([u for u in ua for d in db], np.uint64)
    down = np.array([d for u in ua for d in db], np.uint64)
    ham = Hamiltonian.from_integrals(ints)
    a, b = FCI_File(ham, up=up, down=down), FCI(ham)
    for x, y in zip(a.get_mat().upper(), b.get_mat().upper()):
        assert np.array_equal(x, y)
    # a shuffled list: the same matrix permuted
    perm = np.random.default_rng(1).permutation(len(up))
    c = FCI_File(ham, up=up[perm], down=down[perm])
    m = O.build_dets(ints, up[perm], down[perm])
    assert upper_sha(c) == crs_sha256(m.row, m.col, m.val)
    c.solve(tol=1e-10)
    b.solve(tol=1e-10)
    assert c.get_ci_energy() == pytest.approx(b.get_ci_energy(), abs=1e-10)


@pytest.mark.parametrize("tag", ["beh2", "be70"])
def test_onthefly_matches_stored(tag):
    ints, up, down, words, meta = dets_case(tag)
    ham = Hamiltonian.from_integrals(ints)
    stored = FCI_File(ham, up=up, down=down, words=words)
    fly = CI_Big(ham, up=up, down=down, words=words)
    layout, stored_n = ctypes.c_int(), ctypes.c_int64()
    A.check(A.lib().cigpu_crs_layout(fly.get_mat().handle, ctypes.byref(layout), ctypes.byref(stored_n)))
    assert layout.value == A.LAYOUT_ONTHEFLY and stored_n.value == 0
    x = np.random.default_rng(0).standard_normal(meta["dim"])
    y1, y2 = stored.get_mat().mvprod(x), fly.get_mat().mvprod(x)
    assert np.max(np.abs(y1 - y2)) <= 1e-12 * np.max(np.abs(y1))
    fly.solve(tol=1e-10)
    assert fly.get_ci_energy() == pytest.approx(meta["e0_oracle"], abs=1e-9)


@pytest.mark.parametrize("tag", ["beh2", "be70"])
@pytest.mark.parametrize("frac", [0.0, 0.3, 0.77, 1.0])
def test_ci_big_stored_block_matches_stored(tag, frac):
    """CI_Big with the block of its first `keep` determinants stored (CI_Big::mvprod,
    CIMethod.cpp:943-984): the matvec (stored block + every other element recomputed)
    equals the fully stored matrix's for keep = 0, a part of the list and all of it,
    the stored element count is the block's, and the energy is the known one."""
    ints, up, down, words, meta = dets_case(tag)
    ham = Hamiltonian.from_integrals(ints)
    n = meta["dim"]
    keep = int(round(frac * n))
    stored = FCI_File(ham, up=up, down=down, words=words)
    big = CI_Big(ham, up=up, down=down, words=words, keep=keep)
    layout, stored_n = ctypes.c_int(), ctypes.c_int64()
    A.check(A.lib().cigpu_crs_layout(big.get_mat().handle, ctypes.byref(layout), ctypes.byref(stored_n)))
    assert layout.value == A.LAYOUT_ONTHEFLY
    # the block's elements: those of the stored matrix with row and column below keep
    r, c, _ = stored.get_mat().full()
    rows = np.repeat(np.arange(n), np.diff(r.astype(np.int64)))
    assert stored_n.value == int(np.count_nonzero((rows < keep) & (c < keep)))
    x = np.random.default_rng(2).standard_normal(n)
    y1, y2 = stored.get_mat().mvprod(x), big.get_mat().mvprod(x)
    assert np.max(np.abs(y1 - y2)) <= 1e-12 * np.max(np.abs(y1))
    if frac in (0.3, 0.77):
        big.solve(tol=1e-10)
        assert big.get_ci_energy() == pytest.approx(meta["e0_oracle"], abs=1e-9)


def test_dets_rejections():
    ints, up, down, words, meta = dets_case("beh2")
    ham = Hamiltonian.from_integrals(ints)
    out = ctypes.c_void_p()
    lib = A.lib()
    bad = up.copy()
    u3 = int(up[3])
    bad[3] = np.uint64(u3 | (1 << next(o for o in range(7) if not (u3 >> o) & 1)))  # one electron too many
    assert lib.cigpu_build_dets(ham.device(), len(up), 1, A.ptr(bad), A.ptr(down), A.DETS_CRS, A.FP64, None,
                                ctypes.byref(out)) == A.EINVAL
    outside = up.copy()
    u0 = int(up[0])
    outside[0] = np.uint64((u0 ^ (u0 & -u0)) | (1 << 9))  # lowest electron moved to orbital 9
    assert lib.cigpu_build_dets(ham.device(), len(up), 1, A.ptr(outside), A.ptr(down), A.DETS_CRS, A.FP64, None,
                                ctypes.byref(out)) == A.EINVAL  # orbital 9 of a 7-orbital space
    assert lib.cigpu_build_dets(ham.device(), len(up), 1, A.ptr(up), A.ptr(down), A.DETS_ONTHEFLY, A.MIXED, None,
                                ctypes.byref(out)) == A.ENOTSUP


def rdms(cim_handle, L, c):
    np_ = L * (L - 1) // 2
    one, aa = np.zeros((2, L, L)), np.zeros((np_, np_))
    ab, bb = np.zeros((L * L, L * L)), np.zeros((np_, np_))
    c = np.ascontiguousarray(c)
    A.check(A.lib().cigpu_rdm(cim_handle, A.ptr(c), A.ptr(one), A.ptr(aa), A.ptr(ab), A.ptr(bb)))
    return one, aa, ab, bb


def test_dets_rdm_matches_reference_densfile():
    """The device DensFILE RDMs of the BeH2 list equal the reference's DensFILE
    (tests/golden/dets.npz) to 1e-13 and, as TestDensity.cpp checks, DensFCI's to
    1e-11; two runs are bit-identical (order-independent fixed-point sums)."""
    import json, os
    from .helpers import GOLDEN, beh2_integrals
    ints, up, down, words, meta = dets_case("beh2")
    g = np.load(os.path.join(GOLDEN, "dets.npz"))
    cim = FCI_File(Hamiltonian.from_integrals(ints), up=up, down=down, words=words)
    got = rdms(cim.get_mat().handle, ints.L, g["beh2_c"])
    for x, k in zip(got, ("rdm1", "aa", "ab", "bb")):
        assert np.max(np.abs(x - g[f"beh2_{k}"])) < 1e-13, k
    again = rdms(cim.get_mat().handle, ints.L, g["beh2_c"])
    assert all(np.array_equal(x, y) for x, y in zip(got, again))
    _, _, arr = beh2_integrals()
    for x, k in zip(got, ("rdm1", "aa", "ab", "bb")):
        assert np.max(np.abs(x - arr[f"fci_{k}"])) < 1e-11, k
    cim.solve(tol=1e-10)
    cim.construct_density()
    assert cim.cid.get_dens_energy() == pytest.approx(cim.get_ci_energy(), abs=1e-9)


def test_dets_rdm_matches_oracle_gkci():
    ints, up, down, words, meta = dets_case("be_gkci")
    cim = FCI_File(Hamiltonian.from_integrals(ints), up=up, down=down, words=words)
    cim.solve(tol=1e-10)
    c = cim.get_eigvec()
    got = rdms(cim.get_mat().handle, ints.L, c)
    ref = O.rdm_dets(ints.L, up, down, c)
    for x, y in zip(got, ref):
        assert np.max(np.abs(x - y)) < 1e-13



def random_list(L, na, nb, n, seed):
    """n determinants: the lowest one, then random excitations of it of up to four
    electrons (many pairs connected, many not), distinct, in random order."""
    rng = np.random.default_rng(seed)
    seen = []
    ref = ((1 << na) - 1, (1 << nb) - 1)
    while len(seen) < n:
        d = list(ref)
        for _ in range(int(rng.integers(0, 5))):
            spin = int(rng.integers(0, 2))
            occ = [o for o in range(L) if (d[spin] >> o) & 1]
            emp = [o for o in range(L) if not (d[spin] >> o) & 1]
            if occ and emp:
                d[spin] ^= (1 << int(rng.choice(occ))) | (1 << int(rng.choice(emp)))
        if tuple(d) not in seen:
            seen.append(tuple(d))
    up, down = np.array([s[0] for s in seen], np.uint64), np.array([s[1] for s in seen], np.uint64)
    return up, down


@pytest.mark.parametrize("L,na,nb,n", [(6, 1, 1, 36), (8, 1, 1, 64), (5, 2, 1, 1), (7, 3, 3, 31), (9, 3, 2, 33), (31, 3, 2, 129),
                                       (32, 2, 2, 257), (33, 2, 3, 300), (40, 1, 1, 1000)])
def test_scan_edges(L, na, nb, n):
    """The pair scan at the edges of its rows, words and queue (lists shorter than a
    word, one row over it, every pair connected, 32 and 33 orbitals): the CRS equals the
    oracle's bit for bit, and the matvecs without a stored matrix (none of it, and a
    leading block) equal the stored one's."""
    ints = make_integrals(L, na, nb, nchol=4, seed=L + n)
    up, down = random_list(L, na, nb, n, seed=n)
    ham = Hamiltonian.from_integrals(ints)
    cim = FCI_File(ham, up=up, down=down)
    m = O.build_dets(ints, up, down)
    assert upper_sha(cim) == crs_sha256(m.row, m.col, m.val)
    x = np.random.default_rng(3).standard_normal(n)
    y = cim.get_mat().mvprod(x)
    y_ref = O.sym_mvprod(m, x)
    # a row's terms in another order: n roundings of its largest partial sum
    tol = 2.0 ** -52 * (n + 2) * float(np.abs(m.val).max() * np.abs(x).sum())
    assert np.abs(y - y_ref).max() <= tol
    for keep in (0, n // 3):
        big = CI_Big(ham, up=up, down=down, keep=keep)
        assert np.abs(big.get_mat().mvprod(x) - y_ref).max() <= tol


@pytest.mark.parametrize("kind", ["no zero", "zeros", "vanishing differences"])
@pytest.mark.parametrize("precision", [A.FP64, A.MIXED])
def test_dropped_elements(kind, precision):
    """Lists whose elements are all kept, dropped by zero integrals, and dropped though no
    integral is zero (equal integrals whose difference vanishes: the build that takes the
    connected pairs for the structure has to start again): the oracle's CRS."""
    ints = make_integrals(12, 3, 3, nchol=5, seed=8)
    if kind == "zeros":
        odd = np.arange(12) % 2  # two symmetry classes: (pq|rs) with p q r s odd in all vanish
        ints.eri[((odd[:, None, None, None] + odd[:, None, None] + odd[:, None] + odd) % 2) == 1] = 0.0
    elif kind == "vanishing differences":
        ints.eri[...] = 0.125
    up, down = random_list(12, 3, 3, 400, seed=4)
    m = O.build_dets(ints, up, down)
    cim = FCI_File(Hamiltonian.from_integrals(ints), up=up, down=down, precision=precision)
    row, col, val = cim.get_mat().upper()
    assert np.array_equal(row.astype(np.int64), m.row) and np.array_equal(col, m.col)
    if precision == A.FP64:
        assert np.array_equal(val, m.val)
    else:
        assert np.array_equal(val, m.val.astype(np.float32).astype(np.float64))


@pytest.mark.parametrize("L,na,nb,n,repeat", [(14, 3, 3, 6100, 1), (36, 4, 3, 6001, 1), (40, 1, 1, 1600, 5),
                                              (28, 4, 3, 19500, 1)])
def test_matvec_of_a_longer_list(L, na, nb, n, repeat):
    """The matvec without a stored matrix past the short lists' kernel: 32 and 64-bit
    strings, and a list of repeated determinants whose pairs are all connected (words that
    overflow the queue), whole and with a stored leading block, against the stored CRS."""
    ints = make_integrals(L, na, nb, nchol=3, seed=L)
    up, down = random_list(L, na, nb, n, seed=n)
    up, down = np.tile(up, repeat), np.tile(down, repeat)
    ham = Hamiltonian.from_integrals(ints)
    x = np.random.default_rng(6).standard_normal(len(up))
    stored = FCI_File(ham, up=up, down=down).get_mat()
    y = stored.mvprod(x)
    _, _, val = stored.full()
    tol = 2.0 ** -52 * (len(up) + 2) * float(np.abs(val).max() * np.abs(x).max()) * np.sqrt(len(up))
    for keep in (0, 777):
        assert np.abs(CI_Big(ham, up=up, down=down, keep=keep).get_mat().mvprod(x) - y).max() <= tol


def cisd_list(L, na, nb):
    """(up, down) strings as Python integers: the lowest determinant, its singles and its
    doubles, in the order a program writes them."""
    import itertools

    def excited(n, k):
        ref = (1 << n) - 1
        return [ref ^ sum(1 << o for o in hs + ps) for hs in itertools.combinations(range(n), k)
                for ps in itertools.combinations(range(n, L), k)]

    ra, rb, a1, b1 = (1 << na) - 1, (1 << nb) - 1, excited(na, 1), excited(nb, 1)
    pairs = [(ra, rb)] + [(a, rb) for a in a1] + [(ra, b) for b in b1]
    pairs += [(a, rb) for a in excited(na, 2)] + [(ra, b) for b in excited(nb, 2)]
    return pairs + [(a, b) for a in a1 for b in b1]


@pytest.mark.parametrize("L,na,nb,n", [(70, 3, 2, 6043), (70, 3, 3, 20001), (40, 3, 3, 6100), (24, 4, 4, 6001),
                                       (36, 6, 6, 40001)])
def test_matvec_of_an_ordered_list(L, na, nb, n):
    """The matvec without a stored matrix on lists in order of excitation, whose groups take
    runs of rows from all over the list: one and two words per string, one and two blocks
    per group, groups in order (the longest list), whole and with stored leading blocks of
    whole groups and of a part of one, against the stored CRS."""
    pairs = cisd_list(L, na, nb)[:n]
    words = 1 if L <= 64 else 2
    up, down = (np.array([(s >> (64 * w)) & (2 ** 64 - 1) for s in side for w in range(words)], np.uint64)
                for side in zip(*pairs))
    ints = make_integrals(L, na, nb, nchol=2, seed=L)
    ham = Hamiltonian.from_integrals(ints)
    x = np.random.default_rng(6).standard_normal(len(pairs))
    stored = FCI_File(ham, up=up, down=down).get_mat()
    assert stored.n == len(pairs) > 6000
    y = stored.mvprod(x)
    _, _, val = stored.full()
    tol = 2.0 ** -52 * (len(pairs) + 2) * float(np.abs(val).max() * np.abs(x).max()) * np.sqrt(len(pairs))
    for keep in (0, 777, 3200):
        assert np.abs(CI_Big(ham, up=up, down=down, keep=keep).get_mat().mvprod(x) - y).max() <= tol


@pytest.mark.parametrize("kind", ["no zero", "zeros", "vanishing differences"])
@pytest.mark.parametrize("n", [3, 45, 999, 1001, 1999])
def test_build_groups(n, kind):
    """List builds by groups of 4, 8 and 32 rows, evaluated twice (short lists, vanishing
    integrals), from the structure, and from the structure in vain: the oracle's CRS."""
    ints = make_integrals(13, 3, 3, nchol=4, seed=n)
    if kind == "zeros":
        odd = np.arange(13) % 2
        ints.eri[((odd[:, None, None, None] + odd[:, None, None] + odd[:, None] + odd) % 2) == 1] = 0.0
    elif kind == "vanishing differences":
        ints.eri[...] = 0.125
    up, down = random_list(13, 3, 3, n, seed=n)
    m = O.build_dets(ints, up, down)
    assert upper_sha(FCI_File(Hamiltonian.from_integrals(ints), up=up, down=down)) == crs_sha256(m.row, m.col, m.val)
