"""GPU RDM parity (CIDens::construct_density with DensFCI / DensDOCI).

The device RDMs of a state must equal the reference's for the same CI vector
(golden RDMs of the reference itself for BeH2 and the L=8 / L=10 synthetic
spaces; the oracle's restatement for the larger spaces), to FP64 round-off,
and satisfy CIDens::test_invariants (traces, E_dens == E_CI).
"""
import numpy as np
import pytest

import oracle as O
from ciflow_gb300 import _abi as A
from ciflow_gb300.ciflow import DOCI, FCI, Hamiltonian
from ciflow_gb300.synthetic import make_integrals
from tests.helpers import beh2_integrals, integrals, load_golden

pytestmark = pytest.mark.gpu


def rdm_via_abi(cim, c):
    L = cim.get_l()
    np_ = L * (L - 1) // 2
    r1 = np.empty((2, L, L))
    aa = np.empty((np_, np_))
    ab = np.empty((L * L, L * L))
    bb = np.empty((np_, np_))
    A.check(A.lib().cigpu_rdm(cim.get_mat().handle, A.ptr(np.ascontiguousarray(c)), A.ptr(r1), A.ptr(aa),
                              A.ptr(ab), A.ptr(bb)))
    return r1, aa, ab, bb


def assert_rdm_close(got, ref, atol):
    for g, r, name in zip(got, ref, ("rdm1", "aa", "ab", "bb")):
        err = np.abs(g - r).max()
        assert err <= atol, (name, err)


@pytest.mark.parametrize("tag,cls", [("doci", DOCI), ("fci", FCI)])
def test_beh2_rdm_matches_reference(tag, cls):
    ints, meta, a = beh2_integrals()
    cim = cls(Hamiltonian.from_integrals(ints))
    c = a[f"{tag}_c"]
    got = rdm_via_abi(cim, c)
    assert_rdm_close(got, (a[f"{tag}_rdm1"], a[f"{tag}_aa"], a[f"{tag}_ab"], a[f"{tag}_bb"]), 1e-13)
    assert abs(O.dens_energy(ints, *got) - meta[tag]["dens_energy"]) < 1e-11


@pytest.mark.parametrize("name", ["c0", "c4"])
def test_fci_rdm_of_solved_state(name):
    meta, a = load_golden(name)
    ints = integrals(name)
    cim = FCI(Hamiltonian.from_integrals(ints))
    cim.solve(tol=1e-9)
    c = cim.get_eigvec()
    got = rdm_via_abi(cim, c)
    ref = O.rdm(O.FCI, ints.L, ints.nup, ints.ndown, c)
    assert_rdm_close(got, ref, 1e-12)
    # against the reference's own RDMs of its own eigenvector (sign-invariant quantities)
    assert_rdm_close(got, (a["rdm1"], a["aa"], a["ab"], a["bb"]), 1e-7)
    # CIDens::test_invariants
    N = ints.nup + ints.ndown
    assert abs(np.trace(got[0][0]) + np.trace(got[0][1]) - N) < 1e-10
    assert abs(np.trace(got[1]) + np.trace(got[2]) + np.trace(got[3]) - N * (N - 1) / 2) < 1e-8
    assert abs(O.dens_energy(ints, *got) - cim.get_ci_energy()) < 1e-9


def test_fci_rdm_facade_and_unequal_spins():
    ints = make_integrals(7, 3, 2, nchol=6, seed=77)
    cim = FCI(Hamiltonian.from_integrals(ints))
    c = np.random.default_rng(5).standard_normal(cim.get_dim())
    c /= np.linalg.norm(c)
    got = rdm_via_abi(cim, c)
    ref = O.rdm(O.FCI, ints.L, ints.nup, ints.ndown, c, literal=True)
    assert_rdm_close(got, ref, 1e-13)


@pytest.mark.parametrize("L,na,nb", [(12, 1, 6), (13, 2, 6), (13, 2, 7)])
def test_fci_rdm_many_beta_strings(L, na, nb):
    # enough blocks for 36 excitations per thread: one whole set, and a ragged second one
    ints = make_integrals(L, na, nb, nchol=4, seed=3)
    cim = FCI(Hamiltonian.from_integrals(ints))
    c = np.random.default_rng(L + nb).standard_normal(cim.get_dim())
    c /= np.linalg.norm(c)
    assert_rdm_close(rdm_via_abi(cim, c), O.rdm(O.FCI, L, na, nb, c), 1e-13)


def test_c1_rdm_against_oracle():
    ints = integrals("c1")
    cim = FCI(Hamiltonian.from_integrals(ints), precision=A.MIXED)
    cim.solve(tol=1e-6)
    c = cim.get_eigvec()
    got = rdm_via_abi(cim, c)
    ref = O.rdm(O.FCI, ints.L, ints.nup, ints.ndown, c)
    assert_rdm_close(got, ref, 1e-11)
    assert abs(O.dens_energy(ints, *got) - cim.get_ci_energy()) < 1e-6


@pytest.mark.parametrize("L,n", [(8, 4), (10, 3)])
def test_doci_rdm_against_oracle(L, n):
    ints = make_integrals(L, n, n, nchol=8, seed=3 * L + n)
    cim = DOCI(Hamiltonian.from_integrals(ints))
    cim.solve(tol=1e-9)
    c = cim.get_eigvec()
    got = rdm_via_abi(cim, c)
    ref = O.rdm(O.DOCI, L, n, n, c)
    assert_rdm_close(got, ref, 1e-13)
    assert abs(O.dens_energy(ints, *got) - cim.get_ci_energy()) < 1e-9


def test_c2_doci_rdm():
    meta, a = load_golden("c2")
    ints = integrals("c2")
    cim = DOCI(Hamiltonian.from_integrals(ints), precision=A.MIXED)
    cim.solve(tol=1e-6)
    c = cim.get_eigvec()
    got = rdm_via_abi(cim, c)
    ref = O.rdm(O.DOCI, ints.L, ints.nup, ints.ndown, c)
    assert_rdm_close(got, ref, 1e-10)
    # reference RDMs of the reference eigenvector: agree to the eigenvector accuracy
    assert np.abs(got[0] - a["rdm1"]).max() < 1e-5


def test_python_facade_density():
    ints, meta, _ = beh2_integrals()
    cim = FCI(Hamiltonian.from_integrals(ints))
    cim.solve(tol=1e-10)
    cim.construct_density()
    d = cim.cid
    d.test_invariants()
    assert abs(d.get_dens_energy() - cim.get_ci_energy()) < 1e-10
    # antisymmetry of the same-spin block through the reference getter semantics
    assert d.get_two_rdm(0, 1, 2, 3, 4) == -d.get_two_rdm(0, 2, 1, 3, 4)
    assert d.get_two_rdm(0, 2, 2, 3, 4) == 0.0


@pytest.mark.parametrize("L,n", [(17, 8), (18, 11), (20, 13), (21, 5), (22, 17)])
def test_doci_rdm_split(L, n):
    """The DOCI RDMs by low and high orbitals (spaces past the split's row threshold),
    from a mixed matrix and from a plain one (which makes its plan on the first call):
    the oracle's, and the same bits from both and from a second call."""
    ints = make_integrals(L, n, n, nchol=4, seed=L + n)
    ham = Hamiltonian.from_integrals(ints)
    mixed, plain = DOCI(ham, A.MIXED), DOCI(ham, A.FP64)
    c = np.random.default_rng(n).standard_normal(mixed.get_mat().n)
    c /= np.linalg.norm(c)
    got = rdm_via_abi(mixed, c)
    assert_rdm_close(got, O.rdm(O.DOCI, L, n, n, c), 1e-13)
    for other in (rdm_via_abi(plain, c), rdm_via_abi(plain, c), rdm_via_abi(mixed, c)):
        for g, o in zip(got, other):
            assert np.array_equal(g, o)


@pytest.mark.parametrize("kind", ["unit", "minus", "pair", "tiny", "halves"])
def test_doci_rdm_split_values(kind):
    # the ends of the fixed point: +-1, entries below a unit of the low digit, and digits at
    # their own ends (multiples of 2^-31 and of 2^-30 plus half a low digit)
    L, n = 17, 8
    ints = make_integrals(L, n, n, nchol=4, seed=5)
    cim = DOCI(Hamiltonian.from_integrals(ints))
    rng = np.random.default_rng(3)
    c = np.zeros(cim.get_dim())
    if kind in ("unit", "minus"):
        c[1234] = 1.0 if kind == "unit" else -1.0
    elif kind == "pair":
        c[[100, 101]] = 0.6, -0.8
    elif kind == "tiny":
        c[:] = rng.standard_normal(c.size) * 2.0 ** -45
        c[7] = 1.0
    else:
        c[:] = rng.integers(-3, 4, c.size) * 2.0 ** -30 + rng.integers(-1, 2, c.size) * 2.0 ** -31
        c[11] = -0.5
    got = rdm_via_abi(cim, c)
    assert_rdm_close(got, O.rdm(O.DOCI, L, n, n, c), 1e-13)
