"""RDMs by products (csrc/rdm_mma.cu) against the CPU oracle at the edges of
their blocks: four beta strings, eight columns (P = L (L + 1) / 2), 16 alpha
rows per CTA, 64-wide tiles of the density products; repeated strings keep the
scalar kernels."""
import numpy as np
import pytest

import oracle
import sbd_b200
from sbd_b200 import synth

pytestmark = pytest.mark.gpu

TOL = 1e-11  # the bound of the other RDM tests against the oracle (a normalised vector)


def _check(norb, nea, neb, na, nb, seed, repeat=0):
    ints = synth.make_integrals(norb, seed)
    rng = np.random.default_rng(seed)

    def pick(ne, n):
        s = synth.full_strings(norb, ne)
        return s[np.sort(rng.choice(len(s), min(n, len(s)), replace=False))]
    a, b = pick(nea, na), pick(neb, nb)
    if repeat:
        b = np.concatenate([b, b[:repeat]])
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    W = rng.normal(size=ctx.n)
    W /= np.linalg.norm(W)
    one, two = ctx.rdm(W)
    ref1, ref2 = oracle.Oracle(norb, a, b, ints.ecore, ints.h, ints.eri).correlation(W)
    assert np.abs(one - ref1).max() <= TOL and np.abs(two - ref2).max() <= TOL
    ctx.close()


@pytest.mark.parametrize("nb", [1, 3, 4, 5, 63, 65])
def test_beta_strings(nb):
    _check(9, 3, 3, 40, nb, 10 + nb)


@pytest.mark.parametrize("norb,nea", [(4, 1), (7, 3), (8, 4), (11, 5), (17, 1), (18, 1)])
def test_alpha_rows_and_columns(norb, nea):
    # 10 to 171 columns; full alpha spaces with up to 30 singles per string
    _check(norb, nea, 2, 70, 37, norb)


def test_repeated_strings_keep_the_scalar_kernels():
    _check(8, 3, 3, 20, 21, 3, repeat=2)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_stays_where_its_terms_go(bad):
    ints = synth.make_integrals(9, 8)
    a, b = synth.full_strings(9, 3)[::2], synth.full_strings(9, 3)[1::2]
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    W = np.random.default_rng(8).normal(size=ctx.n)
    W /= np.linalg.norm(W)
    W[7 * ctx.nb + 11] = bad
    got = ctx.rdm(W)
    ref = oracle.Oracle(9, a, b, ints.ecore, ints.h, ints.eri).correlation(W)
    for x, r in zip(got, ref):
        finite = np.isfinite(r)
        assert finite.any() and not finite.all()
        assert np.array_equal(np.isfinite(x), finite)
        assert np.abs(x[finite] - r[finite]).max() <= TOL
    ctx.close()


def test_repeated_alpha_strings():
    ints = synth.make_integrals(8, 5)
    s = synth.full_strings(8, 3)
    a, b = np.concatenate([s[:20], s[5:8]]), s[10:31]
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    W = np.random.default_rng(5).normal(size=ctx.n)
    W /= np.linalg.norm(W)
    for x, r in zip(ctx.rdm(W), oracle.Oracle(8, a, b, ints.ecore, ints.h, ints.eri).correlation(W)):
        assert np.abs(x - r).max() <= TOL
    ctx.close()


@pytest.mark.parametrize("na,nb", [(12000, 3), (3, 12000), (2, 29200)])
def test_long_spins(na, nb):
    # 12,000 strings: two panels of the same-spin products; 29,200 beta strings: more than shared memory holds of a
    # row of W
    s = synth.full_strings(26, 6)
    ints = synth.make_integrals(26, 4)
    rng = np.random.default_rng(na)
    near = s[(s & np.uint64(0x3F)) == 7]  # 1,140 strings that share three orbitals, so that the short spin connects
    a, b = (np.sort(rng.choice(s if n > 100 else near[:20], n, replace=False)) for n in (na, nb))
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    W = rng.normal(size=ctx.n)
    W /= np.linalg.norm(W)
    one, two = ctx.rdm(W)
    ref1, ref2 = oracle.Oracle(26, a, b, ints.ecore, ints.h, ints.eri).correlation(W)
    assert np.abs(one - ref1).max() <= TOL and np.abs(two - ref2).max() <= TOL
    ctx.close()
