"""The FP64 alpha-beta term by tiles (csrc/ab_mma.cu) against the CPU oracle
and the gather kernel: string counts at the edges of its groups of 16 and
tiles of 8, alpha singles at the edges of 8 and 16 per CTA, odd rows (no
16-byte lines), and bases that keep the gather kernel."""
import numpy as np
import pytest

import oracle
import sbd_b200
from sbd_b200 import synth

pytestmark = pytest.mark.gpu

# sums of at most a few thousand FP64 products of O(1) terms: the bound of the sigma parity tests
TOL = 1e-12


def _system(norb, nea, neb, na, nb, seed, shuffle=False):
    ints = synth.make_integrals(norb, seed)
    rng = np.random.default_rng(seed)

    def pick(ne, n):
        s = synth.full_strings(norb, ne)
        s = s[np.sort(rng.choice(len(s), min(n, len(s)), replace=False))]
        return rng.permutation(s) if shuffle else s
    return ints, pick(nea, na), pick(neb, nb)


def _check(ints, a, b, shapes=((0, 0),)):
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = np.random.default_rng(3).normal(size=ctx.n)
    ref = oracle.Oracle(ints.norb, a, b, ints.ecore, ints.h, ints.eri).sigma(C)
    for g, t in shapes:
        ctx.set_tuning(g, t)
        assert np.abs(ctx.sigma(C) - ref).max() <= TOL * np.abs(ref).max(), (g, t)
    ctx.close()


@pytest.mark.parametrize("nb", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 50])
def test_beta_strings_at_group_edges(nb):
    _check(*_system(9, 3, 3, 21, nb, 100 + nb))


@pytest.mark.parametrize("norb,nea", [(3, 1), (5, 1), (9, 1), (10, 1), (17, 1), (18, 1), (8, 4), (10, 5)])
def test_alpha_singles_at_block_edges(norb, nea):
    # full spaces: nea (norb - nea) = 2, 4, 8, 9, 16, 17, 16 and 25 singles per alpha string
    _check(*_system(norb, nea, min(2, nea), 10 ** 6, 40, norb), shapes=((0, 0), (16, 128), (8, 256), (4, 128)))


@pytest.mark.parametrize("shuffle", [False, True])
def test_unequal_spins_and_string_order(shuffle):
    _check(*_system(11, 5, 3, 67, 133, 5, shuffle), shapes=((0, 0), (16, 512), (8, 128), (2, 128)))


def test_wide_orbital_range():
    # 2,016 off-diagonal pairs, the largest pair index
    ints = synth.make_integrals(64, 2)
    rng = np.random.default_rng(2)
    s = np.array([(1 << 63) | (1 << i) for i in range(60)] + [3 << i for i in range(62)], dtype=np.uint64)
    b = np.sort(rng.choice(s, 40, replace=False))
    _check(ints, b[:9], b)


def test_repeated_strings_keep_the_gather_kernel():
    ints, a, b = _system(8, 3, 3, 20, 30, 9)
    _check(ints, a, np.concatenate([b, b[:3]]))


@pytest.mark.parametrize("na,nb", [(1, 70), (33, 31), (64, 64), (65, 126), (126, 17)])
def test_dense_same_spin_product_at_tile_edges(na, nb):
    # full or nearly full spaces of 9 orbitals (126 strings of 4 electrons): the dense product of same_dense.cu,
    # odd and even rows, 32- and 64-wide tiles; the rows kernels as the second shape
    ints, a, b = _system(9, 4, 4, na, nb, 40 + na)
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = np.random.default_rng(4).normal(size=ctx.n)
    ref = oracle.Oracle(9, a, b, ints.ecore, ints.h, ints.eri).sigma(C)
    for method in (0, 1):
        ctx.set_fp64_same_spin(method)
        assert np.abs(ctx.sigma(C) - ref).max() <= TOL * np.abs(ref).max(), method
    ctx.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_stays_where_the_operator_takes_it(bad):
    ints, a, b = _system(9, 4, 4, 60, 61, 8)
    C = np.random.default_rng(5).normal(size=(60, 61))
    C[7, 11] = bad
    orc = oracle.Oracle(9, a, b, ints.ecore, ints.h, ints.eri)
    e = np.zeros((60, 61))
    e[7, 11] = 1.0
    reached = orc.sigma(e.ravel()) != 0.0
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    s = ctx.sigma(C)
    assert not np.isfinite(s[reached]).any()
    ra = np.array([bin(int(x ^ a[7])).count("1") for x in a])
    rb = np.array([bin(int(x ^ b[11])).count("1") for x in b])
    unreached = (ra[:, None] + rb[None, :] > 4).ravel()  # more than two excitations away
    assert unreached.any() and np.isfinite(s[unreached]).all()
    ref = orc.sigma(np.where(np.isfinite(C), C, 0.0).ravel())
    assert np.abs(s - ref)[unreached].max() <= TOL * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("nb", [723, 726, 728])
def test_fp32_sigma_by_tiles(nb):
    # 731 x 723..728 determinants are past the rule's half million; rows of 4, 2 and 1 times 16 bytes
    ints = synth.make_integrals(14, 6)
    rng = np.random.default_rng(nb)
    s = synth.full_strings(14, 5)
    a, b = (s[np.sort(rng.choice(len(s), n, replace=False))] for n in (731, nb))
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = rng.normal(size=ctx.n)
    C /= np.linalg.norm(C)
    ref = ctx.sigma(C)
    got = ctx.sigma(C, precision=sbd_b200.MIXED)
    # the bound of the mixed sigma's other tests against FP64
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("na,nb", [(1028, 1036), (1100, 1100), (1040, 1028)])
def test_integer_products_of_padded_string_counts(na, nb):
    # counts that are padded to multiples of 16, against the rows kernels
    ints, a, b = _system(18, 5, 5, na, nb, 70 + na)
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = np.random.default_rng(6).normal(size=ctx.n)
    ctx.set_fp64_same_spin(1)
    ref = ctx.sigma(C)
    ctx.set_fp64_same_spin(0)
    for x, r in ((C, ref), (np.where(np.arange(ctx.n) == 5, np.inf, C), None)):
        got = ctx.sigma(x)
        if r is not None:
            assert np.abs(got - r).max() <= TOL * np.abs(r).max()
        else:
            assert not np.isfinite(got[5]) and np.isfinite(got).sum() > ctx.n // 2
    ctx.close()


def test_tiles_without_stages():
    # 48 orbitals and 19,990 beta strings leave no shared memory for staged results beside eight singles' integrals
    # and the row of C; more than 20,000 keep the gather kernel
    ints = synth.make_integrals(48, 3)
    b = synth.selected_strings(48, 4, 20100, np.diag(ints.h), 4)
    a = b[[0, 1, 2, 5, 9]]
    for nb in (19990, 20016):
        ctx = sbd_b200.context_from_integrals(ints, a, b[:nb])
        C = np.random.default_rng(nb).normal(size=ctx.n)
        got = ctx.sigma(C)
        ctx.set_tuning(4, 512)  # the gather kernel
        ref = ctx.sigma(C)
        assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
        ctx.close()


@pytest.mark.parametrize("norb,ne,nb", [(36, 4, 15001), (36, 4, 16600), (36, 4, 18200), (48, 4, 16400), (48, 4, 19001)])
def test_launch_shapes_beside_long_rows_of_c(norb, ne, nb):
    # sixteen singles at 24 warps; eight with stages where sixteen leave fewer than 24 (16 and 4 here); eight without
    # stages where those leave fewer than 32 (24 and 4); FP32 vectors from half a million determinants
    ints = synth.make_integrals(norb, 3)
    b = synth.selected_strings(norb, ne, nb, np.diag(ints.h), 4)
    a = b[:36]
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = np.random.default_rng(nb).normal(size=ctx.n)
    C /= np.linalg.norm(C)
    got, mixed = ctx.sigma(C), ctx.sigma(C, precision=sbd_b200.MIXED)
    ctx.set_tuning(4, 512)  # the gather kernel
    ref = ctx.sigma(C)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    assert np.abs(mixed - ref).max() <= 2e-5 * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("nb", [1, 17, 40])
def test_few_beta_strings_of_many_orbitals(nb):
    # fewer groups of beta strings than warps: the integral rows keep the others busy
    ints = synth.make_integrals(30, 5)
    strs = synth.full_strings(30, 3)
    ctx = sbd_b200.context_from_integrals(ints, strs[:500], strs[:nb])
    C = np.random.default_rng(nb).normal(size=ctx.n)
    ref = oracle.Oracle(30, strs[:500], strs[:nb], ints.ecore, ints.h, ints.eri).sigma(C)
    assert np.abs(ctx.sigma(C) - ref).max() <= TOL * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("nea,neb", [((3,), (2, 4)), ((2, 4), (3,)), ((3, 5), (2, 4)), ((3,), (3, 4)), ((2, 3), (3,))])
def test_strings_of_several_electron_counts(nea, neb):
    # the operator keeps each spin's electrons: one block per pair of counts
    ints = synth.make_integrals(9, 7)
    rng = np.random.default_rng(7)

    def pick(counts):
        s = np.concatenate([rng.permutation(synth.full_strings(9, ne))[:25] for ne in counts])
        return np.sort(s), np.array([bin(int(x)).count("1") for x in np.sort(s)])
    (a, ca), (b, cb) = pick(nea), pick(neb)
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = rng.normal(size=(len(a), len(b)))
    C /= np.linalg.norm(C)
    ref = np.zeros_like(C)
    one, two = 0.0, 0.0
    for x in nea:
        for y in neb:
            block = np.ix_(ca == x, cb == y)
            sub = sbd_b200.context_from_integrals(ints, a[ca == x], b[cb == y])
            ref[block] = sub.sigma(C[block].ravel()).reshape(ref[block].shape)
            r = sub.rdm(C[block].ravel())
            one, two = one + r[0], two + r[1]
            sub.close()
    assert np.abs(ctx.sigma(C.ravel()) - ref.ravel()).max() <= TOL * np.abs(ref).max()
    assert np.abs(ctx.sigma(C.ravel(), precision=sbd_b200.MIXED) - ref.ravel()).max() <= 2e-5 * np.abs(ref).max()
    got = ctx.rdm(C.ravel())
    assert np.abs(got[0] - one).max() <= 1e-11 and np.abs(got[1] - two).max() <= 1e-11
    ctx.close()


def test_autotune_keeps_the_default_where_no_listed_shape_is_faster():
    # tiles without stages are none of the shapes that can be set: only the gather kernel's groups of 4 and fewer fit
    ints = synth.make_integrals(48, 3)
    b = synth.selected_strings(48, 4, 19990, np.diag(ints.h), 4)
    ctx = sbd_b200.context_from_integrals(ints, b[:60], b)
    C = np.random.default_rng(1).normal(size=ctx.n)

    def alpha_beta_ms():
        ctx.sigma(C)
        ms = []
        for _ in range(5):
            ctx.sigma(C)
            ms.append(ctx.last_sigma_ms()[2])
        return min(ms)
    default = alpha_beta_ms()
    ctx.set_tuning(4, 1024)
    assert alpha_beta_ms() > 1.5 * default
    g, t, ms = ctx.autotune(3)
    assert (g, t) == (0, 0) and ms > 0
    assert alpha_beta_ms() <= 1.2 * default
    ctx.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_integral_stays_where_the_operator_has_it(bad):
    ints, a, b = _system(9, 3, 3, 40, 41, 11)
    for p, q, r, s in ((1, 4, 2, 7), (2, 7, 1, 4)):  # (pq|rs), all eight orders
        for x, y in ((p, q), (q, p)):
            for u, v in ((r, s), (s, r)):
                ints.eri[x, y, u, v] = bad
    C = np.random.default_rng(11).normal(size=len(a) * len(b))
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    got = ctx.sigma(C)
    ref = oracle.Oracle(9, a, b, ints.ecore, ints.h, ints.eri).sigma(C)
    finite = np.isfinite(ref)
    assert finite.any() and not finite.all()
    assert np.array_equal(np.isfinite(got), finite)
    assert np.abs(got[finite] - ref[finite]).max() <= TOL * np.abs(ref[finite]).max()
    ctx.close()


@pytest.mark.parametrize("na,nb", [(193, 257), (257, 194), (256, 256), (65, 449)])
def test_dense_same_spin_product_of_64_wide_tiles(na, nb):
    # at least 16 tiles of 64 x 64 with and without remainders, odd and even rows; then a NaN and an infinity, whose
    # tiles are evaluated again
    ints, a, b = _system(11, 5, 5, na, nb, 60 + na)
    ctx = sbd_b200.context_from_integrals(ints, a, b)
    C = np.random.default_rng(9).normal(size=(na, nb))
    orc = oracle.Oracle(11, a, b, ints.ecore, ints.h, ints.eri)
    ref = orc.sigma(C.ravel())
    assert np.abs(ctx.sigma(C.ravel()) - ref).max() <= TOL * np.abs(ref).max()
    C[na - 1, 70], C[3, nb - 1] = np.nan, np.inf
    got, ref = ctx.sigma(C.ravel()), orc.sigma(C.ravel())
    finite = np.isfinite(ref)
    assert finite.any() and not finite.all()
    assert np.array_equal(np.isfinite(got), finite)
    assert np.abs(got[finite] - ref[finite]).max() <= TOL * np.abs(ref[finite]).max()
    ctx.close()


@pytest.mark.parametrize("na,nb", [(30, 41), (250, 260)])
def test_repeated_alpha_strings(na, nb):
    # only beta strings have to be distinct: tiles, the dense product and the RDM products take such a basis
    ints, a, b = _system(11, 5, 5, na, nb, 80 + na)
    _check(ints, np.concatenate([a, a[:3]]), b, shapes=((0, 0), (16, 128), (4, 128)))
