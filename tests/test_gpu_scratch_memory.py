"""Device memory of what speeds a context up: the dense same-spin operators
(csrc/same_dense.cu) are made by the FP64 sigma, not by the set-up, and given
back with the choice of the rows kernels; without room for them, or for the
alpha-beta tiles (csrc/ab_mma.cu), the kernels that need none run."""
import numpy as np
import pytest

import sbd_b200
from sbd_b200 import synth

pytestmark = pytest.mark.gpu

TOL = 1e-12  # the bound of the sigma parity tests
MB = 1 << 20
OPERATORS = 8 * (4060 ** 2 + 3 * 4)  # bytes: rows padded to even lengths


def _context():
    # 4,060 x 3 strings: vectors of 0.1 MB beside 132 MB of operators
    ints = synth.make_integrals(30, 6)
    a = synth.full_strings(30, 3)
    ctx = sbd_b200.context_from_integrals(ints, a, a[:3])
    ctx.tables(0)
    return ctx, np.random.default_rng(6).normal(size=ctx.n)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def test_operators_are_made_by_the_fp64_sigma_and_given_back():
    ctx, C = _context()
    free0 = _free()
    ctx.hii()
    assert free0 - _free() < OPERATORS // 2
    got = ctx.sigma(C)
    free1 = _free()
    assert free0 - free1 >= OPERATORS
    ctx.set_fp64_same_spin(1)
    assert _free() - free1 >= OPERATORS
    ref = ctx.sigma(C)
    assert free0 - _free() < OPERATORS // 2
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    ctx.set_fp64_same_spin(0)
    assert np.abs(ctx.sigma(C) - ref).max() <= TOL * np.abs(ref).max()
    assert free0 - _free() >= OPERATORS
    ctx.close()


def test_rows_kernels_without_room_for_the_operators():
    import torch
    small, _ = _context()  # loads every kernel
    small.sigma(np.ones(small.n))
    small.rdm(np.ones(small.n) / small.n ** 0.5)
    small.close()
    ctx, C = _context()
    torch.cuda.empty_cache()
    taken = torch.empty(_free() - 96 * MB, dtype=torch.uint8, device="cuda")
    ctx.hii()
    got = ctx.sigma(C)
    runs = [ctx.davidson(C / np.linalg.norm(C), 1, 4, 1e-10)[:2]]
    e, w, _ = sbd_b200.davidson_batch([ctx], [C / np.linalg.norm(C)], 1, 4, 1e-10)
    runs.append((e[0], w[0]))
    del taken
    torch.cuda.empty_cache()
    ctx.set_fp64_same_spin(1)
    ref = ctx.sigma(C)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    for e, w in runs:  # the energies are the Rayleigh quotients of the vectors
        s = ctx.sigma(w)
        assert abs(e - w @ s) <= TOL * np.abs(s).max() * np.abs(w).sum()
    ctx.close()


def test_gather_kernel_without_room_for_the_tiles():
    import torch

    ints = synth.make_integrals(20, 6)
    b = synth.full_strings(20, 6)[:26000]  # some 14 MB of tiles, allocated last

    def build(leave=None):
        ctx = sbd_b200.context_from_integrals(ints, b[:2], b)
        torch.cuda.empty_cache()
        free = _free()
        taken = torch.empty(free - leave, dtype=torch.uint8, device="cuda") if leave else None
        assert sbd_b200.lib().sbdgpu_build_tables(ctx._h) == 0
        del taken
        torch.cuda.empty_cache()
        return ctx, free - _free()
    ctx, size = build()
    C = np.random.default_rng(6).normal(size=ctx.n)
    W = C / np.linalg.norm(C)
    ref, (ref1, ref2) = ctx.sigma(C), ctx.rdm(W)
    ctx.close()
    ctx, without = build(size - 6 * MB)
    assert without < size - 6 * MB
    assert np.abs(ctx.sigma(C) - ref).max() <= TOL * np.abs(ref).max()
    one, two = ctx.rdm(W)
    assert np.abs(one - ref1).max() <= 1e-11 and np.abs(two - ref2).max() <= 1e-11
    ctx.close()


def test_scalar_rdm_kernels_without_room_for_the_products():
    import torch

    ints = synth.make_integrals(20, 7)
    b = synth.full_strings(20, 6)[:26000]  # panels of 1 GiB
    ctx = sbd_b200.context_from_integrals(ints, b[:2], b)
    W = np.random.default_rng(7).normal(size=ctx.n)
    W /= np.linalg.norm(W)
    ref1, ref2 = ctx.rdm(W)
    torch.cuda.empty_cache()
    taken = torch.empty(_free() - 256 * MB, dtype=torch.uint8, device="cuda")
    one, two = ctx.rdm(W)
    del taken
    torch.cuda.empty_cache()
    assert np.abs(one - ref1).max() <= 1e-11 and np.abs(two - ref2).max() <= 1e-11
    ctx.close()
