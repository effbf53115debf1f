"""The kernels that bench.py names beside its numbers follow the library's rules
(CPU only: plain arithmetic on counts)."""
import numpy as np

import bench
from sbd_b200 import synth

OPTIN = 232448


def test_alpha_beta_kernel():
    s = synth.full_strings(12, 4)
    assert bench.ab_tiles(s, 12, OPTIN)
    assert not bench.ab_tiles(np.concatenate([s, s[:1]]), 12, OPTIN)  # a repeated string
    assert not bench.ab_tiles(np.concatenate([s, synth.full_strings(12, 3)[:1]]), 12, OPTIN)  # two electron counts
    # norb 48: 1,128 pairs of eight integrals beside 20,000 strings of C and the zeros behind it
    b = np.array([3 << i for i in range(47)], dtype=np.uint64)
    many = np.unique(np.array([(1 << i) | (1 << j) | (1 << k) for i in range(48) for j in range(i)
                               for k in range(j)], dtype=np.uint64))
    assert len(many) == 17296 and bench.ab_tiles(many, 48, OPTIN) and bench.ab_tiles(b, 48, OPTIN)
    assert not bench.ab_tiles(many, 48, 1128 * 64 + (17296 + 16) * 8 + 127)


def test_same_spin_path():
    full = {0: (495 * 32, 495 * 168), 1: (495 * 32, 495 * 168)}
    assert bench.same_spin_path(0, 495, 495, full, True) == "dense"
    assert bench.same_spin_path(0, 495, 495, full, False) == "rows"  # without tiles
    assert bench.same_spin_path(1, 495, 495, full, True) == "rows"
    assert bench.same_spin_path(0, 12000, 12000, full, True) == "int8"
    assert bench.same_spin_path(1, 12000, 12000, full, True) == "rows"
    wide = {0: (7777 * 150, 7777 * 900), 1: (6001 * 150, 6001 * 900)}
    assert bench.same_spin_path(0, 7777, 6001, wide, True) == "rows"  # odd counts, beyond 4,096 strings
    sparse = {0: (300 * 2, 300 * 5), 1: (300 * 2, 300 * 5)}
    assert bench.same_spin_path(0, 300, 300, sparse, True) == "rows"
