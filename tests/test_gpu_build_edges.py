"""The build at the edges of its blocks and tiles (256, 4,096 leaves) and on chains: blocks that
leave many subtrees to the second pass, folds of every side and child kind in one round."""

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu


def _check(oracle, codes, rng):
    n = codes.shape[0]
    pos, mass = rng.normal(size=(n, 3)), rng.uniform(0.1, 1.0, n)
    left, right, parent = oracle.reference_karras(codes)
    agg = oracle.reference_aggregate(left, right, pos, mass)
    got = gb.stage_build(codes, pos, mass)
    for name, ref in (("left", left), ("right", right), ("parent", parent)):
        assert np.array_equal(got[name], ref), name
    for name in ("aabb_min", "aabb_max", "com", "mass"):
        assert np.array_equal(got[name], agg[name]), name


@pytest.mark.parametrize("n", [2, 3, 255, 257, 4095, 4097, 65537, 140001])
def test_sizes(oracle, n):
    rng = np.random.default_rng(n)
    codes = np.sort((rng.integers(0, 1 << 10, (n, 3)) ** 2 >> 10) @ np.array([1, 1 << 10, 1 << 20])).astype(np.uint32)
    _check(oracle, codes, rng)


@pytest.mark.parametrize("groups", [5, 16, 40, 63])
def test_chains(oracle, groups):
    # groups of codes 0, 1, 3, 7, ... 2^23 - 1 above a common base, placed so that each block
    # of 256 leaves starts after a group's first code: every later code of the group is a
    # subtree of its own there, 23 a block
    copies = [20] + [10] * 22 + [16]
    codes = np.concatenate([np.repeat((g << 24) + (1 << np.arange(24)) - 1, copies) for g in range(groups)])[20:]
    _check(oracle, codes.astype(np.uint32), np.random.default_rng(groups))
