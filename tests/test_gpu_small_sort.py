"""The one-block Morton sort at the edges of its sizes, with ties: the tree, and so the FP64
accelerations, are the oracle's bit for bit, and the pass kernels' (10-bit digits)."""

import os

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 1023, 1024, 1025, 4095, 4096, 4097])
@pytest.mark.parametrize("morton63", [False, True])
def test_bit_exact(oracle, n, morton63):
    rng = np.random.default_rng(n)
    pos, mass = rng.normal(size=(n, 3)) ** 3, rng.uniform(0.1, 1.0, n)
    pos[n // 2: n // 2 + n // 8] = pos[0]  # coincident: one code, ordered by index
    pos[: n // 16, 0] = np.abs(pos[:, 0]).max()  # the last lane of an axis
    f = oracle.lbvh_accelerations_k63 if morton63 else oracle.lbvh_accelerations
    ref = f(pos, mass, 1.0, 0.05, 0.8, threads=os.cpu_count() or 1)
    got = gb.GpuLbvh(1.0, 0.05, 0.8, precision="f64", morton63=morton63).accelerations(pos, mass=mass)
    assert np.array_equal(got, ref)
    if not morton63:
        wide = gb.GpuLbvh(1.0, 0.05, 0.8, precision="f64", radix_bits=10).accelerations(pos, mass=mass)
        assert np.array_equal(got, wide)
