"""The hydro force where h varies: each target scans only as far as the largest h around it
reaches, so a particle of large h far from the others' cells must still find, and be found
by, every pair within the support of either."""

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 600, 3000])
@pytest.mark.parametrize("spread", [1.0, 8.0, 200.0])
@pytest.mark.parametrize("shift", [0.0, 1e4])
def test_hydro_matches_oracle(oracle, n, spread, shift):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 3)) + shift
    vel, mass, u = rng.normal(size=(n, 3)), rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 1.5, n)
    h = 0.9 / n ** (1 / 3) * np.exp(rng.uniform(-0.5, 0.5, n))
    h[:: max(n // 7, 1)] *= spread  # a few of much larger support
    h = np.minimum(h, 1.0)
    rho = rng.uniform(0.5, 2.0, n)
    s = gb.GpuGravitySph(1.0, 0.01, 0.5, sph=dict(eos="adiabatic"))
    acc, dudt = s.hydro(pos, vel, mass, rho, h, u)
    ref, ref_du = oracle.sph_hydro(pos, vel, mass, rho, h, u, eos=1, eos_param=5.0 / 3.0)
    # sums in another order: rounding of the terms, against the RMS of the sums
    assert np.abs(acc - ref).max() <= 1e-11 * max(np.sqrt((ref ** 2).mean()), 1e-300)
    assert np.abs(dudt - ref_du).max() <= 1e-11 * max(np.sqrt((ref_du ** 2).mean()), 1e-300)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_cells_beyond_the_integer_range(oracle, axis):
    # positions of 1e10 cells: the cell numbers clamp at both ends of a 32-bit integer, where
    # a neighbour's number cannot be formed
    rng = np.random.default_rng(axis)
    n = 90
    pos = rng.random((n, 3)) * 4e-3
    pos[:30, axis] += 1e7
    pos[30:60, axis] -= 1e7
    vel, mass, u = rng.normal(size=(n, 3)), rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 1.5, n)
    h, rho = np.full(n, 1e-3) * rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 2.0, n)
    s = gb.GpuGravitySph(1.0, 0.01, 0.5, sph=dict(eos="adiabatic"))
    acc, dudt = s.hydro(pos, vel, mass, rho, h, u)
    ref, ref_du = oracle.sph_hydro(pos, vel, mass, rho, h, u, eos=1, eos_param=5.0 / 3.0)
    assert (np.abs(ref).max(axis=1) > 0).sum() > n // 2  # pairs in all three groups
    assert np.abs(acc - ref).max() <= 1e-11 * np.sqrt((ref ** 2).mean())
    assert np.abs(dudt - ref_du).max() <= 1e-11 * np.sqrt((ref_du ** 2).mean())
