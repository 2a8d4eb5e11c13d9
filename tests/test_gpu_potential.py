"""The FP64 potential sum at the edges of its tiles, against the oracle's pair sum."""

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 127, 128, 129, 255, 256, 257, 513, 1025, 5121])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_tile_edges(oracle, n, eps):
    pos, _, mass = oracle.fixture_cluster(n, n)
    u = gb.GpuLbvh(1.0, eps, 0.5).potential_energy(pos, mass=mass)
    ref = oracle.potential_serial(pos, mass, 1.0, eps)
    # terms of one sign: the relative error is a few roundings of the longest chain of sums
    assert abs(u - ref) <= 1e-12 * abs(ref)


def test_extreme_distances(oracle):
    pos = np.array([[0, 0, 0], [1e-150, 0, 0], [1e150, 0, 0], [1.0, 2.0, 3.0]])
    mass = np.array([1.0, 2.0, 3.0, 4.0])
    s = gb.GpuLbvh(1.0, 0.0, 0.5)
    ref = oracle.potential_serial(pos, mass, 1.0, 0.0)
    assert abs(s.potential_energy(pos, mass=mass) - ref) <= 1e-12 * abs(ref)
    pos[1] = pos[0]  # coincident, unsoftened: the pair's energy is infinite
    assert s.potential_energy(pos, mass=mass) == -np.inf


def test_rounding_of_many_partial_sums():
    # Against 80-bit sums. The terms' roundings average out over 4e7 pairs, so what is left is
    # the last rounding (1.1e-16 at most) and the sum of the blocks' partials, which a plain
    # sum rounds to 4.6e-16 on average and a compensated one not at all.
    errors = []
    for seed in range(3):
        st = gb.ic.plummer(9000, seed)
        p, m = st.pos.astype(np.longdouble), st.mass.astype(np.longdouble)
        u = np.longdouble(0.0)
        for i in range(0, 9000, 250):
            d2 = ((p[i:i + 250, None, :] - p[None, i:, :]) ** 2).sum(axis=2) + np.longdouble(0.01 * 0.01)
            w = m[i:i + 250, None] * m[None, i:] / np.sqrt(d2)
            u -= np.triu(w, 1).sum()
        errors.append(float(abs((gb.GpuLbvh(1.0, 0.01, 0.5).potential_energy(st) - u) / u)))
    assert np.mean(errors) <= 2.0 ** -53, errors
