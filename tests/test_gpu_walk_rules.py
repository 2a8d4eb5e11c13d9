"""The FP32 walk's opening decisions where its rules change: around the opening angle from
which the inside rule can bind (2 / sqrt 3), and at the edges of its target groups, lists
and batches. Every target takes exactly the oracle's terms, so the counts are equal."""

import os

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


def _check(oracle, pos, mass, theta, eps=0.05, **kw):
    s = gb.GpuLbvh(1.0, eps, theta, stats=True, **kw)
    got = s.accelerations(pos, mass=mass)
    st = s.stats()
    ref, cnt = oracle.lbvh_accelerations(pos, mass, 1.0, eps, theta, threads=THREADS, stats=True)
    assert (st["leaf_interactions"], st["far_interactions"]) == (cnt["leaf"], cnt["far"])
    # FP32 terms and sums: the parity gates of tests/test_gpu_walk.py
    err = oracle.per_particle_rel_err(got, ref)
    assert np.median(err) <= 1e-6 and np.percentile(err, 99) <= 1e-5, (np.median(err), err.max())


@pytest.mark.parametrize("theta", [0.56, 0.58, 1.0, 1.1499, 1.15, 1.1547, 1.16, 1.5])
def test_inside_rule(oracle, theta):
    pos, _, mass = oracle.fixture_cluster(3, 3000)
    # flat and needle-shaped boxes, coincident particles (zero-size boxes), massless ones
    pos[:700, 2] = 0.0
    pos[700:900, 1:] = 0.25
    pos[900:940] = pos[900]
    mass[1000:1100] = 0.0
    for group in (8, 16, 32):
        _check(oracle, pos, mass, theta, walk_group=group)


@pytest.mark.parametrize("n", [2, 3, 5, 9, 31, 32, 33, 63, 65, 129, 1025])
@pytest.mark.parametrize("theta", [0.0, 0.3, 0.8])
def test_list_edges(oracle, n, theta):
    pos, _, mass = oracle.fixture_cluster(n, n)
    mass[: n // 4] = 0.0  # NaN thresholds: decided in FP64
    for group in (8, 16, 32):
        _check(oracle, pos, mass, theta, walk_group=group)


@pytest.mark.parametrize("n", [33, 1025])
def test_list_edges_quad(oracle, n):
    pos, _, mass = oracle.fixture_cluster(n, n)
    ref = oracle.lbvh_accelerations_quad(pos, mass, 1.0, 0.05, 0.6, threads=THREADS)
    for group in (8, 16, 32):
        got = gb.GpuLbvh(1.0, 0.05, 0.6, multipole="quad", walk_group=group).accelerations(pos, mass=mass)
        err = oracle.per_particle_rel_err(got, ref)
        assert np.median(err) <= 1e-6 and np.percentile(err, 99) <= 1e-5


@pytest.mark.parametrize("theta", [0.0, 1e-300, 1e-3, 1.1499, 1.15, 1.1547, 1.2, 2.0, 5.0, 40.0, 1e9, np.inf])
@pytest.mark.parametrize("scale", [1.0, 1e-60, 1e-75, 1e60, 1e71])
def test_fp64_thresholds(oracle, theta, scale):
    # the FP64 walk's squared-distance thresholds: open everything, beyond the box's corners
    # where the inside rule binds, and squares that leave the range of a double
    pos, _, mass = oracle.fixture_cluster(4, 700)
    pos[:150, 2] = 0.0
    pos[150:200, 1:] = 0.25
    pos[200:220] = pos[200]
    mass[300:330] = 0.0
    pos = pos * scale
    got = gb.GpuLbvh(1.0, 0.0 if scale == 1.0 else 0.05 * scale, theta, precision="f64").accelerations(pos, mass=mass)
    ref = oracle.lbvh_accelerations(pos, mass, 1.0, 0.0 if scale == 1.0 else 0.05 * scale, theta, threads=THREADS)
    assert np.array_equal(got, ref, equal_nan=True)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 100, 700])
def test_warp_node_visits(oracle, n):
    # At theta 0 every target goes through the whole tree: a warp's visits are the tree's nodes
    # (FP64, 32 targets a warp) or its sibling pairs (FP32), each counted once a warp.
    pos, _, mass = oracle.fixture_cluster(n, n)
    kw = dict(stats=True)
    s = gb.GpuLbvh(1.0, 0.05, 0.0, precision="f64", **kw)
    ref = oracle.lbvh_accelerations(pos, mass, 1.0, 0.05, 0.0, threads=THREADS)
    assert np.array_equal(s.accelerations(pos, mass=mass), ref)
    assert s.stats()["warp_node_visits"] == -(-n // 32) * (2 * n - 1)
    for group in (8, 16, 32):
        s = gb.GpuLbvh(1.0, 0.05, 0.0, walk_group=group, **kw)
        s.accelerations(pos, mass=mass)
        assert s.stats()["warp_node_visits"] == -(-n // group) * (n - 1)


def test_targets_across_a_morton_jump(oracle):
    # Groups of targets from tight clumps either side of the cube's middle planes: their boxes
    # are wide, and clumps that are undecided for a group lie close to some of its targets.
    # Coordinates relative to the box's centre would lose bits (largest error of a particle
    # 4e-5 at least in each of these walks); the near list keeps them (7.8e-6 at most, which is
    # that of entries accepted for the whole group).
    n = 8000
    rng = np.random.default_rng(11)
    c = (rng.integers(0, 2, (n, 3)) - 0.5) * 2e-4 * rng.uniform(0.1, 1, (n, 1))
    pos = c + rng.normal(size=(n, 3)) * 2e-5
    pos[::9] = rng.uniform(-1, 1, pos[::9].shape)
    mass = rng.uniform(0.5, 1.5, n) / n
    ref = gb.GpuLbvh(1.0, 0.02, 0.7, precision="f64", morton63=True).accelerations(pos, mass=mass)
    size = np.linalg.norm(ref, axis=1)
    act = np.sort(np.random.default_rng(1).choice(n, n // 50, replace=False)).astype(np.int64)
    for group in (8, 16, 32):
        s = gb.GpuLbvh(1.0, 0.02, 0.7, morton63=True, walk_group=group)
        err = np.linalg.norm(s.accelerations(pos, mass=mass) - ref, axis=1) / size
        assert err.max() <= 2e-5, (group, err.max())
    got = s.accelerations_active(pos, act, mass=mass)[act]
    err = np.linalg.norm(got - ref[act], axis=1) / size[act]
    assert err.max() <= 2e-5, err.max()
