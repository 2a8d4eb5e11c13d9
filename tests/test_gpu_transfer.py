"""Copies between callers' arrays and the device at the edges of the staging slots (64 KB
direct, 1 MB slots, 8 of them in turn), from several threads, and with pinned arrays."""

import threading

import numpy as np
import pytest

import galaxy_b200 as gb

pytestmark = pytest.mark.gpu


def _round_trip(n, seed):
    rng = np.random.default_rng(seed)
    st = gb.State(rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), rng.uniform(0.1, 1.0, n))
    r = gb.GpuResidentLeapfrog(1.0, 0.05, 0.7, morton63=True)
    for _ in range(2):
        r.upload(st)
        out = r.snapshot()
        assert np.array_equal(out.pos, st.pos) and np.array_equal(out.vel, st.vel)
    return st


@pytest.mark.parametrize("n", [2, 2730, 2731, 43690, 43691, 349525, 349526, 400001])
def test_round_trip(n):
    _round_trip(n, n)


def test_threads():
    errors = []

    def work(k):
        try:
            for i in range(3):
                _round_trip(30000 + 50000 * k, 10 * k + i)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_pinned_arrays():
    st = gb.ic.disk_galaxy(60000, 3)
    p = gb.PinnedState.from_state(st)
    s = gb.GpuLbvh(1.0, 0.05, 0.6)
    a = s.accelerations(st)
    s._ck(gb._lib.lib().gx_accelerations(s._h, len(st), gb._ptr(p.pos), gb._ptr(p.mass), gb._ptr(p.acc)))
    assert np.array_equal(a, p.acc)
