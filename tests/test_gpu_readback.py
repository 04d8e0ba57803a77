"""Read-back of ball, clump and bond state through the page-locked staging:
single records, a few thousand, and arrays larger than a half of it, every
value exact and in the caller's order."""
import numpy as np
import pytest

from this_studio_b200 import DEMSolver, scenes
from this_studio_b200.scenes import build_dem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4099, 720_001])  # 17.3 MB a vector: more than a half of 16 MB
def test_ball_state_comes_back_exactly(gpu, n):
    rng = np.random.default_rng(n)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    i = np.arange(n)
    pos = np.stack([i % k, i // k % k, i // (k * k)], 1) * 0.03 + rng.uniform(0, 0.01, (n, 3))
    vel, w = rng.normal(0, 1, (n, 3)), rng.normal(0, 1, (n, 3))
    s = DEMSolver()
    s.addBalls(pos, vel, w, 0.005, 2500.0, 0)
    s.initialize((-0.1,) * 3, (k * 0.03 + 0.1,) * 3, (0, 0, -9.81), 1e-5)
    got = s.getBall()
    for key, a in (("position", pos), ("velocity", vel), ("angularVelocity", w)):
        np.testing.assert_array_equal(got[key], a)
    assert not got["force"].any() and not got["torque"].any()
    s.step(3)
    assert np.abs(s.getBall()["velocity"][:, 2] - (vel[:, 2] - 9.81 * 3e-5)).max() < 1e-12


def test_clump_and_bond_state_comes_back_whole(gpu):
    sc = scenes.bonded_beam_clumps(nx=30, ny=5, nz=5, n_clumps=40)
    g = build_dem(sc, "fp64")
    b = g.getBondedInteraction()
    assert b["isBonded"].all() and not b["normalForce"].any()
    p = sc.position
    mid = 0.5 * (p[b["objectPointed"]] + p[b["objectPointing"]])
    np.testing.assert_array_equal(b["point"], mid)
    np.testing.assert_allclose(np.linalg.norm(b["normal"], axis=1), 1.0, rtol=1e-14)
    c = g.getClump()
    np.testing.assert_array_equal(c["position"], [k["centroid"] for k in sc.clumps])
    np.testing.assert_array_equal(c["orientation"], np.tile([1.0, 0, 0, 0], (40, 1)))


def test_read_back_takes_no_device_memory(gpu):
    """A scene that fills the device can still be read: the getters allocate
    nothing there (the staging is host memory)."""
    from .test_zz_no_alloc import _Pool

    rng = np.random.default_rng(3)
    n = 200_000
    pos = np.stack(np.unravel_index(np.arange(n), (59, 59, 59)), 1) * 0.02 + rng.uniform(0, 0.005, (n, 3))
    s = DEMSolver()
    s.addBalls(pos, None, None, 0.005, 2500.0, 0)
    s.initialize((-0.1,) * 3, (1.3,) * 3, (0, 0, -9.81), 1e-5)
    g = build_dem(scenes.bonded_beam_clumps(nx=30, ny=5, nz=5, n_clumps=40), "fp64")
    pool = _Pool()
    used = pool.attr(pool.USED)
    pool.reset_high()
    np.testing.assert_array_equal(s.getBall()["position"], pos)
    g.getBondedInteraction()
    g.getClump()
    assert pool.attr(pool.USED_HIGH) <= used  # (other scenes' memory may be given back meanwhile)
