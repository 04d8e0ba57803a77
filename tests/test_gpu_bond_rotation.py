"""Bonds that turn by almost nothing, by angles on either side of the limit of
the rotation's series (0.01 rad per evaluation) and by large ones: the bond's
shear force and bending torque follow the oracle's rotation (sin and cos of
the angle).  Eight steps of FP64 sums: 1e-10 of the largest value."""
import numpy as np
import pytest

from this_studio_b200.scenes import DEMScene, build_dem

from .helpers import oracle_dem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angle", [1e-11, 1e-3, 9.9e-3, 1.01e-2, 0.3])
def test_bond_state_follows_the_rotation(gpu, angle):
    dt = 1e-4
    r = 0.01
    pos = np.array([[0.0, 0, 0], [1.99 * r, 0, 0], [1.99 * r, 1.99 * r, 0]])
    w = angle / (0.5 * dt)  # twist about the bond per evaluation
    sc = DEMScene(name="spin", position=pos, radius=np.full(3, r), density=np.full(3, 2500.0),
                  material=np.zeros(3, np.int32), velocity=np.array([[0.0, 0, 0], [0, 0.02, 0.01], [0.01, 0, 0.02]]),
                  hertz=[(0, 0, 1e4, 1e4, 0.9, 0.0, 0.0, 0.3, 0.0, 0.0)], bonded=[(0, 0, 1.0, 1e3, 2.5, 0.0, 0.0, 0.0)],
                  minb=(-0.1,) * 3, maxb=(0.1,) * 3, gravity=(0, 0, 0), dt=dt)
    sc.angvel = np.array([[w, 0.3, 0.1], [w, w, -0.2], [0.2, w, 0.1]])
    sc.bond_initial_contacts = True
    g, o = build_dem(sc, "fp64"), oracle_dem(sc)
    for n in (1, 7):
        g.step(n)
        o.step(n)
    a, b = g.getBondedInteraction(), o.bonds()
    assert a["isBonded"].all()
    for k, q in (("shearForce", "shear_force"), ("bendingTorque", "bending_torque")):
        assert np.abs(a[k] - b[q]).max() <= 1e-10 * max(np.abs(b[q]).max(), 1e-300), k
    x, y = g.getBall(), o.balls()
    assert np.abs(x["torque"] - y["torque"]).max() <= 1e-10 * np.abs(y["torque"]).max()
