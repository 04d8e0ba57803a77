"""The pair-parallel force evaluation and the list build at the sizes where
their forms change: crowded stencil rows (more candidates than a row's mask
holds), rows that outgrow their capacity, scenes on either side of the list
build's and the finish's lane limits, walls whose balls touch few or many
triangles, and springs that end with their contact.  Against the FP64 oracle;
FP64 sums in another order differ by their rounding (1e-11 relative leaves a
factor 1000 over the 1e-14 of an evaluation for the steps to amplify it)."""
import numpy as np
import pytest

from this_studio_b200 import scenes
from this_studio_b200.scenes import DEMScene, build_dem, hertz_params

from .helpers import oracle_dem, pair_keys, rel_err

pytestmark = pytest.mark.gpu


def _crowd(n_small, n_big, seed=4):
    """A few large balls (first, so that they point at everything near) among
    many small ones: cells as wide as the large balls hold dozens of candidates."""
    rng = np.random.default_rng(seed)
    L = 0.1 * (n_small / 1500.0) ** (1.0 / 3.0)
    pos = rng.uniform(0, L, (n_big + n_small, 3))
    rad = np.r_[np.full(n_big, 0.012), rng.uniform(0.0012, 0.002, n_small)]
    Es, Gs = hertz_params(1e6, 0.3)
    sc = DEMScene(name="crowd", position=pos, radius=rad, density=np.full(len(rad), 2500.0),
                  material=np.zeros(len(rad), np.int32), velocity=rng.normal(0, 0.05, pos.shape),
                  hertz=[(0, 0, Es, Gs, 0.8, 0.2, 0.1, 0.3, 0.05, 0.05)], minb=(-0.03,) * 3, maxb=(L + 0.03,) * 3,
                  dt=1e-6)
    return sc


def _compare(sc, steps, prec="fp64", tol=1e-11):
    g, o = build_dem(sc, prec), oracle_dem(sc)
    if getattr(sc, "constant_force", None) is not None:
        o.set_constant_force(sc.constant_force)
    for n in steps:
        g.step(n)
        o.step(n)
        p, q = g.getPairs(0), o.pairs(0)
        np.testing.assert_array_equal(pair_keys(p["objectPointed"], p["objectPointing"]), pair_keys(q["a"], q["b"]))
        b, c = g.getBall(), o.balls()
        for k, r in (("position", "pos"), ("velocity", "vel"), ("angularVelocity", "angvel"), ("force", "force")):
            assert rel_err(b[k], c[r]) < tol, (n, k)
    return g, o


@pytest.mark.parametrize("n_small,n_big", [(1500, 6), (20000, 40)])
def test_crowded_rows_and_regrowth(gpu, n_small, n_big):
    _compare(_crowd(n_small, n_big), (3, 9))


@pytest.mark.parametrize("side", [25, 26])  # 15,625 and 17,576: either side of the build's lane limit
def test_list_build_forms_agree_with_the_oracle(gpu, side):
    _compare(scenes.dem_pack(n_side=side), (5, 6))


@pytest.mark.parametrize("n", [900, 17_000])  # balls: either side of the build's lane limit
def test_pairs_at_the_cut_off(gpu, n):
    """Couples of balls at the lists' reach, 1.1 (ra + rb), to within 1e-11 of
    it and more: an FP32 distance cannot tell these in from out.  The positions
    are the reference's input, so only the square's FP64 rounding (below 1e-15)
    separates the two sides, and the nearest couple is 1e-12 from the line.  One
    larger ball apart widens the cells (twice the largest radius) to the couples'
    reach, so that no couple lies beyond the stencil."""
    rng = np.random.default_rng(7)
    m = n // 2
    side = int(np.ceil(m ** (1.0 / 3.0)))
    at = np.stack(np.unravel_index(np.arange(m), (side,) * 3), 1) * 0.08 + 3.0
    ra, rb = rng.uniform(0.004, 0.01, (2, m))
    u = rng.normal(size=(m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    e = 10.0 ** rng.uniform(-12, -4, m) * rng.choice([-1, 1], m)
    b = at + u * (1.1 * (ra + rb) * (1 + e))[:, None]
    pos = np.concatenate([at, b, [[2.95] * 3]])
    rad = np.r_[ra, rb, 0.012]
    Es, Gs = hertz_params(1e6, 0.3)
    sc = DEMScene(name="cut-off", position=pos, radius=rad, density=np.full(2 * m + 1, 2500.0),
                  material=np.zeros(2 * m + 1, np.int32), velocity=np.zeros_like(pos),
                  hertz=[(0, 0, Es, Gs, 0.8, 0.2, 0.1, 0.3, 0.05, 0.05)], minb=(2.9,) * 3,
                  maxb=(3.1 + 0.08 * side,) * 3, dt=1e-9)
    g = build_dem(sc, "fp64")
    g.step(1)
    p = g.getPairs(0)
    d2 = ((at - b) ** 2).sum(1)
    inside = np.flatnonzero((1.1 * (ra + rb)) ** 2 >= d2)
    assert 0.4 * m < len(inside) < 0.6 * m
    ab = np.sort(np.stack([p["objectPointed"], p["objectPointing"]]), axis=0)
    np.testing.assert_array_equal(np.sort(pair_keys(*ab)), pair_keys(inside, inside + m))


@pytest.mark.parametrize("n", [30_000, 36_000, 70_000])  # 29,791 and 35,937: either side of the finish's lane limit; sparse walls
def test_finish_forms_agree_with_the_oracle(gpu, n):
    sc = scenes.dem_drop_poly(n, seed=2)
    rng = np.random.default_rng(1)
    sc.position[:, 2] -= 0.1 * 0.005 * np.sqrt(3.0)
    sc.position[:, :2] *= 0.8  # neighbours in a row touch
    sc.velocity = rng.normal(0, 0.2, sc.position.shape) + np.array([0, 0, -0.5])
    _compare(sc, (6,))


def test_springs_end_with_their_contact(gpu):
    """Spheres that touch, slide and part: a pair apart keeps neither its force
    nor its springs, and a restored state evaluates afresh."""
    sc = scenes.dem_pack(n_side=5, overlap=0.002, vel=0.6)
    g, o = _compare(sc, (1, 7, 12, 30))
    p, q = g.getPairs(0), o.pairs(0)
    apart = np.linalg.norm(p["force"], axis=1) == 0
    assert apart.any() and not apart.all()
    assert np.abs(p["sliding"][apart]).max() == 0 and np.abs(p["torqueB"][apart]).max() == 0
    snap = g.snapshot()
    g.step(13)
    a = g.getBall()
    snap.restore()
    g.step(13)
    for k, v in g.getBall().items():
        np.testing.assert_array_equal(v, a[k])


@pytest.mark.parametrize("segments", [(4, 1), (10, 3), (40, 40)])  # 16 triangles with the caps, 80, 3,280
def test_walls_of_few_and_many_triangles(gpu, segments):
    """Balls pressed onto a capped cylinder: up to dozens of candidate
    triangles per ball on the fine mesh, a handful on the coarse ones."""
    rng = np.random.default_rng(9)
    mesh = scenes.cylinder_mesh((0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 0.05, 0.08, *segments)
    r = 0.006
    t = rng.uniform(0, 2 * np.pi, 120)
    pos = np.stack([(0.05 + 0.9 * r) * np.cos(t), (0.05 + 0.9 * r) * np.sin(t), rng.uniform(-0.03, 0.03, 120)], 1)
    keep = [0]
    for k in range(1, len(pos)):
        if np.linalg.norm(pos[keep] - pos[k], axis=1).min() > 2.0 * r:
            keep.append(k)
    pos = pos[keep]
    Es, Gs = hertz_params(1e7, 0.3)
    sc = DEMScene(name="cyl", position=pos, radius=np.full(len(pos), r), density=np.full(len(pos), 2500.0),
                  material=np.zeros(len(pos), np.int32), velocity=rng.normal(0, 0.1, pos.shape) - 2.0 * pos,
                  hertz=[(0, 0, Es, Gs, 0.8, 0.2, 0.1, 0.3, 0.05, 0.05)],
                  walls=[dict(mesh, position=(0.0, 0.0, 0.0), material=0)], minb=(-0.1,) * 3, maxb=(0.1,) * 3, dt=5e-6)
    g, o = _compare(sc, (1, 10), tol=1e-10)
    p, q = g.getPairs(1), o.pairs(1)
    np.testing.assert_array_equal(pair_keys(p["objectPointed"], p["objectPointing"]), pair_keys(q["a"], q["b"]))
    assert len(p["objectPointed"]) > 0


def _boxed(n_side, faces=6, **kw):
    """A touching pack pressed against the faces of its box (two triangles a
    face, first the floor): a ball on an edge or in a corner has four or six
    candidate triangles."""
    sc = scenes.dem_pack(n_side=n_side, **kw)
    r = sc.radius[0]
    (x0, y0, z0), (x1, y1, z1) = sc.position.min(0) - 0.97 * r, sc.position.max(0) + 0.97 * r
    v = np.array([[x, y, z] for z in (z0, z1) for x, y in ((x0, y0), (x1, y0), (x1, y1), (x0, y1))])
    q = [(0, 1, 2, 3), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7), (4, 5, 6, 7)][:faces]
    t = np.array([(a, b, c) for a, b, c, _ in q] + [(a, c, d) for a, _, c, d in q], np.int32)
    sc.walls = [dict(vertices=v, tri0=t[:, 0], tri1=t[:, 1], tri2=t[:, 2], position=(0.0, 0.0, 0.0), material=0)]
    return sc


@pytest.mark.parametrize("n_side", [2, 9, 41])  # every ball in a corner; a small scene; 68,921: the sparse form
def test_balls_on_the_edges_and_in_the_corners_of_a_box(gpu, n_side):
    """Wall pairs as the oracle's, and the springs they carry over the steps
    (rolling and torsion among them); 1e-9 against the oracle as the pack's
    contacts amplify the rounding of an evaluation."""
    g, o = _compare(_boxed(n_side), (1, 9) if n_side < 40 else (2,), tol=1e-9)
    p, q = g.getPairs(1), o.pairs(1)
    np.testing.assert_array_equal(pair_keys(p["objectPointed"], p["objectPointing"]), pair_keys(q["a"], q["b"]))
    assert np.bincount(p["objectPointed"]).max() > 2
    for k in ("sliding", "rolling", "torsion"):
        assert rel_err(p[k], q[k]) < 1e-8, k


def test_corners_do_not_hold_up_a_step(gpu):
    """The few balls with more than two candidate triangles are not what a step
    waits for: a boxed pack takes 2.5 times the step of one on a floor alone
    (its six faces' contacts included), and took 5.2 times when each such ball
    searched and settled its contacts in one thread."""
    import time

    def step_us(sc):
        s = build_dem(sc, "mixed")
        best = 1e9
        for _ in range(6):
            t0 = time.perf_counter()
            s.step(200)
            s.getBall()
            best = min(best, time.perf_counter() - t0)
        return best

    assert step_us(_boxed(16)) < 3.7 * step_us(_boxed(16, faces=1))


@pytest.mark.parametrize("size,steps,limit", [((30, 5), 20, 1.0e-9), ((30, 5), 60, 3.5e-9), ((60, 10), 110, 4.2e-9)])
def test_mixed_contacts_of_like_spheres_keep_their_error(gpu, size, steps, limit):
    """A steel beam in mixed precision against FP64.  All its contacts round the
    law's coefficients alike, so their rounding does not average out: in the
    reference's order of operations the velocities are off by 5.7e-10, 2.7e-9
    and 3.2e-9, a third more is allowed (with tabulated damping 1.8e-9, 4.5e-9
    and 5.7e-9)."""
    nx, ny = size
    sc = scenes.bonded_beam_clumps(nx=nx, ny=ny, nz=ny, n_clumps=50, seed={20: 1, 60: 1, 110: 3}[steps])
    v = {}
    for prec in ("fp64", "mixed"):
        g = build_dem(sc, prec)
        g.step(steps)
        v[prec] = g.getBall()["velocity"]
    assert rel_err(v["mixed"], v["fp64"]) < limit


def test_device_memory_of_a_scene(gpu):
    """What a scene takes per ball at the default capacities (16 pairs, 16
    reverse entries, 8 wall candidates): 2,508 B of pair rows and lists, 584 B
    of wall rows and some 380 B of state and sort (111 of them for a cell of
    this domain each).  The torques on the pointed balls have no buffer of their
    own, which would be 512 B."""
    from .test_zz_no_alloc import _Pool

    n = 200_000
    pos = np.stack(np.unravel_index(np.arange(n), (59, 59, 59)), 1) * 0.02
    sc = DEMScene(name="grid", position=pos, radius=np.full(n, 0.005), density=np.full(n, 2500.0),
                  material=np.zeros(n, np.int32), hertz=[(0, 0, 1e7, 1e7, 0.8, 0.0, 0.0, 0.3, 0.0, 0.0)],
                  minb=(-0.1,) * 3, maxb=(1.3,) * 3, dt=1e-5)
    build_dem(sc, "fp64")  # the library's module and pool
    pool = _Pool()
    used = pool.attr(pool.USED)
    g = build_dem(sc, "fp64")
    per_ball = (pool.attr(pool.USED) - used) / n
    assert g.capacity()[:2] == (16, 16)
    assert per_ball < 3600
