"""The forms of the fluid passes and of their list build at the sizes and
states where they change: a single particle, partly filled blocks, either side
of the sixteen-lane limit, no dummies, particles outside the domain, a domain
one cell wide, rows that overflow and are walked, exact lists every step.
The specialised passes against the general ones (FP32: the regrouped terms'
rounding, 1e-5 as the force target; FP64: sums in another order, 1e-12 over
the 1e-15 of an evaluation), the pair sets against all pairs within the cutoff."""
import numpy as np
import pytest

from this_studio_b200 import scenes
from this_studio_b200.solvers import WCSPHSolver

from .helpers import pair_keys, rel_err

pytestmark = pytest.mark.gpu

TOL = {"mixed": 1e-5, "fp64": 1e-12}


def _scene(nx, ny, nz, dummies=True, seed=1, dx=0.01):
    sc = scenes.sph_dam_break(nx, ny, nz, dx, tank=(2 * nx * dx, ny * dx, (nz + 2) * dx), column_height=nz * dx)
    rng = np.random.default_rng(seed)
    sc.fluid = sc.fluid + rng.uniform(-0.1 * dx, 0.1 * dx, sc.fluid.shape)
    sc.velocity = rng.normal(0, 0.2, sc.fluid.shape)
    if not dummies:
        sc.dummy = np.zeros((0, 3))
    return sc


def _build(sc, prec, uniform=True, skin=None, headroom=None, minb=None, maxb=None):
    s = WCSPHSolver()
    if skin is not None:
        s.setSkin(skin)
    if headroom is not None:
        s.setListHeadroom(headroom)
    s.addSPHs(sc.fluid, sc.velocity, sc.sound_speed, sc.spacing, sc.density, sc.viscosity)
    if len(sc.dummy):
        s.addDummies(sc.dummy, None, sc.sound_speed, sc.spacing, sc.density, sc.viscosity)
    s.initialize(minb or sc.minb, maxb or sc.maxb, sc.gravity, sc.dt, prec)
    s.setUniformKernels(uniform)
    return s


def _same(a, b, tol):
    for k in ("velocity", "acceleration", "density", "densityChange"):
        assert rel_err(a[k], b[k]) < tol or np.abs(a[k] - b[k]).max() < 1e-300, k


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [(1, 1, 1), (3, 2, 2), (5, 7, 9), (20, 20, 20), (21, 20, 20)])  # 8,000 and 8,400 last
def test_specialised_passes_against_general(gpu, prec, n):
    sc = _scene(*n)
    a, b = _build(sc, prec), _build(sc, prec, uniform=False)
    for steps in (1, 18):
        a.step(steps)
        b.step(steps)
    _same(a.getSPH(), b.getSPH(), TOL[prec])
    for w in (0, 1):
        np.testing.assert_array_equal(pair_keys(*a.getPairs(w)), pair_keys(*b.getPairs(w)))


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [(9, 8, 7), (24, 22, 20)])
def test_no_dummies_and_exact_lists(gpu, prec, n):
    sc = _scene(*n, dummies=False)
    ref = _build(sc, prec, uniform=False)
    free, exact = _build(sc, prec), _build(sc, prec, skin=0.0)
    for s in (ref, free, exact):
        s.step(12)
    _same(free.getSPH(), ref.getSPH(), TOL[prec])
    _same(exact.getSPH(), ref.getSPH(), TOL[prec])


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [(10, 10, 10), (24, 22, 20)])
def test_overflowed_rows_are_walked(gpu, prec, n):
    """No headroom and a compressed start: rows overflow at the first rebuild
    and the passes walk the cells for them.  After the drift a walked row also
    takes the pairs that came within the cutoff during it (the listed row does
    not): a particle moves at most 1e-4 m = 0.004 x 2 h in a step, where the
    kernel gradient, which falls as the cube of the distance to its edge, is
    below 1e-6 of its usual size; 1e-5 leaves room for several such pairs."""
    sc = _scene(*n)
    a, b = _build(sc, prec, headroom=0.0), _build(sc, prec, uniform=False, headroom=1.0)
    pos = sc.fluid.copy()
    pos[:, 2] *= 0.9
    for s in (a, b):
        s.setSPH(position=pos)
        s.step(4)
    _same(a.getSPH(), b.getSPH(), 1e-5)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("width", [0.02, 0.05, 0.2])  # domains from less than one cell to several cells along x
def test_pair_sets_with_particles_outside_the_domain(gpu, prec, width):
    """A domain narrower than the fluid: the particles beyond its face are
    sorted into the last cells, and every pair within the cutoff is found."""
    sc = _scene(12, 6, 6)
    minb, maxb = tuple(sc.minb), (sc.minb[0] + width, sc.maxb[1], sc.maxb[2])
    g = _build(sc, prec, minb=minb, maxb=maxb)
    g.neighborSearch()
    cut = 2.0 * 1.3 * sc.spacing
    for w, other in ((0, sc.fluid), (1, sc.dummy)):
        d = sc.fluid[:, None] - other[None]
        near = (d * d).sum(-1) <= cut * cut
        if w == 0:
            np.fill_diagonal(near, False)
        a = pair_keys(*g.getPairs(w))
        np.testing.assert_array_equal(np.sort(a), np.sort(pair_keys(*np.nonzero(near))))
    ref = _build(sc, prec, uniform=False, skin=0.0, minb=minb, maxb=maxb)
    for s in (g, ref):
        s.step(5)
    _same(g.getSPH(), ref.getSPH(), TOL[prec])


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [1, 4200])  # couples: sixteen lanes a particle; 8,400 particles: four
@pytest.mark.parametrize("bad", ["velocity", "pressure", "far"])
def test_a_blown_up_particle_reaches_as_far_as_the_kernel(gpu, prec, n, bad):
    """Couples of particles 2% beyond the cutoff of each other, within the skin
    of the lists.  One of each couple has an infinite velocity, a NaN pressure
    or (as the step before such a one leaves it) a velocity that takes it out of
    all numbers: the other falls freely, to the bit."""
    dx = 0.01
    rng = np.random.default_rng(2)
    at = np.stack(np.unravel_index(np.arange(n), (17, 17, 17)), 1) * 0.1 + 0.1
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    pos = np.concatenate([at, at + 1.02 * 2.6 * dx * u])
    s = WCSPHSolver()
    s.addSPHs(pos, None, 10.0, dx, 1000.0, 1e-3)
    s.initialize((0.0,) * 3, (1.9,) * 3, (0.0, 0.0, -9.81), 1e-5, prec)
    vel, p = np.zeros_like(pos), np.zeros(2 * n)
    if bad == "velocity":
        vel[n:] = [np.inf, -np.inf, np.nan]
    elif bad == "pressure":
        p[n:] = np.nan
    else:
        vel[n:] = 1e300
    s.setSPH(velocity=vel, pressure=p)
    s.step(1)
    got = s.getSPH()
    assert len(s.getPairs(0)[0]) == 0
    free = WCSPHSolver()
    free.addSPHs(pos[:n], None, 10.0, dx, 1000.0, 1e-3)
    free.initialize((0.0,) * 3, (1.9,) * 3, (0.0, 0.0, -9.81), 1e-5, prec)
    free.step(1)
    want = free.getSPH()
    for k in ("position", "velocity", "acceleration", "density"):
        np.testing.assert_array_equal(got[k][:n], want[k])


def _squeezed(n, seed=5):
    """A tank whose lower half is pressed together to 0.55 of its height: up to
    forty particles to a cell below, rows of 60 to 160 entries."""
    sc = _scene(*n, seed=seed)
    z = sc.fluid[:, 2]
    mid = 0.5 * (z.min() + z.max())
    sc.fluid[:, 2] = np.where(z < mid, mid - 0.55 * (mid - z), z)
    sc.velocity *= 0.5
    return sc


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
@pytest.mark.parametrize("n", [(28, 27, 25), (35, 34, 33)])  # 18,900 and 39,270
def test_list_build_of_large_fluids(gpu, prec, n):
    """A fluid large enough for the list build with a particle per lane, whose
    cells hold more than a warp's 32 particles and more than a stage's 128
    candidates: after every step the pairs are those of exact lists built from
    the step's start, and the state stays with it (sums in another order)."""
    sc = _squeezed(n)
    a, b = _build(sc, prec, headroom=0.2), _build(sc, prec, skin=0.0, headroom=0.2)
    a.setGraphs(False)  # (a replayed step leaves no lists to read after a change of state)
    b.setGraphs(False)
    assert a.skinStats()[0] > 0 and b.skinStats()[0] == 0
    cell = np.floor((sc.fluid - np.array(sc.minb)) / (2.6 * sc.spacing * 1.04)).astype(int)
    assert np.unique(cell, axis=0, return_counts=True)[1].max() > 32
    for _ in range(6):
        a.step(1)
        b.step(1)
        for w in (0, 1):
            p, q = pair_keys(*a.getPairs(w)), pair_keys(*b.getPairs(w))
            np.testing.assert_array_equal(np.sort(p), np.sort(q))
        rows = np.bincount(a.getPairs(0)[0])
        assert rows.max() > 128 and len(np.unique(rows % 8)) == 8
        _same(a.getSPH(), b.getSPH(), TOL[prec])
        x = b.getSPH()  # both go on from one state, so that no pair at the cutoff differs
        a.setSPH(x["position"], x["velocity"], x["density"], x["pressure"], x["densityChange"])
        b.setSPH(x["position"], x["velocity"], x["density"], x["pressure"], x["densityChange"])


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_rows_of_a_large_fluid_overflow_and_are_walked(gpu, prec):
    """As test_overflowed_rows_are_walked, at the size of the build with a
    particle per lane."""
    sc = _scene(35, 34, 33)
    a, b = _build(sc, prec, headroom=0.0), _build(sc, prec, uniform=False, headroom=1.0)
    pos = sc.fluid.copy()
    pos[:, 2] *= 0.9
    for s in (a, b):
        s.setSPH(position=pos)
        s.step(4)
    _same(a.getSPH(), b.getSPH(), 1e-5)


@pytest.mark.parametrize("n,empty", [((24, 24, 26), 1.0), ((25, 24, 25), 1.0), ((25, 24, 25), 2.0), ((25, 24, 25), 3.0)])
def test_pair_sets_with_plain_and_with_split_cells(gpu, n, empty):
    """The sort's cells are split along x for fluids of at least 15,000 particles
    (14,976 and 15,000 here) in domains of no more cells than particles (about
    2,600, 10,000 and 22,000 here): every pair within the cutoff either way."""
    sc = _scene(*n)
    wide = tuple(a + empty * (b - a) if k < 2 else b for k, (a, b) in enumerate(zip(sc.minb, sc.maxb)))
    g = _build(sc, "mixed", maxb=wide)
    g.setGraphs(False)
    g.step(1)
    x, cut = sc.fluid, 2.0 * 1.3 * sc.spacing
    key = pair_keys(*g.getPairs(0))
    from scipy.spatial import cKDTree
    p = cKDTree(x).query_pairs(cut, output_type="ndarray")
    d = x[p[:, 0]] - x[p[:, 1]]
    p = p[(d * d).sum(1) <= cut * cut]
    both = np.concatenate([p, p[:, ::-1]])
    np.testing.assert_array_equal(np.sort(key), np.sort(pair_keys(both[:, 0], both[:, 1])))


def test_which_scenes_run_the_fp64_passes(gpu):
    """Uniform constants, lengths and densities inside the range of the FP32
    approximations their reciprocals start from, and no coupled bodies."""
    for n in ((4, 4, 4), (21, 20, 20)):
        assert _build(_scene(*n), "fp64").uniformKernelsFP64() and _build(_scene(*n), "mixed").uniformKernels()
        assert not _build(_scene(*n), "mixed").uniformKernelsFP64()
        assert not _build(_scene(*n), "fp64", uniform=False).uniformKernelsFP64()
    light = _scene(4, 4, 4)
    light.density = 1e-10
    assert not _build(light, "fp64").uniformKernelsFP64()
    sc = scenes.balls_in_tank(nx=10, ny=10, depth=10, balls=((0.5, 0.5, 0.5, 2.0, 1200.0),))
    f, d, c = scenes.build_coupled(sc, "fp64")
    c.step(1, sc.dem_substeps)
    assert not f.uniformKernelsFP64()
