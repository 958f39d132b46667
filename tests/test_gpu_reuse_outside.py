"""The FP32-mixed step with neighbour reuse on fixed-point positions where their
repetition every 32 cells, or the edge of what a key holds, could show: against the
step without reuse (cell-relative positions), with the bars of the mixed step
against the FP64 oracle (test_gpu_parity.py)."""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _run(p, r, v, rho, itype, steps, reuse):
    from sph2d_gb300 import Solver

    pairs, t = [], 0.0
    with Solver(p, "mixed") as s:
        s.set_neighbour_reuse(reuse)
        s.upload(r, v, rho, itype)
        for _ in range(steps):
            t = s.step(1, t)
            pairs.append(s.pair_count()[0])
        return s.download() | s.download_rates(), pairs


def _same(p, c, steps=2):
    a, pa = _run(p, c.r, c.v, c.rho, c.itype, steps, True)
    b, pb = _run(p, c.r, c.v, c.rho, c.itype, steps, False)
    assert pa == pb
    assert np.array_equal(a["itype"], b["itype"])
    for k, bar in (("r", 1e-8), ("v", 1e-4), ("rho", 1e-6), ("p", 1e-3)):
        x, y = a[k], b[k]
        assert np.array_equal(np.isnan(x), np.isnan(y)), k
        assert rel_l2(np.nan_to_num(x), np.nan_to_num(y)) < bar, (k, rel_l2(np.nan_to_num(x), np.nan_to_num(y)))


def _at_the_last_key(crowd, near, extent, max_neighbours):
    """`crowd` fluid particles in a half ball at the far side of the last cell along x
    whose coordinate a 3D key holds (1023), and `near` others in the first cell, on
    the same y and z: the stencil of cell 1023 ends in cell 0."""
    from sph2d_gb300 import cases

    c = cases.dam_break_3d(dx=0.1, tank=(0.5, 0.5, 0.5), block=(0.4, 0.5, 0.3))
    c.model["intf_hsml_coef"] = 1.0
    c.model["max_neighbours"] = max_neighbours
    rng = np.random.default_rng(crowd)
    n = crowd + near
    geom = {"x_mingeom": 0.0, "x_maxgeom": 1023.9, "y_mingeom": 0.0, "y_maxgeom": 4.0, "z_mingeom": 0.0, "z_maxgeom": 4.0}
    c.particle.update(geom, delta=0.5, ntotal=n, nfluid=n, nvirt=0)  # cells of 1
    d = rng.standard_normal((crowd, 3))
    d *= (extent * rng.uniform(0.0, 1.0, (crowd, 1)) ** (1 / 3)) / np.linalg.norm(d, axis=1, keepdims=True)
    d[:, 0] = -np.abs(d[:, 0])
    c.r = np.concatenate([np.array([1023.85, 1.5, 1.5]) + d,
                          np.array([0.05, 1.0, 1.0]) + rng.uniform(0.0, 0.9, (near, 3)) * np.array([0.3, 1.0, 1.0])])
    c.v = rng.standard_normal((n, 3)) * 0.01
    c.rho = np.full(n, 1000.0)
    c.itype = np.full(n, 2, dtype=np.int32)
    return c


# 299 candidates within cutoff and skin: searched. Within 0.49 all of them are neighbours; within 1.18
# at most 256 are, and the whole step runs in the force gather
@pytest.mark.parametrize("crowd,extent,max_neighbours", [(300, 0.49, 1000), (300, 1.18, 257)])
def test_stencil_of_the_last_key(gpu_available, crowd, extent, max_neighbours):
    c = _at_the_last_key(crowd, 40, extent, max_neighbours)
    _same(c.params(), c, steps=1)


@pytest.mark.parametrize("name", ["2d", "3d_split"])
def test_absent_particles_far_outside_ask_for_no_rebuild(gpu_available, name):
    """Non-existent particles parked far below the geometry are nobody's neighbours:
    the lists of the others hold as long as without them."""
    from test_gpu_moved_uploads import _scene

    from sph2d_gb300 import Solver

    builds = []
    for parked in (False, True):
        c = _scene(name)
        c.model["consistency_check"] = False
        c.model["consistency_treatment"] = 0
        p = c.params()
        c.itype[:40] = 0
        if parked:
            c.r[:40, 0] = p.x_mingeom - 100.0 * p.hsml
            c.r[20:40, 1] = p.y_mingeom - 1e6
        with Solver(p, "mixed") as s:
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(6)
            builds.append(s.neighbour_rebuilds())
    assert builds[0] == builds[1] == 1


@pytest.mark.parametrize("dim,treatment", [(2, 0), (2, 1), (3, 0), (3, 1)])
def test_cells_wider_than_the_cubic_kernel(gpu_available, dim, treatment):
    """cell_scale_k above 2 with cubic kernels: pairs beyond 2h are neighbours (and
    counted) whose kernel is zero."""
    from sph2d_gb300 import cases

    if dim == 2:
        c = cases.dam_break_2d(seed=2, nx=300, ny=150, dx=0.02, tank=(6.6, 3.4), density_treatment=treatment)
    else:
        c = cases.dam_break_3d(dx=0.02, tank=(0.5, 0.2, 0.3), block=(0.3, 0.2, 0.2), density_treatment=treatment)
    c.model["max_neighbours"] = 700
    c.v = np.random.default_rng(dim).standard_normal(c.v.shape) * 0.3
    p = c.params()
    p.cell_scale_k = 2.6
    _same(p, c)


@pytest.mark.parametrize("name,reuse", [("2d", True), ("2d_small", True), ("2d_small", False), ("3d_split", True),
                                         ("3d_split", False)])
def test_coincident_particles_count_each_other(gpu_available, name, reuse):
    """Summation density of two particles on one point holds W(0) twice, as in FP64,
    for any number of particles and with and without reuse."""
    from test_gpu_moved_uploads import _scene

    from sph2d_gb300 import Solver

    c = _scene(name)
    c.model["density_treatment"] = 0
    first = np.arange(3, 1203, 12)  # (many: cell-relative separations of some are exactly zero)
    c.r[first] = c.r[first + 1]
    p = c.params()
    rho = []
    for precision in ("fp64", "mixed"):
        with Solver(p, precision) as s:
            if precision == "mixed":
                s.set_neighbour_reuse(reuse)
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(1)
            rho.append(s.download()["rho"])
    assert rel_l2(rho[1], rho[0]) < 1e-6
    both = np.concatenate([first, first + 1])
    assert np.all(np.abs(rho[1][both] / rho[0][both] - 1.0) < 1e-6)


def test_fp64_masks_at_the_last_key(gpu_available):
    """The stored-pair FP64 step's masks at the same place, against the directed gathers."""
    from sph2d_gb300 import Solver

    for crowd in (20, 300):
        c = _at_the_last_key(crowd, 40, 0.49, 1000)
        with Solver(c.params(), "fp64") as s:
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(1)
            rates, pairs = s.download_rates(), s.pair_count()[0]
            s.upload(c.r, c.v, c.rho, c.itype)
            drho = s.density()[0]
            a = s.forces()[0]
            assert pairs == s.neighbours(1000)[2]
        assert rel_l2(rates["drho"], drho) < 1e-11 and rel_l2(rates["a"], a) < 1e-11


def _large(dim):
    """Fixed-point positions and one thread a particle: 2D above 36,000, 3D above 128,000."""
    from sph2d_gb300 import cases

    c = cases.dam_break_2d(seed=2, nx=300, ny=150, dx=0.02, tank=(6.6, 3.4)) if dim == 2 else \
        cases.dam_break_3d(dx=0.0115, tank=(2.2, 0.5, 0.5))
    c.v = np.random.default_rng(dim).standard_normal(c.v.shape) * 0.3
    return c


@pytest.mark.parametrize("dim", [2, 3])
def test_large_sets_with_particles_outside_and_absent(gpu_available, dim):
    """No consistency check: groups below the geometry minimum, within a cell of its
    edge and 16, 32 and 64 cells away, and non-existent particles."""
    c = _large(dim)
    c.model["consistency_check"] = False
    c.model["consistency_treatment"] = 0
    p = c.params()
    cell = 2.0 * p.hsml
    c.itype[60:120:9] = 0
    for first, cells in ((0, 0.4), (10, 16.0), (20, 32.0), (30, 64.0)):
        for j in range(6):
            c.r[first + j] = c.r[first]
            c.r[first + j, 0] = p.x_mingeom - (cells + 0.3 * j) * cell
            c.v[first + j] = 0.0
    _same(p, c)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("cut", [0, 1, 127, 128, 129, 255])
def test_large_sets_around_whole_blocks(gpu_available, dim, cut):
    """The last `cut` + n % 256 particles left out."""
    c = _large(dim)
    n = c.ntotal - c.ntotal % 256 - cut
    c.r, c.v, c.rho, c.itype = c.r[:n].copy(), c.v[:n].copy(), c.rho[:n].copy(), c.itype[:n].copy()
    c.particle.update(ntotal=n, nvirt=n - c.particle["nfluid"])
    _same(c.params(), c, steps=1)


def _coincident(name, what):
    from test_gpu_moved_uploads import _scene

    c = _scene(name)
    m = c.model
    m["density_treatment"] = 0 if what == "gauss_sum" else 1
    m["max_neighbours"] = 900
    if what.startswith("gauss"):
        for k in ("density_skf", "intf_skf", "artificial_viscosity_skf", "average_velocity_skf",
                  "artificial_pressure_skf"):
            m[k] = 2
        m["intf_hsml_coef"] = 1.0
    if what == "xsph":
        m.update(average_velocity=True, average_velocity_coef=0.05, average_velocity_skf=1)
    if what == "delta":
        m.update(density_treatment=2, density_delta_sph_coef=0.1)
    rng = np.random.default_rng(4)
    c.v = rng.standard_normal(c.v.shape) * 0.1 * (c.itype > 0)[:, None]
    c.rho = c.rho * (1.0 + 1e-3 * rng.uniform(-1, 1, len(c.rho)))
    first = np.arange(3, 1203, 12)
    c.r[first] = c.r[first + 1]
    return c, first


@pytest.mark.parametrize("what", ["gauss_sum", "gauss_rate", "xsph"])
@pytest.mark.parametrize("name,reuse", [("2d", True), ("2d_small", True), ("2d_small", False), ("3d_split", True),
                                         ("3d_split", False)])
def test_coincident_particles_in_the_other_sums(gpu_available, name, reuse, what):
    """Gauss kernel (whose exponential of a NaN is one) and XSPH velocity: as in FP64."""
    from sph2d_gb300 import Solver

    c, first = _coincident(name, what)
    p = c.params()
    out = []
    for precision in ("fp64", "mixed"):
        with Solver(p, precision) as s:
            if precision == "mixed":
                s.set_neighbour_reuse(reuse)
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(1)
            out.append(s.download() | s.download_rates())
    for k, bar in (("v", 1e-5), ("a", 1e-5), ("rho", 1e-6)):
        assert np.all(np.isfinite(out[1][k])) and rel_l2(out[1][k], out[0][k]) < bar, k
    both = np.concatenate([first, first + 1])
    assert rel_l2(out[1]["v"][both], out[0]["v"][both]) < 1e-5


@pytest.mark.parametrize("name,reuse", [("2d", True), ("2d_small", True), ("2d_small", False), ("3d_split", True),
                                         ("3d_split", False)])
def test_the_delta_sph_term_of_coincident_particles(gpu_available, name, reuse):
    """Its limit: the rate of particles 1e-6 h apart (the reference's is 0/0)."""
    from sph2d_gb300 import Solver

    c, first = _coincident(name, "delta")
    p = c.params()
    drho = []
    for apart in (0.0, 1e-6 * p.hsml):
        r = c.r.copy()
        r[first, 0] += apart
        with Solver(p, "mixed") as s:
            s.set_neighbour_reuse(reuse)
            s.upload(r, c.v, c.rho, c.itype)
            s.step(1)
            drho.append(s.download_rates()["drho"])
    both = np.concatenate([first, first + 1])
    assert rel_l2(drho[0][both], drho[1][both]) < 1e-4
