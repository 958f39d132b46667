"""The FP64 loop's pair sums that evaluate each pair once (kernels_pairs64.cu),
where their bookkeeping can go wrong: particle counts around whole warps,
more neighbours than a particle stores, cells with more particles than a mask
has bits, coincident and non-existent particles, particles outside the grid.

The first step from an upload (no predictor yet) is compared with the
general directed gathers behind rrsph_density / rrsph_forces and with the C
oracle. Bars: each term is good to a few units in the last place (1e-15) and
the terms of an acceleration, rate or pressure exceed their sum by up to 1e3
in these scenes, so 1e-11 (1e-13 for the density, a sum of positive terms).
"""

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _scene(dim, treatment, coef, nx, ny):
    from sph2d_gb300 import cases

    if dim == 2:
        c = cases.dam_break_2d(seed=nx, nx=nx, ny=ny, dx=0.02, tank=(1.0, 0.6), density_treatment=min(treatment, 1))
    else:
        c = cases.dam_break_3d(seed=nx, dx=0.02, tank=(0.5, 0.2, 0.3), block=(0.02 * nx, 0.2, 0.02 * ny),
                               density_treatment=min(treatment, 1))
    c.model["intf_hsml_coef"] = coef
    c.model["max_neighbours"] = 700
    c.model["artificial_bulk_visc"] = 0.1
    if treatment == 2:
        c.model["density_treatment"] = 2
        c.model["density_delta_sph_coef"] = 0.1
    rng = np.random.default_rng(17 * nx + ny)
    c.v = rng.standard_normal(c.v.shape) * 0.3
    return c


def _step(p, c):
    from sph2d_gb300 import Solver

    with Solver(p, "fp64") as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        s.step(1, 0.0)
        out = s.download() | s.download_rates()
        out["pairs"] = s.pair_count()[0]
    return out


def _pieces(p, c):
    """The same evaluation through the loop pieces (the directed gathers)."""
    from sph2d_gb300 import Solver

    with Solver(p, "fp64") as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        d, pres = s.density()
        a, _, _ = s.forces()
        counts, _, tot = s.neighbours(700)
    return d, pres, a, tot


def _err(x, want):
    """Relative L2 over the numbers; NaN where, and only where, it is wanted."""
    assert np.array_equal(np.isnan(x), np.isnan(want))
    return rel_l2(np.nan_to_num(x), np.nan_to_num(want))


def _check(p, c, treatment):
    st = _step(p, c)
    d, pres, a, pairs = _pieces(p, c)
    assert st["pairs"] == pairs
    assert _err(st["rho" if treatment == 0 else "drho"], d) < (1e-13 if treatment == 0 else 1e-11)
    assert _err(st["p"], pres) < 1e-11
    assert _err(st["a"], a) < 1e-11
    return st


# 2D: h 1.4 dx (the usual 20 neighbours), 2 dx (50: more than the 48 stored), 3 dx
# (110, cells of 36 particles: more than 32 bits); 3D: 1.3 dx (70), 1.8 dx (190: more
# than the 160 stored, wall cells above 64 particles)
@pytest.mark.parametrize("treatment", [0, 1, 2])
@pytest.mark.parametrize("dim,coef,nx,ny", [(2, 1.4, 1, 1), (2, 1.4, 17, 9), (2, 1.4, 24, 13), (2, 2.0, 23, 14),
                                             (2, 3.0, 25, 15), (3, 1.3, 8, 6), (3, 1.8, 9, 7)])
def test_step_against_the_directed_gathers_and_the_oracle(gpu_available, dim, coef, nx, ny, treatment):
    from oracle import binding as O

    c = _scene(dim, treatment, coef, nx, ny)
    p = c.params()
    st = _check(p, c, treatment)
    ref = O.run(p, c.r, c.v, c.rho, c.itype, nsteps=1)
    for k in ("r", "v", "rho", "p"):
        assert rel_l2(st[k], ref[k]) < 1e-11, k
    assert np.array_equal(st["itype"], ref["itype"])


@pytest.mark.parametrize("treatment", [0, 2])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 63, 64, 65, 97])
def test_particle_counts_around_whole_warps(gpu_available, count, treatment):
    """The first `count` fluid particles alone (no wall)."""
    c = _scene(2, treatment, 1.4, 12, 9)
    c.r, c.v, c.rho, c.itype = c.r[:count].copy(), c.v[:count].copy(), c.rho[:count].copy(), c.itype[:count].copy()
    c.particle.update(ntotal=count, nfluid=count, nvirt=0)
    _check(c.params(), c, treatment)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("treatment", [0, 2])
def test_coincident_absent_and_outside_particles(gpu_available, dim, treatment):
    """Two fluid particles on one point (0/0 in the reference's delta-SPH term), every ninth fluid particle
    non-existent, and (no consistency check) a group of particles below the
    geometry minimum, whose cell coordinate is 0: some cells away, where the
    float offsets are still good, and 1e4 cells away, where they are not."""
    c = _scene(dim, treatment, 1.4 if dim == 2 else 1.3, 10, 8)
    c.model["consistency_check"] = False
    c.model["consistency_treatment"] = 0
    c.r[3] = c.r[4]
    c.itype[9:60:9] = 0
    p = c.params()
    cell = 2.0 * p.hsml
    for first, cells in ((20, 3.0), (30, 1e4)):
        for j in range(6):
            c.r[first + j] = c.r[20]
            c.r[first + j, 0] = p.x_mingeom - (cells + 0.21 * j) * cell
    _check(p, c, treatment)


@pytest.mark.parametrize("dim,treatment", [(2, 0), (2, 1), (3, 1)])
def test_block_sizes_give_the_same_bits(gpu_available, dim, treatment):
    from sph2d_gb300 import Solver

    c = _scene(dim, treatment, 1.3, 23, 11)
    out = []
    for threads in (None, 64, 128, 256):
        with Solver(c.params(), "fp64") as s:
            if threads:
                s.set_gather_threads(threads, threads)
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(3)
            out.append(s.download())
    for o in out[1:]:
        for k in ("r", "v", "rho", "p"):
            assert np.array_equal(o[k], out[0][k]), k
