"""The FP32-mixed step with neighbour reuse (fixed-point positions, split
gathers) where its bookkeeping can go wrong, against the step without reuse,
which searches the stencil with cell-relative floats: pair counts equal, and
states within the bars of the mixed step against the FP64 oracle
(test_gpu_parity.py)."""

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
        return s.download(), pairs


def _same(p, c, steps=4):
    a, pa = _run(p, c.r, c.v, c.rho, c.itype, steps, True)
    b, pb = _run(p, c.r, c.v, c.rho, c.itype, steps, False)
    assert pa == pb
    assert np.array_equal(a["itype"], b["itype"])
    for k, bar in (("r", 1e-8), ("v", 1e-4), ("rho", 1e-6), ("p", 1e-3)):
        x, y = a[k], b[k]
        assert np.array_equal(np.isnan(x), np.isnan(y)), k
        assert rel_l2(np.nan_to_num(x), np.nan_to_num(y)) < bar, (k, rel_l2(np.nan_to_num(x), np.nan_to_num(y)))


def _scene(dim, treatment, nx, ny):
    from sph2d_gb300 import cases

    if dim == 2:
        c = cases.dam_break_2d(seed=nx, nx=nx, ny=ny, dx=0.02, tank=(0.02 * nx + 0.6, 0.02 * ny + 0.4),
                               density_treatment=min(treatment, 1))
    else:
        c = cases.dam_break_3d(seed=nx, dx=0.02, tank=(0.5, 0.2, 0.3), block=(0.02 * nx, 0.2, 0.02 * ny),
                               density_treatment=min(treatment, 1))
    if treatment == 2:
        c.model["density_treatment"] = 2
        c.model["density_delta_sph_coef"] = 0.1
    c.model["artificial_bulk_visc"] = 0.1
    rng = np.random.default_rng(5 * nx + ny)
    c.v = rng.standard_normal(c.v.shape) * 0.3
    return c


@pytest.mark.parametrize("treatment", [0, 1, 2])
@pytest.mark.parametrize("dim,nx,ny", [(2, 1, 1), (2, 17, 9), (2, 300, 150), (3, 8, 6)])
def test_reuse_against_search(gpu_available, dim, nx, ny, treatment):
    """Both sides of the split (36,000 particles in 2D), wall and bulk viscosity terms."""
    c = _scene(dim, treatment, nx, ny)
    _same(c.params(), c)


@pytest.mark.parametrize("count", [1, 31, 32, 33, 127, 128, 129])
def test_particle_counts_around_whole_blocks(gpu_available, count):
    c = _scene(2, 0, 12, 11)
    c.r, c.v, c.rho, c.itype = c.r[:count].copy(), c.v[:count].copy(), c.rho[:count].copy(), c.itype[:count].copy()
    c.particle.update(ntotal=count, nfluid=count, nvirt=0)
    _same(c.params(), c)


@pytest.mark.parametrize("dim", [2, 3])
def test_particles_outside_the_grid_and_absent_ones(gpu_available, dim):
    """No consistency check: groups of particles below the geometry minimum (cell
    coordinate 0), within a cell of the edge, and 16, 32 and 64 cells away, where
    fixed point modulo 32 cells repeats; and non-existent particles."""
    c = _scene(dim, 0, 10, 8)
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
    _same(p, c, steps=2)


@pytest.mark.parametrize("dim,nx,ny", [(2, 12, 9), (2, 300, 150), (3, 8, 6)])
@pytest.mark.parametrize("factor", [0.5, 0.6])
def test_crowded_cells(gpu_available, dim, nx, ny, factor):
    """Every other particle of a patch drawn together: cells with several batches of
    candidates, lists full to the last group and (0.5 in 2D) particles with more
    candidates than a list holds, but no more neighbours than the model allows."""
    c = _scene(dim, 1, nx, ny)
    c.v[:] = 0.0
    k = min(100 if dim == 2 else 300, c.particle["nfluid"])
    centre = c.r[:k].mean(axis=0)
    patch = np.argsort(np.abs(c.r - centre).max(axis=1), kind="stable")[:k][::2]
    c.r[patch] = centre + (c.r[patch] - centre) * factor
    _same(c.params(), c, steps=2)
