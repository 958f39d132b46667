"""Neighbour reuse across uploads on one handle: an upload keeps the lists, and the
first key pass after it has to see every particle that was moved, by whatever
distance (the fixed-point positions repeat every 32 cells)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(name):
    from sph2d_gb300 import cases

    if name == "2d":  # 46,341 particles: fixed-point positions
        return cases.dam_break_2d(seed=1, nx=300, ny=150, dx=0.02, tank=(6.6, 3.4))
    if name == "2d_small":  # cell-relative positions
        return cases.dam_break_2d(seed=1, nx=240, ny=20, dx=0.02, tank=(6.6, 1.0))
    if name == "3d_split":  # four warps per 32 particles
        return cases.dam_break_3d(dx=0.02, tank=(3.6, 0.2, 0.3), block=(1.5, 0.2, 0.2))
    return cases.dam_break_3d(dx=0.0115, tank=(2.2, 0.5, 0.5))  # 3D, a thread per particle


@pytest.mark.parametrize("name", ["2d", "2d_small", "3d_split", "3d"])
@pytest.mark.parametrize("cells", [32.0, 64.0, 32.1, 31.95])
def test_particles_carried_along_an_axis(gpu_available, name, cells):
    """Some fluid particles moved by about a multiple of 32 cells in x, uploaded to a
    handle that has stepped: the step of a fresh handle, bit for bit."""
    from sph2d_gb300 import Solver

    c = _scene(name)
    p = c.params()
    cell = 2.0 * p.hsml
    r = c.r.copy()
    move = np.arange(0, 7)  # of the column at the left wall
    r[move, 0] += cells * cell
    with Solver(p, "mixed") as s:
        s.upload(r, c.v, c.rho, c.itype)
        s.step(1)
        want, pairs = s.download(), s.pair_count()[0]
    with Solver(p, "mixed") as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        s.step(2)
        builds = s.neighbour_rebuilds()
        s.upload(r, c.v, c.rho, c.itype)
        s.step(1)
        assert s.neighbour_rebuilds() == builds + 1
        assert s.pair_count()[0] == pairs
        out = s.download()
    for k in ("r", "v", "rho", "p"):
        assert np.array_equal(out[k], want[k]), k


def test_an_upload_of_the_same_positions_keeps_the_lists(gpu_available):
    from sph2d_gb300 import Solver

    for name in ("2d", "3d_split"):
        c = _scene(name)
        with Solver(c.params(), "mixed") as s:
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(2)
            builds = s.neighbour_rebuilds()
            s.upload(c.r, c.v, c.rho, c.itype)
            s.step(1)
            assert s.neighbour_rebuilds() == builds
