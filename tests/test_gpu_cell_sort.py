"""The grid's counting sort (sort.cu, cell_sort) and the radix sort that larger
tables keep, against the oracle's make_grid: keys, sorted ids and cell starts
bit for bit, around whole blocks of particles and tiles of cells, with empty
tables, crowded cells, and repeated on one handle (the counts have to be clear
again)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(n, dim, extent):
    """n fluid particles in a box of `extent` cells a side (h = 0.5: cells of 1)."""
    from sph2d_gb300 import cases

    c = cases.dam_break_2d(nx=2, ny=2) if dim == 2 else cases.dam_break_3d(dx=0.1, tank=(0.5, 0.5, 0.5), block=(0.4, 0.5, 0.3))
    c.model["intf_hsml_coef"] = 1.0
    geom = {f"{a}_{m}geom": (0.0 if m == "min" else float(extent)) for a in "xyz"[:dim] for m in ("min", "max")}
    c.particle.update(geom, delta=0.5, ntotal=n, nfluid=n, nvirt=0)
    c.r = np.zeros((n, dim))
    return c


# (dim, cells a side): 2-cell table, tables around a few tiles of 1024 cells, many tiles;
# 30,000 cells a side (2^30 keys): the radix sort
@pytest.mark.parametrize("dim,extent", [(2, 1), (2, 40), (2, 50), (2, 700), (2, 30000), (3, 12), (3, 100)])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
def test_grid_against_the_oracle(gpu_available, dim, extent, n):
    from oracle import binding as O
    from sph2d_gb300 import Solver

    c = _params(n, dim, extent)
    rng = np.random.default_rng(n + extent)
    spread = rng.uniform(0.0, extent, size=(n, dim))
    crowd = spread.copy()
    crowd[: n // 2] = rng.uniform(0.0, 1.0, size=(n // 2, dim)) * min(1.0, extent) * 0.999  # half of them in one cell
    c.r = spread
    p = c.params()
    v, rho, itype = np.zeros((n, dim)), np.full(n, 1000.0), np.full(n, 2, dtype=np.int32)
    big = int(p.max_cells) > 1 << 24
    with Solver(p, "fp64") as s:
        for r in (spread, crowd, spread):
            s.upload(r, v, rho, itype)
            keys, grid, cs = s.grid_find(with_cells_start=not big)
            if big:
                order = np.lexsort((np.arange(n), keys))
                assert np.array_equal(grid, order.astype(np.uint32))
            else:
                k_o, g_o, cs_o = O.grid(p, r)
                assert np.array_equal(keys, k_o) and np.array_equal(grid, g_o) and np.array_equal(cs, cs_o)
