"""One call on the caller's arrays (rrsph_step_host) on either side of the number
of particles above which p and rho come back during the force gather, against
the separate calls: the same bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [214, 216])  # 99,468 and 100,397 particles with the walls
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("treatment", [0, 1])
def test_step_host_around_the_early_copies(gpu_available, ny, precision, treatment):
    from sph2d_gb300 import Solver, cases

    c = cases.dam_break_2d(seed=3, nx=440, ny=ny, dx=0.5 / ny, density_treatment=treatment)
    p = c.params()
    with Solver(p, precision) as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        t = s.step(2)
        want = s.download()
    with Solver(p, precision) as s:
        h = {"r": c.r.copy(), "v": c.v.copy(), "rho": c.rho.copy(), "itype": c.itype.copy(), "p": np.zeros(c.rho.shape)}
        assert s.step_host(h, 2, 0.0) == t
    for k in ("r", "v", "rho", "p", "itype"):
        assert np.array_equal(h[k], want[k]), k
