"""rrsph_autotune never leaves a solver slower than it found it: the sizes in use (the
kernels' own, which no candidate names, unless set) are timed too."""

import pytest

pytestmark = pytest.mark.gpu


def test_trials_of_both_kinds_run(gpu_available):
    """Nine candidates, and the sizes in use before and after them."""
    from sph2d_gb300 import Solver, cases

    c = cases.dam_break_2d(nx=60, ny=30)
    with Solver(c.params(), "fp64") as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        s.step(3)
        n0 = s.kernel_launches()
        s.step(10)
        step = (s.kernel_launches() - n0) / 10.0
        n0 = s.kernel_launches()
        s.autotune(steps=9)
        trials = (s.kernel_launches() - n0) / (10.0 * step)
        assert 10.5 <= trials < 12.0  # (a single step reports its end too)
