"""The adjoint where particles have more neighbours than stored-pair slots (48),
so that some pairs are evaluated in place by both sides, and by the directed
gathers (pressure form 1), against the oracle's forward-mode reference with the
bar of test_gpu_adjoint.py (a change of the start by 1e-15 moves these gradients
by less than 3e-12)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coef,steps", [(2.2, 120), (3.0, 50)])  # up to 60 and 112 neighbours
@pytest.mark.parametrize("form", [1, 2])
def test_gradient_with_pairs_past_the_slots(gpu_available, coef, steps, form):
    from oracle import binding as O

    from sph2d_gb300 import Solver, cases

    gauge_x = 0.15
    c = cases.adjoint_flume_2d(nx=60, ny=15, dx=0.01, steps=steps, gauge_x=gauge_x, window=0.005, sample_every=5)
    c.model["intf_hsml_coef"] = coef
    c.model["max_neighbours"] = 200
    c.model["intf_sph_approximation"] = form
    p = c.params()
    sample = {"sample_from": c.notes["sample_from"], "sample_every": c.notes["sample_every"]}
    _, dg, _ = O.piston_tangent_run(p, c.r, c.v, c.rho, c.itype, steps, c.notes["omega"], c.notes["coef"], gauge_x,
                                    **sample)
    with Solver(p, "fp64") as s:
        s.upload(c.r, c.v, c.rho, c.itype)
        s.set_piston_fourier(c.notes["omega"], c.notes["coef"])
        g = s.adjoint_forward(steps, gauge_x, checkpoint_every=40, **sample)[0]
        w = np.linspace(1.0, 2.0, len(g))
        dcoef, _ = s.adjoint_reverse(w)
    want = dg.T @ w
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(dcoef - want) < 1e-8 * np.linalg.norm(want)
