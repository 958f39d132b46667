"""The stored pairs of the FP64 step are memory a handle can do without: it takes
them only where little of the free memory goes, and gives them back to a call that
needs it. The rest of the card is filled here, down to a few GB."""

import contextlib

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

GB = 1 << 30


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _room(leave):
    """The card with `leave` bytes free."""
    import torch

    torch.cuda.empty_cache()
    filler = torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def _case():
    from sph2d_gb300 import cases

    return cases.piston_flume_2d(nx=4000, ny=100)  # 409k: 0.7 GB of stored pairs


def _steps(s, c):
    s.upload(c.r, c.v, c.rho, c.itype)
    s.step(3)
    return s.download() | {"pairs": s.pair_count()}


def _same(got, want):
    """Both routes are good to a few 1e-15 a term; three steps."""
    for k in ("r", "v", "rho", "p"):
        assert rel_l2(got[k], want[k]) < 1e-11, k
    assert got["pairs"] == want["pairs"]


def test_a_card_with_little_room_keeps_the_directed_gathers(gpu_available):
    from sph2d_gb300 import Solver

    c = _case()
    p = c.params()
    with Solver(p, "fp64") as s:
        want = _steps(s, c)
    with _room(5 * GB // 2):
        before = _free()
        with Solver(p, "fp64") as s:
            assert before - _free() < GB // 2
            got = _steps(s, c)
    _same(got, want)


def test_a_call_that_needs_the_memory_gets_it(gpu_available):
    """A neighbour list longer than what is free, by less than the stored pairs take;
    the steps before and after it, the latter on the directed gathers."""
    from sph2d_gb300 import Solver

    c = _case()
    p = c.params()
    with Solver(p, "fp64") as s:
        want = _steps(s, c)
        s.upload(c.r, c.v, c.rho, c.itype)
        pairs = s.neighbours(64)[2]
    with _room(10 * GB // 3):
        before = _free()
        with Solver(p, "fp64") as s:
            assert before - _free() > GB // 2
            _same(_steps(s, c), want)
            s.upload(c.r, c.v, c.rho, c.itype)
            longest = -(-(_free() + GB // 4) // (4 * s.n))
            assert s.neighbours(longest)[2] == pairs
            got = _steps(s, c)
    _same(got, want)
