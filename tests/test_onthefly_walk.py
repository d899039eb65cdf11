"""The on-the-fly sweep where one reference thread walks many sites (grids with
few threads, odd extents): one launch per barrier step however long the walk.
Needs a B200.  Tolerance as tests/test_onthefly.py."""
import time

import numpy as np
import pytest

from helpers import per_order_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,grid", [((4, 4, 4, 4), (1, 1, 1, 1)), ((5, 4, 4, 4), (1, 1, 1, 1)),
                                    ((4, 4, 3, 7), (2, 2, 1, 1))],
                         ids=["256_sites", "320_sites", "84_sites"])
def test_long_walks(engine_mod, oracle_mod, L, grid):
    """Both sides of the number of sites up to which a walk goes in parts."""
    P, O, N = engine_mod, oracle_mod, 5
    o = O.Oracle(L, N)
    o.random_start(21, 0.5)
    noise = O.Rand55(7).gauss(o.V * 32)
    with P.NsptEngine(L, N, update="onthefly") as e:
        e.set_gf_grid(grid)
        e.upload(o.links)
        e.set_noise(noise)
        e.gauge_wilson(0.01)
        got = e.download()
    o.sweep(0.01, noise, onthefly=True, grid=grid)
    assert per_order_rel(got, o.links, N).max() <= 1e-12


def test_the_time_limit_holds_on_a_long_walk(engine_mod):
    """A step of some 0.3 s with a limit a twentieth of it: the call comes back
    with NSPT_ERR_TIMEOUT in less than half the step (the host launches no more
    than the stream's queue takes), and the field is that of a run without one."""
    from prlgt2020_b200 import _lib
    P = engine_mod
    L, N = (7, 7, 7, 7), 8
    with P.NsptEngine(L, N, update="onthefly") as a, P.NsptEngine(L, N, update="onthefly") as b:
        for e in (a, b):
            e.seed(77, 0)
            e.NsptEvolve(0.01, 1, 0)  # loads the kernels
        t = time.perf_counter()
        b.NsptEvolve(0.01, 1, 0)
        full = time.perf_counter() - t
        a.set_timeout(full / 20)
        t = time.perf_counter()
        with pytest.raises(P.NsptError) as err:
            a.NsptEvolve(0.01, 1, 0)
        waited = time.perf_counter() - t
        assert err.value.code == _lib.NSPT_ERR_TIMEOUT
        a.set_timeout(0.0)
        a.NsptEvolve(0.01, 1, 0)
        b.NsptEvolve(0.01, 1, 0)
        assert np.array_equal(a.download(), b.download())
    assert waited < full / 2, (waited, full)
