"""The forms of the grid-ordered kernels (nspt_set_local_gf_form) give the same
links, bit for bit: they have the same lanes per link and form every sum alike.
Needs a B200."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(P, O, L, N, grid, run, **kw):
    o = O.Oracle(L, N, twist_mask=sum({"y": 2, "z": 4, "t": 8}[d] for d in kw.get("twist", "")))
    o.random_start(7, 0.5)
    noise = O.Rand55(5).gauss(o.V * 32)
    out = []
    for form in ("group", "team", "auto"):
        with P.NsptEngine(L, N, **kw) as e:
            e.set_gf_grid(grid)
            e.set_local_gf_form(form)
            e.upload(o.links)
            e.set_noise(noise)
            run(e)
            out.append(e.download())
    return out


@pytest.mark.parametrize("N,kw", [(1, {}), (8, dict(twist="yz")), (9, {}), (14, dict(twist="t")),
                                  (15, {}), (16, dict(zero_modes=True)), (24, dict(twist="yz"))],
                         ids=["n1", "n8_yz", "n9", "n14_t", "n15", "n16_ordered", "n24_yz"])
@pytest.mark.parametrize("L,grid", [((4, 6, 4, 4), (2, 3, 2, 2)), ((4, 2, 4, 3), (2, 1, 2, 1))],
                         ids=["one_site", "three_sites"])
def test_local_gauge_fixing(engine_mod, oracle_mod, L, grid, N, kw):
    g, t, a = fields(engine_mod, oracle_mod, L, N, grid,
                     lambda e: e.stochastic_gauge_fixing(-0.05), **kw)
    assert np.array_equal(g, t) and np.array_equal(g, a)


@pytest.mark.parametrize("N,kw", [(5, {}), (8, dict(zero_modes=True)), (12, dict(twist="yz")),
                                  (16, {})], ids=["n5", "n8_logs", "n12_yz", "n16"])
def test_on_the_fly_sweep(engine_mod, oracle_mod, N, kw):
    g, t, a = fields(engine_mod, oracle_mod, (4, 6, 4, 4), N, (2, 3, 2, 2),
                     lambda e: e.gauge_wilson(0.01), update="onthefly", **kw)
    assert np.array_equal(g, t) and np.array_equal(g, a)
