"""What an upload makes of the links' flags (GPU): across a twisted face a flag
other than 1 takes the sweep link by link, wherever in the field it is, in either
layout of the host field, and until another field comes.  Tolerance as
tests/test_series_forms.py."""
import numpy as np
import pytest

from helpers import flag_diff, per_order_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 2], ids=["same_orders", "more_orders"])
@pytest.mark.parametrize("link", [0, 700, -1])
def test_one_flag(engine_mod, oracle_mod, extra, link):
    P, O, L, N = engine_mod, oracle_mod, (4, 6, 3, 4), 4
    o = O.Oracle(L, N, twist_mask=6)
    o.random_start(8, 0.5)
    unit = o.links.copy()
    o.links.reshape(-1, o.links.shape[-1])[link, :2] = (0.5, -0.25)
    noise = O.Rand55(3).gauss(o.V * 32)

    def host(links):
        a = np.zeros(links.shape[:2] + (P.series_len(N + extra),))
        a[:, :, :links.shape[2]] = links
        return a

    with P.NsptEngine(L, N, twist="yz") as e, P.NsptEngine(L, N, twist="yz") as f:
        for start in (o.links.copy(), unit):
            e.upload(host(start), allocORD=N + extra)
            e.set_noise(noise)
            e.gauge_wilson(0.01)
            o.set_links(start)
            o.sweep(0.01, noise)
            assert per_order_rel(e.download(), o.links, N).max() <= 1e-12
            assert flag_diff(e.download(), o.links, N) <= 1e-15
        f.upload(unit)
        f.set_noise(noise)
        f.gauge_wilson(0.01)
        assert np.array_equal(e.download(), f.download())
