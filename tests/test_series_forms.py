"""The series kernels where their forms and blocks change, against the oracle
(GPU, through the C ABI).

A launch takes one of three forms of the Cauchy product: 9 lanes per link
(launches of at least 24 links per SM, up to 14 orders), a warp per link, and
the ordered sums (zero modes or Fourier-accelerated gauge fixing above 14
orders).  A product works on blocks of 8 orders, the lowest of which may stick
out below order 1; the exponential serves two orders per lane.  The Wilson
sweep goes plaquette by plaquette, in slabs of direction 0 on large lattices,
and link by link where a flag other than 1 meets a twisted face.

Tolerance: that of tests/test_gpu_parity.py, 1e-12 per order after one sweep
(a few hundred roundings of 1e-16 in sums of terms of the coefficients' size).
"""
import numpy as np
import pytest

from helpers import flag_diff, obs_close, per_order_rel

pytestmark = pytest.mark.gpu

TWIST = {"y": 2, "z": 4, "t": 8}


def one_sweep(P, O, L, N, twist="", start=3, links=None, **kw):
    o = O.Oracle(L, N, twist_mask=sum(TWIST[d] for d in twist))
    o.random_start(start, 0.5)
    if links is not None:
        links(o.links)
    e = P.NsptEngine(L, N, twist=twist, **kw)
    e.upload(o.links)
    nz = O.Rand55(11).gauss(o.V * 32)
    e.set_noise(nz)
    eo = e.gauge_wilson(0.01)
    oo = o.sweep(0.01, nz, zero_modes=bool(kw.get("zero_modes")))
    for a, b in ((eo.plaq, oo.plaq), (eo.norm, oo.norm), (eo.tru, oo.tru)):
        ok, worst = obs_close(a, b, 1e-12)
        assert ok, worst
    return e, o


@pytest.mark.parametrize("L", [(2, 2, 2, 2), (6, 6, 5, 6)], ids=["warp_per_link", "nine_lanes"])
@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 14])
def test_block_edges(engine_mod, oracle_mod, L, N):
    """One sweep at the edges of the product's blocks, in the form for few
    links (64) and for many (4320)."""
    e, o = one_sweep(engine_mod, oracle_mod, L, N)
    assert per_order_rel(e.download(), o.links, N).max() <= 1e-12
    assert flag_diff(e.download(), o.links, N) == 0.0


@pytest.mark.parametrize("N", [15, 17, 18, 31, 33])
def test_high_order_edges(engine_mod, oracle_mod, N):
    """One sweep at orders above the 9-lane form: past two blocks, and where
    the exponential's second order per lane begins."""
    e, o = one_sweep(engine_mod, oracle_mod, (2, 2, 2, 4), N)
    assert per_order_rel(e.download(), o.links, N).max() <= 1e-12


@pytest.mark.parametrize("L,N,twist", [((9, 10, 10, 12), 2, ""), ((9, 10, 10, 12), 2, "yzt"),
                                       ((3, 4, 3, 5), 5, "yz")],
                         ids=["slabs_4_4_1", "slabs_twisted", "whole_odd_twisted"])
def test_plaquette_slabs(engine_mod, oracle_mod, L, N, twist):
    """The sweep in slabs (the first needs the last plane's plaquettes, the
    last slab is shorter) and on a whole odd lattice."""
    e, o = one_sweep(engine_mod, oracle_mod, L, N, twist=twist)
    assert per_order_rel(e.download(), o.links, N).max() <= 1e-12
    ok, worst = obs_close(e.plaquette_measure(), o.plaquette(), 1e-12)
    assert ok, worst


@pytest.mark.parametrize("twist", ["", "yz"])
def test_flags_other_than_one(engine_mod, oracle_mod, twist):
    """Flags that are not 1: general flag terms of every product and, across a
    twisted face, the link-by-link sweep and the four views of a plaquette."""
    def flags(links):
        rng = np.random.default_rng(5)
        links[:, :, :2] = rng.normal(size=links[:, :, :2].shape)

    e, o = one_sweep(engine_mod, oracle_mod, (4, 2, 3, 4), 5, twist=twist, links=flags)
    assert per_order_rel(e.download(), o.links, 5).max() <= 1e-12
    ok, worst = obs_close(e.plaquette_measure(), o.plaquette(), 1e-12)
    assert ok, worst


@pytest.mark.parametrize("N", [14, 15, 20])
def test_logarithms_across_the_ordered_form(engine_mod, oracle_mod, N):
    """A sweep with zero modes on the two sides of the order where the sums
    are kept in order.  The logarithm amplifies rounding by about 4 per order:
    max(1e-12, 1e-16 * 4^k) per order."""
    e, o = one_sweep(engine_mod, oracle_mod, (4, 4, 2, 4), N, zero_modes=True)
    e.zero_modes_subtraction()
    o.zero_modes()
    rel = per_order_rel(e.download(), o.links, N)
    assert np.all(rel <= np.maximum(1e-12, 1e-16 * 4.0 ** np.arange(1, N + 1))), rel


@pytest.mark.parametrize("zero_modes,N", [(False, 1), (False, 9), (False, 19), (True, 15)],
                         ids=["n1", "n9", "n19", "ordered"])
def test_local_gf_teams(engine_mod, oracle_mod, zero_modes, N):
    """Local gauge fixing by a team and by a group per reference thread, three
    sites to a thread (odd t), across a twisted face (zero modes: periodic)."""
    L, twist = (4, 2, 4, 3), "" if zero_modes else "z"
    for form in ("team", "group"):
        o = oracle_mod.Oracle(L, N, twist_mask=TWIST.get(twist, 0))
        o.random_start(7, 0.5)
        e = engine_mod.NsptEngine(L, N, twist=twist, zero_modes=zero_modes)
        e.set_gf_grid((2, 1, 2, 1))
        e.set_local_gf_form(form)
        e.upload(o.links)
        e.stochastic_gauge_fixing(-0.05)
        o.local_gauge_fix(-0.05, grid=(2, 1, 2, 1))
        assert per_order_rel(e.download(), o.links, N).max() <= 1e-12, form


@pytest.mark.parametrize("N", [3, 9, 15], ids=["one_launch", "parts_nine_lanes", "parts_warp"])
def test_onthefly_many_threads(engine_mod, oracle_mod, N):
    """The on-the-fly sweep with 4096 reference threads: a 4^4 field and noise,
    repeated over 16^4, stay repeated (blocks of 2 sites a side divide both)."""
    P, O = engine_mod, oracle_mod
    o = O.Oracle((4, 4, 4, 4), N)
    o.random_start(13, 0.5)
    nz = O.Rand55(17).gauss(o.V * 32)

    def tiled(v):
        v = np.asarray(v).reshape(4, 4, 4, 4, -1)
        return np.ascontiguousarray(np.tile(v, (4, 4, 4, 4, 1)))

    shape = (-1,) + o.links.shape[1:]
    with P.NsptEngine((16, 16, 16, 16), N, update="onthefly") as e:
        e.set_gf_grid((8, 8, 8, 8))
        e.upload(tiled(o.links).reshape(shape))
        e.set_noise(tiled(nz).ravel())
        e.gauge_wilson(0.01)
        got = e.download()
    o.sweep(0.01, nz, onthefly=True, grid=(2, 2, 2, 2))
    assert per_order_rel(got, tiled(o.links).reshape(shape), N).max() <= 1e-12


def test_large_fields_cross_the_bus_whole(engine_mod):
    """Upload and download of a field that goes through the pinned buffers
    (28.7 MB: 14 chunks and a part of one), and of part of its orders."""
    P = engine_mod
    L, N = (8, 8, 8, 12), 8
    rng = np.random.default_rng(9)
    a = rng.normal(size=(int(np.prod(L)), 4, P.series_len(N)))
    with P.NsptEngine(L, N) as e, P.NsptEngine(L, N - 1) as f:
        e.upload(a)
        assert np.array_equal(e.download(), a)
        f.upload(a, allocORD=N)
        assert np.array_equal(f.download(), a[:, :, :P.series_len(N - 1)])
