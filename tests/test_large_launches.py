"""The kernels' forms that only some launches reach, against the oracle (GPU,
through the C ABI).

Up to 14 orders a launch of at least 24 links per SM (3552 on 148 SMs) runs
with 9 lanes per link; a smaller one, and every higher order, with a warp per
link; runs with logarithms above 14 orders keep the order of their sums.  The
lattices here are as small as these launches can be, and each case names the
kernels that it is for.

Tolerances: 1e-12 per order after one sweep (tests/test_gpu_parity.py), 1e-11
with float-float products (tests/test_ff_precision.py).  Where logarithms are
taken, rounding grows with the order: the oracle is run a second time from a
start whose entries differ by 2^-52 of themselves, and the engine is held to 32
times that difference (a sum of some 1000 roundings, root 1000 = 32).
"""
import numpy as np
import pytest

from helpers import flag_diff, obs_close, per_order_rel

pytestmark = pytest.mark.gpu

TWIST = {"y": 2, "z": 4, "t": 8}
NINE = (6, 6, 5, 6)  # 4320 links, 6480 plaquettes


def other_flags(links):
    rng = np.random.default_rng(5)
    links[:, :, :2] = rng.normal(size=links[:, :, :2].shape)


def last_bit(links, seed):
    rng = np.random.default_rng(seed)
    links[:, :, 2:] *= 1.0 + 2.0 ** -52 * rng.choice([-1.0, 1.0], size=links[:, :, 2:].shape)


def run(P, O, L, N, tol, twist="", c1=0.0, flags=False, fa=False, onthefly=None, **kw):
    """One step of the engine and of the oracle (twice, see above), compared."""
    noise = O.Rand55(11).gauss(4 * 8 * int(np.prod(L)))
    zm = bool(kw.get("zero_modes"))
    outs = []
    for perturbed in (False, True):
        o = O.Oracle(L, N, twist_mask=sum(TWIST[d] for d in twist))
        o.random_start(3, 0.5)
        if flags:
            other_flags(o.links)
        if c1:
            o.set_action(c1)
        start = o.links.copy()
        if perturbed:
            last_bit(o.links, 7)
        how = dict(onthefly=True, grid=onthefly) if onthefly else {}
        obs = o.sweep(0.01, noise, zero_modes=zm, **how)
        if zm:
            o.zero_modes()
        if fa:
            o.fa_gauge_fix(0.05)
        outs.append((obs, o.links.copy(), o))
        if not (zm or fa):
            break
    obs, want, o = outs[0]
    bound = np.full(N, tol)
    if len(outs) == 2:
        bound = np.maximum(bound, 32 * per_order_rel(outs[1][1], want, N))
    with P.NsptEngine(L, N, twist=twist, fa=fa, **kw) as e:
        if onthefly:
            e.set_gf_grid(onthefly)
        e.upload(start)
        e.set_noise(noise)
        got = e.gauge_wilson(0.01)
        if c1:
            ok, worst = obs_close(e.rect_observables(), o.last_w2(), tol)
            assert ok, ("w2", worst)
        if zm:
            e.zero_modes_subtraction()
        if fa:
            e.FAstochastic_gauge_fixing(0.05)
        links = e.download()
    for a, b in ((got.plaq, obs.plaq), (got.norm, obs.norm), (got.tru, obs.tru)):
        ok, worst = obs_close(a, b, tol)
        assert ok, worst
    rel = per_order_rel(links, want, N)
    assert np.all(rel <= bound), (rel, bound)
    assert flag_diff(links, want, N) <= (tol if flags else 0.0)


@pytest.mark.parametrize("L,N", [((8, 8, 8, 8), 5), ((6, 6, 10, 10), 9), ((6, 6, 10, 10), 14)])
def test_zero_modes_and_fa(engine_mod, oracle_mod, L, N):
    """9 lanes: the sweep's logarithm, k_zero_modes, k_fa_gt, k_fa_apply."""
    run(engine_mod, oracle_mod, L, N, 1e-12, zero_modes=True, fa=True)


def test_fa_takes_its_own_logarithms(engine_mod, oracle_mod):
    """9 lanes: k_log_links (no zero modes)."""
    run(engine_mod, oracle_mod, (6, 6, 10, 10), 8, 1e-12, fa=True)


@pytest.mark.parametrize("L,N,twist", [(NINE, 5, ""), (NINE, 9, "yz"), (NINE, 14, ""),
                                       ((9, 10, 10, 12), 2, "t")])
def test_float_float(engine_mod, oracle_mod, L, N, twist):
    """k_plaq and k_update in float-float on large launches; the last in slabs."""
    run(engine_mod, oracle_mod, L, N, 1e-11, twist=twist, precision="ff")


@pytest.mark.parametrize("L", [(4, 2, 3, 4), NINE], ids=["warp", "large"])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("ff", 1e-11)])
def test_other_flags_across_twisted_faces(engine_mod, oracle_mod, L, precision, tol):
    """k_sweep_link, both precisions."""
    run(engine_mod, oracle_mod, L, 5, tol, twist="yz", flags=True, precision=precision)


@pytest.mark.parametrize("L,N,zm", [(NINE, 5, False), (NINE, 9, True), ((4, 4, 4, 4), 15, True)],
                         ids=["nine_n5", "nine_n9", "ordered"])
def test_improved_action(engine_mod, oracle_mod, L, N, zm):
    """k_sweep_imp with 9 lanes and with ordered sums."""
    run(engine_mod, oracle_mod, L, N, 1e-12, c1=-1.0 / 12.0, action="tlsym", zero_modes=zm)


@pytest.mark.parametrize("kind", ["onthefly", "onthefly_imp", "ff"])
def test_ordered_sums(engine_mod, oracle_mod, kind):
    """The ordered form of the on-the-fly and the float-float sweeps."""
    P, O, N = engine_mod, oracle_mod, 15
    if kind == "onthefly":
        run(P, O, (4, 4, 2, 4), N, 1e-12, zero_modes=True, update="onthefly", onthefly=(1, 2, 1, 2))
    elif kind == "onthefly_imp":
        run(P, O, (6, 6, 6, 4), N, 1e-12, zero_modes=True, update="onthefly", onthefly=(2, 2, 2, 1),
            c1=-1.0 / 12.0, action="tlsym")
    else:
        run(P, O, (4, 4, 2, 4), N, 1e-11, zero_modes=True, precision="ff")


@pytest.mark.parametrize("N", [5, 9, 14])
def test_wilson_loops(engine_mod, oracle_mod, N):
    """k_lines and k_loops with 9 lanes."""
    o = oracle_mod.Oracle(NINE, N)
    o.random_start(31 + N, 0.5)
    with engine_mod.NsptEngine(NINE, N) as e:
        e.upload(o.links)
        got = e.ComputeLoops()
    want = o.wilson_loops()
    for q in range(4):
        ok, worst = obs_close(got[q], want[q], 1e-12)
        assert ok, (q, worst)


def tiled(v, l, times):
    """A field (or noise) of an l^4 lattice repeated `times` in each direction."""
    v = np.asarray(v).reshape((l,) * 4 + (-1,))
    return np.ascontiguousarray(np.tile(v, (times,) * 4 + (1,)))


@pytest.mark.parametrize("N", [4, 14])
def test_local_gauge_fixing_of_many_threads(engine_mod, oracle_mod, N):
    """k_local_gf with 9 lanes: 4096 reference threads on 16^4, a 4^4 field
    repeated (blocks of 2 sites a side divide both)."""
    o = oracle_mod.Oracle((4, 4, 4, 4), N)
    o.random_start(13, 0.5)
    shape = (-1,) + o.links.shape[1:]
    with engine_mod.NsptEngine((16, 16, 16, 16), N) as e:
        e.set_gf_grid((8, 8, 8, 8))
        e.upload(tiled(o.links, 4, 4).reshape(shape))
        e.stochastic_gauge_fixing(-0.05)
        got = e.download()
    o.local_gauge_fix(-0.05, grid=(2, 2, 2, 2))
    assert per_order_rel(got, tiled(o.links, 4, 4).reshape(shape), N).max() <= 1e-12


def test_improved_action_on_the_fly_of_many_threads(engine_mod, oracle_mod):
    """k_sweep_imp_otf with 9 lanes: 4096 reference threads on 24^4, a 6^4 field
    repeated (blocks of 3 sites a side)."""
    N = 2
    o = oracle_mod.Oracle((6, 6, 6, 6), N)
    o.random_start(13, 0.5)
    o.set_action(-1.0 / 12.0)
    noise = oracle_mod.Rand55(17).gauss(o.V * 32)
    shape = (-1,) + o.links.shape[1:]
    with engine_mod.NsptEngine((24, 24, 24, 24), N, update="onthefly", action="tlsym") as e:
        e.set_gf_grid((8, 8, 8, 8))
        e.upload(tiled(o.links, 6, 4).reshape(shape))
        e.set_noise(tiled(noise, 6, 4).ravel())
        e.gauge_wilson(0.01)
        got = e.download()
    o.sweep(0.01, noise, onthefly=True, grid=(2, 2, 2, 2))
    assert per_order_rel(got, tiled(o.links, 6, 4).reshape(shape), N).max() <= 1e-12
