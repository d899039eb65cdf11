"""The plaquette records of the Jacobi sweep are memory that a context can do
without: what else is on the GPU changes neither a field nor whether a context
can be had.  Needs a B200 with a few hundred megabytes to leave free."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def fields(L, N):
    """Bytes of a context without the records, at most: both fields, the
    observables and the rows that their sums take (296 of up to 8 series)."""
    return (4 * int(np.prod(L)) * (2 * 16 * (1 + 9 * N) + 24 * N + 16 * (N + 1))
            + 296 * 64 * (1 + 9 * N) + 2 * MB)


class room:
    """All of the GPU's memory but `keep` bytes taken for a while."""

    def __init__(self, keep):
        import torch
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        assert free > keep
        self.block = torch.empty(free - keep, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def two_steps(P, L, N, **kw):
    with P.NsptEngine(L, N, **kw) as e:
        e.seed(7, 0)
        e.NsptEvolve(0.01, 2, 1)
        obs = e.observables()
        return e.download(), obs.plaq, obs.norm, obs.tru, e.device_bytes


@pytest.mark.parametrize("L,N,spare", [((8, 8, 8, 8), 24, 300), ((8, 8, 8, 8), 24, 180),
                                       ((4, 8, 16, 16), 16, 400)],
                         ids=["slabs_of_two", "slabs_of_one", "four_planes"])
def test_same_bits_in_smaller_slabs(engine_mod, L, N, spare):
    """Megabytes to spare for a part of the records."""
    P = engine_mod
    want = two_steps(P, L, N, twist="y")
    with room(fields(L, N) + spare * MB):
        got = two_steps(P, L, N, twist="y")
    assert fields(L, N) < got[-1] < want[-1]
    for a, b in zip(got[:-1], want[:-1]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("L,N,kw", [
    ((8, 8, 8, 8), 24, dict(twist="yz")),
    ((8, 8, 8, 8), 24, dict(precision="ff")),
    ((12, 12, 12, 12), 4, dict(twist="t", local_gf=True, alpha=-0.05)),
    ((12, 12, 12, 12), 4, dict(precision="ff")),
    ((12, 12, 12, 12), 5, dict(zero_modes=True)),
], ids=["warp", "warp_ff", "nine_lanes", "nine_lanes_ff", "nine_lanes_logs"])
def test_same_bits_without_the_records(engine_mod, L, N, kw):
    P = engine_mod
    want = two_steps(P, L, N, **kw)  # also loads the kernels and their local memory
    keep = fields(L, N) * (3 if kw.get("zero_modes") else 2) // 2 + 24 * MB
    with room(keep):
        got = two_steps(P, L, N, **kw)
    assert got[-1] < want[-1]  # this one had no records
    for a, b in zip(got[:-1], want[:-1]):
        assert np.array_equal(a, b)


def fill_until_the_records_go(P, L, N, kw, held, one):
    """Contexts created until those in `held` have given their records back."""
    more = []
    try:
        for _ in range(64):
            if sum(e.device_bytes for e in held) <= len(held) * one:
                return more
            more.append(P.NsptEngine(L, N, **kw))
        raise AssertionError("the records are still held")
    except BaseException:
        for e in more:
            e.close()
        raise


def test_contexts_find_the_room_they_had(engine_mod):
    """Contexts are created until the memory is full: the last is given the records
    of the first, and the first goes on as it would have."""
    P = engine_mod
    L, N, kw = (8, 8, 8, 8), 24, dict(twist="yz")
    one, records = fields(L, N), 4 * 1024 * 18 * 16 * (1 + 9 * N)
    with P.NsptEngine(L, N, **kw) as e:
        e.seed(7, 0)
        e.NsptEvolve(0.01, 4, 1)
        want = e.download()
    with room(one + 4 * records + 16 * MB), P.NsptEngine(L, N, **kw) as e:
        e.seed(7, 0)
        e.NsptEvolve(0.01, 2, 1)
        assert e.device_bytes > one + records // 2
        more = fill_until_the_records_go(P, L, N, kw, [e], one)
        e.NsptEvolve(0.01, 2, 1)
        assert e.device_bytes < one + records  # no more than a part of them
        assert np.array_equal(e.download(), want)
        for m in more:
            m.close()
        e.NsptEvolve(0.01, 1, 1)


def test_a_batch_finds_its_room_and_goes_on_without_records(engine_mod):
    """A batch whose fields fit but not its records; and a graph that was captured
    with records that are then taken back."""
    P = engine_mod
    L, N, kw = (8, 8, 8, 8), 24, dict(twist="yz")
    one, records = fields(L, N), 4 * 1024 * 18 * 16 * (1 + 9 * N)
    args = ([L, L], N, [0.01, 0.005], [3, 4])
    with P.NsptBatch(*args, **kw) as b:
        b.step(4, 1)
        want = [e.download() for e in b.replicas]
    with room(2 * one + 32 * MB), P.NsptBatch(*args, **kw) as b:
        b.step(4, 1)
        for e, w in zip(b.replicas, want):
            assert np.array_equal(e.download(), w)
    with room(2 * one + 6 * records), P.NsptBatch(*args, **kw) as b:
        b.step(2, 1)
        assert sum(e.device_bytes for e in b.replicas) > 2 * one
        more = fill_until_the_records_go(P, L, N, kw, b.replicas, one)
        b.step(2, 1)
        for e, w in zip(b.replicas, want):
            assert np.array_equal(e.download(), w)
        for m in more:
            m.close()
