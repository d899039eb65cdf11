"""The plaquette records of the Jacobi sweep are memory that a context can do
without: what else is on the GPU changes neither a field nor whether a context
can be had.  Needs a B200 with a few hundred megabytes to leave free."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def fields(L, N):
    """Bytes of a context without the records: both fields, the observables."""
    return 4 * int(np.prod(L)) * (2 * 16 * (1 + 9 * N) + 24 * N + 16 * (N + 1)) + 4 * MB


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
