"""The allocation-free plaquette on lattices with extents of 1, which contexts do
not take (GPU): against the sum over links of Tr(U * staples), nspt.cc:1362-1383,
written out link by link in numpy.  Flags other than 1 as well: a link read across a
twisted face has flag 1 (nspt.cc:115-121), so the four links of a plaquette see
flags of their own.

Tolerance 1e-13 of the largest order: a few hundred roundings of 1e-16."""
import ctypes
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def omega(d):
    w = np.exp(2j * np.pi / 3)
    m = np.zeros((3, 3), complex)
    if d == 1:
        m[0, 0], m[1, 1], m[2, 2] = w.conjugate(), 1, w
    elif d == 2:
        m[0, 1] = m[1, 2] = m[2, 0] = 1
    else:
        m[0, 1], m[1, 2], m[2, 0] = w.conjugate(), 1, w
    return m


def mul(a, b):
    return np.array([sum(a[i] @ b[k - i] for i in range(k + 1)) for k in range(len(a))])


def dag(a):
    return np.conj(np.swapaxes(a, 1, 2))


def plaquette(U, L, twist):
    """U[site][mu] a series (N + 1, 3, 3); sum over links of Tr(U * staples) / 72 V."""
    strides = [L[1] * L[2] * L[3], L[2] * L[3], L[3], 1]

    def link(mu, x, *moves):
        y = list(x)
        for d, s in moves:
            y[d] += s
        u, crossed = None, []
        for d in range(4):
            if not 0 <= y[d] < L[d]:
                if d in twist:
                    crossed.append((d, y[d] < 0))
                y[d] %= L[d]
        u = U[sum(y[d] * strides[d] for d in range(4))][mu]
        for back in (True, False):
            for d, b in crossed:
                if b == back:
                    o = omega(d).conj().T if b else omega(d)
                    u = o @ u @ o.conj().T
        if crossed:
            u = u.copy()
            u[0] = np.eye(3)
        return u

    total = 0
    for x in itertools.product(*map(range, L)):
        for mu in range(4):
            for nu in range(4):
                if nu == mu:
                    continue
                up = mul(mul(link(nu, x, (mu, 1)), dag(link(mu, x, (nu, 1)))), dag(link(nu, x)))
                low = mul(mul(dag(link(nu, x, (mu, 1), (nu, -1))), dag(link(mu, x, (nu, -1)))),
                          link(nu, x, (nu, -1)))
                total = total + np.trace(mul(link(mu, x), up + low), axis1=1, axis2=2)
    return total / (72 * np.prod(L))


@pytest.mark.parametrize("flags", [False, True], ids=["unit", "other_flags"])
@pytest.mark.parametrize("L,twist", [((1, 2, 3, 1), ()), ((1, 2, 3, 1), (1, 2)), ((2, 1, 1, 3), (1, 2, 3)),
                                     ((1, 1, 1, 1), (3,)), ((3, 4, 2, 1), (3,)), ((2, 3, 2, 4), (1, 2, 3))])
def test_thin_lattices(engine_mod, L, twist, flags):
    import torch
    lib = engine_mod._lib.load()
    N, V = 3, int(np.prod(L))
    rng = np.random.default_rng(4)
    c = rng.normal(size=(V, 4, 1 + 9 * N)) + 1j * rng.normal(size=(V, 4, 1 + 9 * N))
    if not flags:
        c[:, :, 0] = 1
    U = np.zeros((V, 4, N + 1, 3, 3), complex)
    U[:, :, 0] = c[:, :, 0, None, None] * np.eye(3)
    U[:, :, 1:] = c[:, :, 1:].reshape(V, 4, N, 3, 3)
    want = plaquette(U, L, twist)
    dev = torch.from_numpy(c.view(np.float64).reshape(-1)).to("cuda")
    torch.cuda.synchronize()
    got = np.zeros((N + 1, 2))
    rc = lib.nspt_plaquette_measure_noalloc(
        ctypes.c_void_p(dev.data_ptr()), N, (ctypes.c_int * 4)(*L), N, sum(1 << d for d in twist),
        got.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
    assert rc == 0
    got = got[:, 0] + 1j * got[:, 1]
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max(), (got, want)
