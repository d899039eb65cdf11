"""Performance cases of the NSPT engine: what its users run, from the smallest
call to the largest.

A case is a plain dict.  `listed()` gives the named cases, `draw(rng)` one
more of the same ranges, `prepare(case, seed)` what a program holds before the
call (an engine with its field on the GPU, or a batch of them), `run(state)`
one pass through the public entry points, `work(case)` the bytes and FP64
operations the pass cannot do without, and `exact(case, seed)` the outputs of
that pass in plain torch, complex128, without the engine.

Keys of a case:
  call     "evolve"  NsptEvolve(dt, beat, gf_every), then the observables and
                     the links (a BEAT of the reference's driver and its
                     configuration)
           "sweep"   gauge_wilson(dt), which returns the sweep's observables
           "measure" plaquette_measure and, on periodic lattices,
                     ComputeLoops: what the driver prints after a BEAT
           "batch"   NsptBatch.step(beat) over replicas of three volumes, then
                     plaquettes and links
  x y z t  extents;  n  perturbative order;  twist  twisted directions
  zero_modes, gf ("none", "local", "fa"), alpha, gf_every, action, update,
  precision, dt, beat, and for a batch replicas
"""
from __future__ import annotations

import math

import numpy as np
import torch

import prlgt2020_b200 as nspt


def _case(call, L, n, **more):
    c = {"call": call, "x": L[0], "y": L[1], "z": L[2], "t": L[3], "n": n, "twist": "",
         "zero_modes": False, "gf": "none", "alpha": 0.0, "gf_every": 1, "action": "wil",
         "update": "jacobi", "precision": "fp64", "dt": 0.01, "beat": 1}
    c.update(more)
    return c


def listed():
    quench = {"zero_modes": True, "gf": "local", "alpha": -0.05}
    fourier = {"zero_modes": True, "gf": "fa", "alpha": 0.05}
    return [
        # one step of the smallest lattice a test or a first run uses: latency
        _case("evolve", (4, 4, 4, 4), 8, name="quench_4x4_n8", **quench),
        # the shipped Quench.cfg run (12^4, 8 orders, dt 0.005, zero modes and
        # local gauge fixing every step): a BEAT with the Jacobi update ...
        _case("evolve", (12, 12, 12, 12), 8, name="quench_12x4_n8", dt=0.005, beat=50, **quench),
        # ... and with the reference's default update
        _case("evolve", (12, 12, 12, 12), 8, name="quench_12x4_n8_onthefly", dt=0.005, beat=20,
              update="onthefly", **quench),
        # what the driver measures after every BEAT of that run
        _case("measure", (12, 12, 12, 12), 8, name="measure_12x4_n8"),
        # the Fourier-accelerated workload: 16^4, 20 orders
        _case("evolve", (16, 16, 16, 16), 20, name="fourier_16x4_n20", beat=20, **fourier),
        # 24 orders, twisted y and z, gauge fixing every 10 steps, on a lattice
        # of a finite-volume study
        _case("evolve", (8, 8, 8, 8), 24, name="twisted_8x4_n24", twist="yz", gf="local",
              alpha=-0.05, gf_every=10, dt=0.005, beat=60),
        # the headline benchmark's sweep; its 14.6 GB field stays on the GPU,
        # the program reads the sweep's observables
        _case("sweep", (32, 32, 32, 32), 24, name="twisted_32x4_n24", twist="yz", dt=0.005),
        # low order on a larger volume, one twisted direction
        _case("evolve", (16, 16, 16, 16), 4, name="twisted_t_16x4_n4", twist="t", gf="local",
              alpha=-0.05, dt=0.005, beat=50),
        # an improved action
        _case("evolve", (8, 8, 8, 8), 20, name="tlsym_8x4_n20", action="tlsym", beat=12,
              gf="local", alpha=-0.05),
        # float-float products at 40 orders (without the logarithms, which amplify
        # rounding a thousandfold every few orders and would hide it)
        _case("evolve", (8, 8, 8, 8), 40, name="floatfloat_8x4_n40", precision="ff", beat=8,
              gf="local", alpha=-0.05),
        # odd extents, one of them without a compile-time FFT plan, odd order
        _case("evolve", (5, 6, 7, 10), 13, name="fourier_5x6x7x10_n13", beat=40, **fourier),
        # replicas of three volumes and three time steps, 12 orders
        _case("batch", (4, 6, 8, 0), 12, name="replicas_n12", replicas=12, beat=20, **fourier),
    ]


def _links(case):
    return 4 * case["x"] * case["y"] * case["z"] * case["t"]


def _step_flops(case, n_links):
    """FP64 operations of one Langevin step, all links.  P(N) = N(N-1)/2
    products of 3x3 matrices are one truncated series product; a series exp or
    log counts as three of them (X^2, X^3's trace, the combination)."""
    N = case["n"]
    prod = 216.0 * N * (N - 1) / 2 + 216.0 * N
    count = {"wil": 12, "tlsym": 84, "iwa": 84, "dbw2": 84}[case["action"]] + 1 + 1 + 3
    if case["zero_modes"]:
        count += 3 + 3  # the sweep's log, the subtraction's exp
    if case["gf"] == "fa":
        count += 2 + 3 / 4
    elif case["gf"] == "local":
        count += (2 + 3 / 4) / case["gf_every"]
    return n_links * prod * count


def _volumes(case):
    """Replica extents of a batch: x^4, y^4, z^4 in turn."""
    return [(case["xyz"[r % 3]],) * 4 for r in range(case["replicas"])]


def work(case):
    N = case["n"]
    series = 16.0 * (1 + 9 * N)
    if case["call"] == "batch":
        nl = sum(4 * math.prod(L) for L in _volumes(case))
    else:
        nl = _links(case)
    if case["call"] == "measure":
        # per plane and site: a plaquette (4 links, closed by a trace) and six
        # loops of 28 path products, each closed by a trace
        prod = 216.0 * N * (N - 1) / 2
        planes = nl * 6 / 4
        return {"bytes": nl * series, "flops": planes * prod * (2 + 1 / 3 + 28 + 6 / 3)}
    passes = 2.0  # the field read and the field written
    if case["zero_modes"]:
        passes += 2.0  # the subtraction needs a sum over the whole updated field first
    if case["gf"] == "fa":
        passes += 2.0
    elif case["gf"] == "local":
        passes += 2.0 / case["gf_every"]
    return {"bytes": case["beat"] * passes * nl * series,
            "flops": case["beat"] * _step_flops(case, nl)}


def draw(rng):
    """A case of the listed ranges; sizes log-uniform, odd extents and orders
    among them, cheaper than the largest listed case."""
    call = rng.choice(["evolve", "evolve", "evolve", "evolve", "sweep", "measure"])
    N = int(round(math.exp(rng.uniform(math.log(3), math.log(32)))))
    L = [max(4, int(round(math.exp(rng.uniform(math.log(4), math.log(16.4)))))) for _ in range(4)]
    more = {"dt": rng.choice([0.005, 0.01, 0.02])}
    kind = rng.choice(["twist", "quench", "quench", "fourier", "fourier", "onthefly", "improved"])
    if call == "evolve":
        if kind == "twist":
            more.update(twist=rng.choice(["y", "t", "yz", "yzt"]), gf="local", alpha=-0.05,
                        gf_every=rng.choice([1, 5, 10]))
        elif kind == "fourier":
            more.update(zero_modes=True, gf="fa", alpha=0.05)
        else:
            more.update(zero_modes=rng.random() < 0.7, gf="local", alpha=-0.05)
        if more.get("zero_modes"):
            # the logarithm's order k is a sum of 2^(k-1) products that cancel:
            # past 16 orders its rounding drowns the comparison of two programs
            N = min(N, 16)
        if kind == "onthefly":
            L = [v + v % 2 for v in L]
            more.update(update="onthefly")
        elif kind == "improved":
            more.update(action=rng.choice(["tlsym", "iwa"]))
        if more["gf"] == "local":
            # the walk along an odd extent is serial, as the reference's is
            L = [v + v % 2 if i < 3 else v for i, v in enumerate(L)]
    elif call == "sweep":
        more.update(twist=rng.choice(["", "yz"]))
    while math.prod(L) * N * N > 4.0e6:  # about 12^4 at 14 orders
        i = max(range(4), key=lambda d: L[d])
        L[i] = max(4, L[i] // 2)
        if L[i] % 2 and more.get("gf") == "local":
            L[i] += 1
        if max(L) <= 4:
            break
    case = _case(call, L, N, **more)
    if call == "evolve":
        cost = _step_flops(case, _links(case)) / 5.0e12 + 4e-4  # seconds a step, roughly
        if more["gf"] == "local":
            cost += 3e-3 / case["gf_every"]
        if kind == "onthefly":
            cost += 6e-3
        case["beat"] = max(1, min(60, int(rng.uniform(0.1, 0.3) / cost)))
    return case


# ---------------- the start field: plain torch, seed alone ----------------
#
# Series are tensors (N + 1, ..., 3, 3) complex128, order 0 first.

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _mul(a, b):
    """Truncated Cauchy product."""
    n = a.shape[0]
    out = torch.zeros(torch.broadcast_shapes(a.shape, b.shape), dtype=a.dtype, device=a.device)
    for i in range(n):
        out[i:] += torch.matmul(a[i], b[: n - i])
    return out


def _dag(a):
    return a.conj().transpose(-1, -2)


def _one_like(a):
    o = torch.zeros_like(a)
    o[0] = torch.eye(3, dtype=a.dtype, device=a.device)
    return o


def _exp(x):
    """exp of a series without order 0: Horner, orders 1..N."""
    n = x.shape[0] - 1
    s = _one_like(x)
    for m in range(n, 0, -1):
        # only orders up to n - (m - 1) of this partial sum reach the result
        top = n - m + 2
        t = _mul(x[:top], s[:top]) / m
        t[0] += torch.eye(3, dtype=x.dtype, device=x.device)
        s = torch.zeros_like(x)
        s[:top] = t
    return s


def _log(u):
    """log of a series with order 0 = 1."""
    n = u.shape[0] - 1
    x = u.clone()
    x[0] = 0
    s = torch.zeros_like(x)
    for m in range(n, 0, -1):
        top = n - m + 2
        c = (1.0 if m % 2 else -1.0) / m
        t = s[:top].clone()
        t[0] += c * torch.eye(3, dtype=x.dtype, device=x.device)
        t = _mul(x[:top], t)
        s = torch.zeros_like(x)
        s[:top] = t
    return s


def _reh(a):
    """Traceless antihermitian part, no order 0."""
    b = 0.5 * (a - _dag(a))
    tr = torch.diagonal(b, dim1=-2, dim2=-1).sum(-1) / 3.0
    b = b - tr[..., None, None] * torch.eye(3, dtype=a.dtype, device=a.device)
    b[0] = 0
    return b


def _start(L, N, seed):
    """U_mu(x), a series (N + 1, 4, V, 3, 3): order-k coefficients of the
    logarithm Gaussian with standard deviation 0.5^k, projected to su(3)."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))
    V = math.prod(L)
    a = torch.randn((N + 1, 4, V, 3, 3, 2), generator=g, device=dev, dtype=torch.float64)
    a = torch.view_as_complex(a)
    a *= torch.tensor([0.5 ** k for k in range(N + 1)], device=dev,
                      dtype=torch.float64).reshape(-1, 1, 1, 1, 1)
    return _exp(_reh(a))


def _to_host(U):
    """The engine's host layout: (V, 4, 2 + 18 N) float64."""
    n, _, V = U.shape[:3]
    out = torch.empty((V, 4, 2 + 18 * (n - 1)), dtype=torch.float64, device=U.device)
    out[:, :, 0] = U[0, :, :, 0, 0].real.T
    out[:, :, 1] = U[0, :, :, 0, 0].imag.T
    v = torch.view_as_real(U[1:].resolve_conj().contiguous())  # (N, 4, V, 3, 3, 2)
    out[:, :, 2:] = v.permute(2, 1, 0, 3, 4, 5).reshape(V, 4, -1)
    return out.cpu().numpy()


def _extents(case):
    return (case["x"], case["y"], case["z"], case["t"])


def _batch_table(case, seed):
    """(extents, dt, noise seed, start seed) of every replica."""
    return [(L, case["dt"] * (0.5, 1.0, 2.0)[(r // 3) % 3], 1000 * seed + r, 7919 * seed + r)
            for r, L in enumerate(_volumes(case))]


# ---------------- what is measured ----------------

def prepare(case, seed):
    seed = int(seed)
    if case["call"] == "batch":
        table = _batch_table(case, seed)
        b = nspt.NsptBatch([L for L, _, _, _ in table], case["n"], [dt for _, dt, _, _ in table],
                           [s for _, _, s, _ in table], zero_modes=case["zero_modes"],
                           fa=case["gf"] == "fa", local_gf=case["gf"] == "local",
                           alpha=case["alpha"])
        for e, (L, _, _, start) in zip(b.replicas, table):
            e.upload(_to_host(_start(L, case["n"], start)))
        return {"case": case, "batch": b}
    L = _extents(case)
    e = nspt.NsptEngine(L, case["n"], twist=case["twist"], zero_modes=case["zero_modes"],
                        fa=case["gf"] == "fa", local_gf=case["gf"] == "local",
                        alpha=case["alpha"], action=case["action"],
                        precision=case["precision"], update=case["update"])
    e.seed(seed)
    if _links(case) * case["n"] > 4 * 16 ** 4 * 20:
        # too large to make on the host in good time: a run's first steps
        e.cold_start()
        e.NsptEvolve(0.05, 2, 0)
    else:
        e.upload(_to_host(_start(L, case["n"], seed)))
    return {"case": case, "engine": e}


def run(state):
    case = state["case"]
    if case["call"] == "batch":
        b = state["batch"]
        b.step(case["beat"], case["gf_every"])
        return [b.plaquettes()] + [e.download() for e in b.replicas]
    e = state["engine"]
    if case["call"] == "measure":
        plaq = e.plaquette_measure()
        return [plaq] if case["twist"] else [plaq, e.ComputeLoops()]
    if case["call"] == "sweep":
        obs = e.gauge_wilson(case["dt"])
        return [obs.plaq, obs.norm, obs.tru]
    e.NsptEvolve(case["dt"], case["beat"], case["gf_every"])
    obs = e.observables()
    return [obs.plaq, obs.norm, obs.tru, e.download()]


# ---------------- the same in plain torch, 64 bits ----------------

def _philox(link, q, step, seed):
    """Philox-4x32-10, counter (link, q, step), vectorised over link."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [link.astype(np.uint64), np.full_like(link, q, dtype=np.uint64),
         np.full_like(link, step & 0xFFFFFFFF, dtype=np.uint64),
         np.full_like(link, step >> 32, dtype=np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32,
             (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _noise(V, seed, step, dev):
    """su(3) Gaussian noise of every link, (4, V, 3, 3)."""
    link = np.arange(4 * V, dtype=np.uint64)
    g = []
    for q in range(4):
        r = _philox(link, q, step, seed)
        u1, u2 = ((((a << np.uint64(32)) | b) >> np.uint64(11)).astype(np.float64) + 1.0
                  for a, b in ((r[0], r[1]), (r[2], r[3])))
        u1, u2 = u1 * 2.0 ** -53, u2 * 2.0 ** -53
        rad = np.sqrt(-np.log(u1))
        g += [rad * np.cos(2 * np.pi * u2), rad * np.sin(2 * np.pi * u2)]
    m = np.zeros((4 * V, 3, 3), dtype=np.complex128)
    m[:, 0, 1], m[:, 1, 0] = g[1] + 1j * g[0], -g[1] + 1j * g[0]
    m[:, 0, 2], m[:, 2, 0] = g[3] + 1j * g[2], -g[3] + 1j * g[2]
    m[:, 1, 2], m[:, 2, 1] = g[5] + 1j * g[4], -g[5] + 1j * g[4]
    gg = g[7] / math.sqrt(3.0)
    m[:, 0, 0], m[:, 1, 1], m[:, 2, 2] = 1j * (gg + g[6]), 1j * (gg - g[6]), -2j * gg
    return torch.from_numpy(m).to(dev).reshape(4, V, 3, 3)


def _omega(d):
    w = complex(math.cos(2 * math.pi / 3), math.sin(2 * math.pi / 3))
    m = np.zeros((3, 3), dtype=np.complex128)
    if d == 1:
        m[0, 0], m[1, 1], m[2, 2] = w.conjugate(), 1, w
    elif d == 2:
        m[0, 1] = m[1, 2] = m[2, 0] = 1
    else:
        m[0, 1], m[1, 2], m[2, 0] = w.conjugate(), 1, w
    return m


class _Plain:
    """The Langevin step on a field U (N + 1, 4, V, 3, 3)."""

    def __init__(self, case, L, U, seed):
        self.c, self.L, self.U, self.seed, self.step = case, L, U, int(seed), 0
        self.dev, self.V, self.N = U.device, math.prod(L), U.shape[0] - 1
        self.x = torch.from_numpy(np.stack(np.unravel_index(np.arange(self.V), L))).to(self.dev)
        self.twist = ["xyzt".index(d) for d in case["twist"]]
        self.om = {d: torch.from_numpy(_omega(d)).to(self.dev) for d in self.twist}
        self.stale = None  # on the fly: what a read across a twisted face sees

    def site(self, sites, *moves):
        """Site reached by the (direction, steps) moves, and the faces crossed."""
        y = self.x[:, sites].clone()
        for d, s in moves:
            y[d] += s
        wrap = {}
        for d in range(4):
            wrap[d] = (y[d] < 0, y[d] >= self.L[d])
            y[d] %= self.L[d]
        s = ((y[0] * self.L[1] + y[1]) * self.L[2] + y[2]) * self.L[3] + y[3]
        return s, wrap

    def link(self, mu, sites, *moves):
        s, wrap = self.site(sites, *moves)
        u = self.U[:, mu, s]
        if not self.twist:
            return u
        cross = torch.zeros_like(s, dtype=torch.bool)
        for d in self.twist:
            cross |= wrap[d][0] | wrap[d][1]
        if self.stale is not None:
            u = torch.where(cross[:, None, None], self.stale[:, mu, s], u)
        for side in (0, 1):
            for d in self.twist:
                o = self.om[d] if side else self.om[d].conj().T
                tw = torch.matmul(torch.matmul(o, u), o.conj().T)
                u = torch.where(wrap[d][side][:, None, None], tw, u)
        return u

    def chain(self, sites, path):
        out = None
        for mu, moves, dag in path:
            u = self.link(mu, sites, *moves)
            u = _dag(u) if dag else u
            out = u if out is None else _mul(out, u)
        return out

    def staples(self, mu, sites):
        w = w2 = 0
        for nu in range(4):
            if nu == mu:
                continue

            def at(i, j, nu=nu):
                return ((mu, i), (nu, j))

            w = w + self.chain(sites, [(nu, at(1, 0), 0), (mu, at(0, 1), 1), (nu, at(0, 0), 1)])
            w = w + self.chain(sites, [(nu, at(1, -1), 1), (mu, at(0, -1), 1), (nu, at(0, -1), 0)])
            if self.c["action"] == "wil":
                continue
            # the six 2x1 rectangles: direction (m: mu, n: nu), offset along
            # mu and nu, and the dagger of every link
            for path in ("n+1+0 m+0+1' m-1+1' n-1+0' m-1+0", "n+1-1' m+0-1' m-1-1' n-1-1 m-1+0",
                         "n+1+0 n+1+1 m+0+2' n+0+1' n+0+0'", "m+1+0 n+2+0 m+1+1' m+0+1' n+0+0'",
                         "n+1-1' n+1-2' m+0-2' n+0-2 n+0-1", "m+1+0 n+2-1' m+1-1' m+0-1' n+0-1"):
                w2 = w2 + self.chain(sites, [(mu if p[0] == "m" else nu,
                                              at(int(p[1:3]), int(p[3:5])), p.endswith("'"))
                                             for p in path.split()])
        return w, w2

    def update(self, mu, sites, eta):
        """New links and the sums of the observables."""
        u = self.U[:, mu, sites]
        w, w2 = self.staples(mu, sites)
        p = _mul(u, w)
        tr = torch.diagonal(p, dim1=-2, dim2=-1).sum((-1, -2))
        f = p
        if self.c["action"] != "wil":
            c1 = {"tlsym": -1.0 / 12.0, "iwa": -0.331, "dbw2": -1.4088}[self.c["action"]]
            f = (1 - 8 * c1) * p + c1 * _mul(u, w2)
        f = _reh(f) * (-self.c["dt"] / 6.0)
        f[1] -= math.sqrt(self.c["dt"]) * eta[mu, sites]
        norm = (u.abs() ** 2).sum((-1, -2, -3))
        tru = torch.diagonal(u, dim1=-2, dim2=-1).sum((-1, -2))
        return _mul(_exp(f), u), tr, norm, tru

    def thread_grid(self):
        """Sites of each barrier step of the default thread grid, in order:
        a list of lists of site tensors (the walk inside a barrier step)."""
        minb = 3 if self.c["update"] == "onthefly" and self.c["action"] != "wil" else 2
        n = []
        for v in self.L:
            b = minb
            while minb == 3 and v % b:
                b += 1
            n.append(v // b if v % b == 0 else 1)
        bs = [v // k for v, k in zip(self.L, n)]
        dmax = max([d for d in range(4) if n[d] > 1], default=-1)
        th = np.stack(np.unravel_index(np.arange(math.prod(n)), n))
        walked = [self.L[d] for d in range(dmax + 1, 4)]
        for p in np.ndindex(*bs[: dmax + 1]):
            for q in np.ndindex(*walked):
                x = [bs[d] * th[d] + p[d] if d <= dmax else np.full_like(th[0], q[d - dmax - 1])
                     for d in range(4)]
                yield torch.from_numpy(np.ravel_multi_index(x, self.L)).to(self.dev)

    def sweep(self):
        eta = _noise(self.V, self.seed, self.step, self.dev)
        self.step += 1
        n1 = self.N + 1
        tr = torch.zeros(n1, dtype=torch.complex128, device=self.dev)
        norm = torch.zeros(n1, dtype=torch.float64, device=self.dev)
        tru = torch.zeros((4, n1), dtype=torch.complex128, device=self.dev)
        if self.c["update"] == "onthefly":
            self.stale = self.U.clone() if self.twist else None
            for sites in self.thread_grid():
                for mu in range(4):
                    new, a, b, c = self.update(mu, sites, eta)
                    self.U[:, mu, sites] = new
                    tr, norm = tr + a, norm + b
                    tru[mu] += c
        else:
            every = torch.arange(self.V, device=self.dev)
            out = torch.empty_like(self.U)
            for mu in range(4):
                out[:, mu], a, b, c = self.update(mu, every, eta)
                tr, norm = tr + a, norm + b
                tru[mu] += c
            self.U = out
        return [torch.view_as_real(tr / (72 * self.V)), norm[1:] / (12 * self.V),
                torch.view_as_real(tru[:, 1:] / (3 * self.V))]

    def zero_modes(self):
        lg = _log(self.U)
        self.U = _exp(_reh(lg - lg.mean(dim=2, keepdim=True)))

    def fourier(self, alpha):
        lg = _log(self.U)
        every = torch.arange(self.V, device=self.dev)
        w = 0
        for mu in range(4):
            w = w + lg[:, mu] - lg[:, mu, self.site(every, (mu, -1))[0]]
        w = torch.fft.fftn(w.reshape(-1, *self.L, 3, 3), dim=(1, 2, 3, 4))
        p2 = 0
        for d, v in enumerate(self.L):
            n = torch.arange(v, device=self.dev, dtype=torch.float64)
            q = 4 * torch.sin(math.pi * n / v) ** 2
            p2 = p2 + q.reshape([-1 if i == d else 1 for i in range(4)])
        p2[0, 0, 0, 0] = math.inf
        w = torch.fft.ifftn(w * (-alpha / p2)[None, ..., None, None], dim=(1, 2, 3, 4))
        g = _exp(_reh(w.reshape(-1, self.V, 3, 3)))
        for mu in range(4):
            up = g[:, self.site(every, (mu, 1))[0]]
            self.U[:, mu] = _mul(_mul(g, self.U[:, mu]), _dag(up))

    def local(self, alpha):
        for sites in self.thread_grid():
            w = 0
            for mu in range(4):
                w = w + self.U[:, mu, sites] - self.link(mu, sites, (mu, -1))
            w = 2 * _reh(w) * alpha
            e1, e2 = _exp(w), _exp(-w)
            for mu in range(4):
                self.U[:, mu, sites] = _mul(e1, self.U[:, mu, sites])
                back, wrap = self.site(sites, (mu, -1))
                r = e2
                if mu in self.twist:
                    o = self.om[mu]
                    tw = torch.matmul(torch.matmul(o, e2), o.conj().T)
                    r = torch.where(wrap[mu][0][:, None, None], tw, e2)
                self.U[:, mu, back] = _mul(self.U[:, mu, back], r)

    def evolve(self, beat):
        obs = None
        for _ in range(beat):
            obs = self.sweep()
            if self.c["zero_modes"]:
                self.zero_modes()
            if self.step % self.c["gf_every"] == 0:
                if self.c["gf"] == "fa":
                    self.fourier(self.c["alpha"])
                elif self.c["gf"] == "local":
                    self.local(self.c["alpha"])
            self.stale = None
        return obs

    def plaquette(self):
        every = torch.arange(self.V, device=self.dev)
        tr = 0
        for mu in range(4):
            p = _mul(self.U[:, mu], self.staples(mu, every)[0])
            tr = tr + torch.diagonal(p, dim1=-2, dim2=-1).sum((-1, -2))
        return torch.view_as_real(tr / (72 * self.V))

    def loops(self):
        """1x2, 2x2, 2x4 and 4x4 loops, the first and third in both
        orientations."""
        every = torch.arange(self.V, device=self.dev)
        sums = torch.zeros((4, self.N + 1), dtype=torch.complex128, device=self.dev)
        for mu in range(4):
            for nu in range(mu + 1, 4):
                for q, i, j in ((0, 2, 1), (0, 1, 2), (1, 2, 2), (2, 2, 4), (2, 4, 2), (3, 4, 4)):
                    one = self.chain(every, [(mu, ((mu, a),), 0) for a in range(i)]
                                     + [(nu, ((mu, i), (nu, b)), 0) for b in range(j)])
                    two = self.chain(every, [(nu, ((nu, b),), 0) for b in range(j)]
                                     + [(mu, ((nu, j), (mu, a)), 0) for a in range(i)])
                    p = _mul(one, _dag(two))
                    sums[q] += torch.diagonal(p, dim1=-2, dim2=-1).sum((-1, -2))
        half = torch.tensor([0.5, 1.0, 0.5, 1.0], device=self.dev, dtype=torch.float64)
        return torch.view_as_real(sums * (half / (18.0 * self.V))[:, None])


def exact(case, seed):
    """run()'s outputs in complex128 torch, or None where that takes long (a
    large lattice) or the start field is the engine's own."""
    seed = int(seed)
    if case["call"] == "batch":
        plaq, links = [], []
        for L, dt, noise, start in _batch_table(case, seed):
            p = _Plain(dict(case, dt=dt), L, _start(L, case["n"], start), noise)
            plaq.append(p.evolve(case["beat"])[0])
            links.append(_to_host(p.U))
        return [torch.stack(plaq)] + links
    times = 7 if case["action"] != "wil" else 2 if case["update"] == "onthefly" else 1
    if _links(case) * case["n"] ** 2 * case["beat"] * times > 1.2e9:
        return None
    p = _Plain(case, _extents(case), _start(_extents(case), case["n"], seed), seed)
    if case["call"] == "measure":
        plaq = p.plaquette()
        return [plaq] if case["twist"] else [plaq, p.loops()]
    obs = p.evolve(case["beat"] if case["call"] == "evolve" else 1)
    return obs + [_to_host(p.U)] if case["call"] == "evolve" else obs
