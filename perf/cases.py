"""Performance cases of the SPME framework: what its users have it do, by public entry points.

``listed()`` are the fixed cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a
program holds before the call (inputs from the seed, solver handles, result buffers), ``run`` is one pass,
``work`` the bytes and operations a pass cannot do without, and ``exact`` the same outputs in FP64 by plain
torch.  Units are nm and e, as in the benchmark configurations (ewaldcorrel_b200/configs.py).

Kinds:
  solve   SpmeSolver.solve: energy, virial, forces and potentials of device-resident charges (an MD step)
  real    SpmeSolver.real_space: the short-range Ewald term of the same step
  batch   SpmeBatch forward and backward: dE/dx, dE/dq and dE/dL of many small systems (a training step)
  host    the ewald.py interface on numpy arrays: sfac, de1, de2, potl
  frames  structure factors over trajectory frames: sfac and |S|^2 sums, then the sums are read
  serve   a burst of uneven requests through SpmeServer, host arrays in and out
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

MAX_M_FACTOR = math.sqrt(math.log(1e16)) / math.pi  # reciprocal cutoff per beta (configs.py)
DENSITY = 100.0  # atoms per nm^3, as water's

_stream = None


def _compute_stream():
    """The one stream on which the program's solvers work, one solve after another."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---------------------------------------------------------------- cases

def _box(case):
    return np.array([case[k] for k in ("ax", "by", "cz", "bx", "cx", "cy")], dtype=np.float64)


def _grid(case):
    return (case["K0"], case["K1"], case["K2"])


def _system(kind, n, K, order, beta, L, data="uniform", **more):
    return dict(kind=kind, n=n, K0=K[0], K1=K[1], K2=K[2], order=order, beta=beta, ax=L[0], by=L[1], cz=L[2],
                bx=L[3], cx=L[4], cy=L[5], data=data, **more)


def listed():
    cube = [0.0, 0.0, 0.0]
    return [
        # the plain configuration: 1000 charges, where launches and latency count
        dict(name="solve_plain", **_system("solve", 1000, (32, 32, 32), 4, 3.47, [3.0, 3.0, 3.0] + cube)),
        # an odd triclinic cell: order 8, an odd last axis, a factor 7, a ragged atom count
        dict(name="solve_odd", **_system("solve", 50021, (84, 90, 75), 8, 3.2, [8.9, 8.6, 7.7, 1.3, -0.8, 2.1])),
        # the water box: the usual size of a biomolecular simulation
        dict(name="solve_water", **_system("solve", 98304, (96, 96, 96), 4, 3.12, [10.0] * 3 + cube, "water")),
        # the large triclinic system
        dict(name="solve_large", **_system("solve", 1048576, (256, 256, 256), 6, 3.5,
                                           [20.0, 17.320508075688775, 20.0, 10.0, 0.0, 0.0])),
        # the real-space term of the water box at the usual cutoff
        dict(name="real_water", **_system("real", 98304, (96, 96, 96), 4, 3.12, [10.0] * 3 + cube, "water",
                                          rcut=1.0)),
        # a training step over small periodic systems of different sizes
        dict(name="batch_grad", kind="batch", count=16, shapes=4),
        # the drop-in interface on a program's own numpy arrays
        dict(name="host_numpy", **_system("host", 24000, (64, 64, 64), 6, 3.12, [6.2145] * 3 + cube, "water")),
        # S(k) of a trajectory, four frames read as one sum
        dict(name="frames_sk", **_system("frames", 30000, (72, 72, 72), 4, 3.12, [6.6943] * 3 + cube, "water",
                                         frames=4)),
        # requests of a serving stream that arrive together
        dict(name="serve_burst", kind="serve", count=24, shapes=5, nmax=60000),
    ]


def _smooth(v, primes=(2, 3, 5)):
    m = max(1, int(math.ceil(v)))
    while True:
        r = m
        for p in primes:
            while r % p == 0:
                r //= p
        if r == 1:
            return m
        m += 1


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_system(rng, kind, lo, hi, orders=(4, 4, 6, 6, 8), **more):
    order = rng.choice(orders)
    n = int(round(_log_uniform(rng, lo, min(hi, 300000) if order == 8 else hi)))
    data = rng.choice(("uniform", "water"))
    if data == "water":
        n = max(3, n // 3 * 3)
    side = (n / rng.uniform(0.6 * DENSITY, 1.3 * DENSITY)) ** (1.0 / 3.0)
    asp = [rng.uniform(0.85, 1.2) for _ in range(3)]
    L = [side * a for a in asp] + [0.0, 0.0, 0.0]
    if rng.random() < 0.4:  # triclinic
        L[3], L[4], L[5] = (rng.uniform(-0.5, 0.5) * L[k] for k in (0, 0, 1))
    h = rng.uniform(0.08, 0.12)
    primes = rng.choice(((2, 3, 5), (2, 3, 5), (2, 3, 5, 7)))
    K = [min(256, max(24, _smooth(L[d] / h, primes))) for d in range(3)]
    return _system(kind, n, K, order, round(rng.uniform(2.6, 3.6), 3), L, data, **more)


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "solve", "real", "batch", "host", "frames", "serve"))
    if kind == "solve":
        return _draw_system(rng, kind, 500, 1000000)
    if kind == "real":
        c = _draw_system(rng, kind, 6000, 300000)
        c["rcut"] = round(rng.uniform(0.8, 1.2), 3)
        return c
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 24), shapes=rng.randint(10, 10 ** 6))
    if kind == "host":
        return _draw_system(rng, kind, 1000, 150000)
    if kind == "frames":
        return _draw_system(rng, kind, 3000, 100000, frames=rng.randint(2, 5))
    return dict(kind=kind, count=rng.randint(8, 32), shapes=rng.randint(10, 10 ** 6),
                nmax=int(_log_uniform(rng, 4000, 100000)))


def _batch_systems(case):
    """The batch's systems: 64 to 2048 charges in cubes of 1.5 to 4 nm, 24^3 to 48^3 grids."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        n, side = int(round(_log_uniform(r, 64, 2048))), r.uniform(1.5, 4.0)
        k = min(48, max(24, _smooth(side / 0.1)))
        out.append(_system("batch", n, (k, k, k), 4, 3.47, [side] * 3 + [0.0, 0.0, 0.0]))
    return out


def _serve_systems(case):
    """The burst's requests: atoms log-uniform from 500, cubes at water's density, order 4 or 6."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        n = int(round(_log_uniform(r, 500, case["nmax"])))
        side = (n / DENSITY) ** (1.0 / 3.0)
        k = min(128, max(24, _smooth(round(side / 0.1))))
        out.append(_system("serve", n, (k, k, k), r.choice((4, 6)), 3.12, [side] * 3 + [0.0, 0.0, 0.0]))
    return out


# ---------------------------------------------------------------- inputs

def _rows(L, like):
    return torch.tensor([[L[0], 0.0, 0.0], [L[3], L[1], 0.0], [L[4], L[5], L[2]]], dtype=torch.float64,
                        device=like.device)


def _water(n, L, g, dev):
    """Rigid 3-site molecules (O-H 0.09572 nm, 104.52 deg) at uniform centres and orientations."""
    m = (n + 2) // 3
    c = torch.rand((m, 3), generator=g, device=dev, dtype=torch.float64)
    c = c @ _rows(L, c)
    v = torch.randn((m, 4), generator=g, device=dev, dtype=torch.float64)
    w, x, y, z = (v / v.norm(dim=1, keepdim=True)).unbind(1)
    a, half = 0.09572, math.radians(104.52) / 2
    e1 = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], 1) * (a * math.sin(half))
    e2 = torch.stack([2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w)], 1) * (a * math.cos(half))
    pos = torch.stack([c, c + e2 + e1, c + e2 - e1], 1).reshape(-1, 3)[:n].contiguous()
    q = torch.tensor([-0.834, 0.417, 0.417], dtype=torch.float64, device=dev).repeat(m)[:n].contiguous()
    return pos, q


def _inputs(case, seed, dev=None):
    """Positions (n x 3) and charges (n), FP64."""
    dev = dev or torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    n, L = case["n"], _box(case)
    if case["data"] == "water":
        return _water(n, L, g, dev)
    s = torch.rand((n, 3), generator=g, device=dev, dtype=torch.float64)
    q = 0.5 * torch.randn(n, generator=g, device=dev, dtype=torch.float64)
    return (s @ _rows(L, s)).contiguous(), q - q.mean()


def _many(cases, seed):
    return [_inputs(c, 1000 * int(seed) + i) for i, c in enumerate(cases)]


def _frames(case, seed):
    return [_inputs(case, 1000 * int(seed) + i) for i in range(case["frames"])]


def _pinned(a):
    return torch.empty(a.shape, dtype=torch.float64, pin_memory=True).copy_(a).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "real"):
        from ewaldcorrel_b200.device import SpmeSolver

        x, q = _inputs(case, seed)
        n = case["n"]
        s = SpmeSolver(_box(case), _grid(case), case["order"], case["beta"], MAX_M_FACTOR * case["beta"],
                       stream=_compute_stream())
        st = dict(kind=kind, solver=s, x=x, q=q, dx=torch.empty((n, 3), dtype=torch.float64, device=x.device))
        if kind == "solve":
            st["phi"] = torch.empty(n, dtype=torch.float64, device=x.device)
            st["ev"] = torch.empty(7, dtype=torch.float64, device=x.device)
        else:
            st.update(out=torch.empty(10, dtype=torch.float64, device=x.device), eta=case["beta"], rcut=case["rcut"])
        return st
    if kind == "batch":
        from ewaldcorrel_b200.autograd import SpmeBatch

        systems = _batch_systems(case)
        xq = _many(systems, seed)
        x = torch.cat([a for a, _ in xq]).requires_grad_()
        q = torch.cat([b for _, b in xq]).requires_grad_()
        L = torch.tensor(np.stack([_box(c) for c in systems]), requires_grad=True)
        batch = SpmeBatch([(c["n"], _grid(c), c["order"], c["beta"]) for c in systems])
        batch(x, q, L)  # a training program's plans know their boxes after the first step
        return dict(kind=kind, batch=batch, x=x, q=q, L=L)
    if kind in ("host", "frames"):
        from ewaldcorrel_b200.ewald import Sfac

        sets = [_inputs(case, seed)] if kind == "host" else _frames(case, seed)
        s = Sfac(_box(case), np.array(_grid(case)), case["order"])
        s.set_ewald(case["beta"], MAX_M_FACTOR * case["beta"])
        return dict(kind=kind, sfac=s, sets=[(a.cpu().numpy(), b.cpu().numpy()) for a, b in sets])
    from ewaldcorrel_b200.serve import Request, SpmeServer

    systems = _serve_systems(case)
    calls = []
    for i, (c, (x, q)) in enumerate(zip(systems, _many(systems, seed))):
        x, q = _pinned(x), _pinned(q)
        req = Request(i, x, q, _box(c), _grid(c), c["order"], c["beta"], MAX_M_FACTOR * c["beta"])
        calls.append((req, x, torch.empty(7 + 4 * c["n"], dtype=torch.float64, pin_memory=True).numpy()))
    st = dict(kind="serve", server=SpmeServer(budget_bytes=8 << 30, max_inflight=64), calls=calls)
    run(st)  # a server in use has its solvers resident
    return st


# ---------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["solver"]
        ev = s.solve(state["x"], state["q"], state["dx"], state["phi"], state["ev"])
        return ev, state["dx"], state["phi"]
    if kind == "real":
        out = state["solver"].real_space(state["x"], state["q"], state["eta"], state["rcut"], state["out"],
                                         state["dx"])
        return out, state["dx"]
    if kind == "batch":
        x, q, L = state["x"], state["q"], state["L"]
        E = state["batch"](x, q, L)
        return (E.detach(), *torch.autograd.grad(E.sum(), (x, q, L)))
    s = state.get("sfac")
    if kind == "host":
        x, q = state["sets"][0]
        s.sfac(q, x)
        vir, dx, phi = np.zeros(6), np.zeros_like(x), np.zeros_like(q)
        E = s.de1(vir)
        s.de2(len(q), q, x, dx)
        s.potl(len(q), x, phi)
        return E, vir, dx, phi
    if kind == "frames":
        s.sk_reset()
        for x, q in state["sets"]:
            s.sfac(q, x)
            s.sk_accumulate()
        return s.sk_get()
    server, calls = state["server"], state["calls"]
    left, nxt = len(calls), 0
    while left:
        while nxt < len(calls):
            rc = server.submit(*calls[nxt])
            if rc == 1:
                break
            if rc != 0:
                raise RuntimeError("request refused")
            nxt += 1
        for _, status in server.poll():
            if status != 0:
                raise RuntimeError("request failed")
            left -= 1
    return [out for _, _, out in calls]


# ---------------------------------------------------------------- work

def _solve_work(c, gather=True):
    G, n, P = float(c["K0"] * c["K1"] * c["K2"]), c["n"], c["order"]
    fft = 2.5 * G * math.log2(G)
    fl = n * 2.0 * P ** 3 + fft
    if gather:
        fl += n * (4.0 * P ** 3 + 6.0 * P * P) + fft + 10.0 * G
    return fl


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        cs = _batch_systems(case) if kind == "batch" else _serve_systems(case)
        return dict(bytes=sum(64.0 * c["n"] + 104.0 for c in cs), flops=sum(_solve_work(c) for c in cs))
    n = case["n"]
    if kind in ("solve", "host"):
        return dict(bytes=64.0 * n + 56.0, flops=_solve_work(case))
    if kind == "frames":
        modes = case["K0"] * case["K1"] * (case["K2"] // 2 + 1)
        return dict(bytes=case["frames"] * 32.0 * n + 8.0 * modes,
                    flops=case["frames"] * (_solve_work(case, False) + 8.0 * modes))
    V = case["ax"] * case["by"] * case["cz"]
    pairs = 0.5 * n * (n / V) * 4.0 / 3.0 * math.pi * case["rcut"] ** 3
    return dict(bytes=56.0 * n + 80.0, flops=45.0 * pairs)


# ---------------------------------------------------------------- FP64 values

def _inverse_box(L):
    iV = 1.0 / (L[0] * L[1] * L[2])
    return iV, [[1.0 / L[0], 0.0, 0.0], [-L[3] * L[2] * iV, 1.0 / L[1], 0.0],
                [(L[3] * L[5] - L[1] * L[4]) * iV, -L[0] * L[5] * iV, 1.0 / L[2]]]


def _spline(P, f):
    """M_P(f + P - 1 - i) and its derivative for i = 0..P-1, f in [0, 1): (n x P) each."""
    m = [1.0 - f, f]  # M_2(f + 1), M_2(f): index i of order 2
    for k in range(3, P + 1):
        lower = m  # lower[i] = M_{k-1}(f + k - 2 - i)
        m = []
        for i in range(k):
            t = f + (k - 1 - i)
            a = lower[i - 1] if i >= 1 else 0.0  # M_{k-1}(t)
            b = lower[i] if i < k - 1 else 0.0   # M_{k-1}(t - 1)
            m.append((t * a + (k - t) * b) / (k - 1))
    if P == 2:
        return torch.stack(m, 1), torch.stack([-torch.ones_like(f), torch.ones_like(f)], 1)
    d = [(lower[i - 1] if i >= 1 else 0.0) - (lower[i] if i < P - 1 else 0.0) for i in range(P)]
    return torch.stack(m, 1), torch.stack(d, 1)


def _moduli(K, P, dev):
    M = _spline(P, torch.zeros(1, dtype=torch.float64))[0][0]  # M_P(P - 1 - i)
    k = torch.arange(K, dtype=torch.float64, device=dev)
    s = sum(float(M[P - 1 - j]) * torch.cos(2 * math.pi * k * (j - P // 2) / K) for j in range(1, P))
    return 1.0 / s


class _Mesh:
    """The SPME sums of one system in FP64."""

    def __init__(self, case, x, q):
        self.K, self.P, L = _grid(case), case["order"], _box(case)
        self.L, self.x, self.q, self.dev = L, x, q, x.device
        self.iV, self.iL = _inverse_box(L)
        iL = torch.tensor(self.iL, dtype=torch.float64, device=self.dev)
        s = x @ iL
        u = (s - s.floor()) * torch.tensor(self.K, dtype=torch.float64, device=self.dev)
        c = u.floor()
        self.cell, self.frac = c.long(), u - c
        self.iLt = iL

    def _chunks(self):
        P, step = self.P, max(1, (8 << 20) // self.P ** 3)
        off = torch.arange(P, device=self.dev) + 1 - P // 2
        for a in range(0, self.x.shape[0], step):
            ix = [((self.cell[a:a + step, d, None] + off) % self.K[d]) for d in range(3)]
            w = [_spline(P, self.frac[a:a + step, d]) for d in range(3)]
            idx = (ix[0][:, :, None, None] * self.K[1] + ix[1][:, None, :, None]) * self.K[2] + ix[2][:, None, None, :]
            yield slice(a, a + step), idx, w

    def structure(self):
        """S on the stored half space (F(Q) over the spline moduli)."""
        Q = torch.zeros(self.K[0] * self.K[1] * self.K[2], dtype=torch.float64, device=self.dev)
        for sl, idx, w in self._chunks():
            v = torch.einsum("a,ai,aj,ak->aijk", self.q[sl], w[0][0], w[1][0], w[2][0])
            Q.index_add_(0, idx.reshape(-1), v.reshape(-1))
        S = torch.fft.rfftn(Q.reshape(self.K))
        iB = [_moduli(self.K[d], self.P, self.dev) for d in range(3)]
        self.iB = iB[0][:, None, None] * iB[1][:, None] * iB[2][:S.shape[2]]
        return S * self.iB

    def solve(self, beta, max_m):
        """E, virial (xx, yy, zz, yx, zx, zy), dE/dx, phi."""
        S = self.structure()
        K, nz, iL = self.K, S.shape[2], self.iL
        rows = np.array([[self.L[0], 0, 0], [self.L[3], self.L[1], 0], [self.L[4], self.L[5], self.L[2]]])
        reach = [int(max_m * np.linalg.norm(rows[d])) + 1 for d in range(3)]
        shifts = [range(-((reach[d] + K[d] - 1) // K[d]), reach[d] // K[d] + 1) for d in range(3)]
        half = torch.full((nz,), 2.0, dtype=torch.float64, device=self.dev)  # modes stored once for +m and -m
        half[0] = 1.0
        if K[2] % 2 == 0:
            half[-1] = 1.0
        s2 = (S.real ** 2 + S.imag ** 2) * half
        A = torch.zeros(S.shape, dtype=torch.float64, device=self.dev)
        W = torch.zeros(6, dtype=torch.float64, device=self.dev)
        n = [torch.arange(k, dtype=torch.float64, device=self.dev) for k in (K[0], K[1], nz)]
        fac = -(math.pi / beta) ** 2
        for si in shifts[0]:
            i = (n[0] + si * K[0])[:, None, None]
            for sj in shifts[1]:
                j = (n[1] + sj * K[1])[:, None]
                for sk in shifts[2]:
                    k = n[2] + sk * K[2]
                    m = (i * iL[0][0], i * iL[1][0] + j * iL[1][1], i * iL[2][0] + j * iL[2][1] + k * iL[2][2])
                    m2 = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
                    ok = (m2 < max_m ** 2) & (m2 > 1e-10)
                    if not bool(ok.any()):
                        continue
                    f = torch.where(ok, torch.exp(m2 * fac) / (math.pi * m2), torch.zeros_like(m2))
                    A += f
                    t = torch.where(ok, (fac - 1.0 / m2) * f, torch.zeros_like(m2)) * s2
                    for c, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (1, 0), (2, 0), (2, 1))):
                        W[c] += (t * m[a] * m[b]).sum()
        e = 0.5 * (A * s2).sum()
        vir = W.clone()
        vir[:3] += e
        V = torch.fft.irfftn(S * self.iB * A, s=K, norm="forward").reshape(-1)
        phi = torch.empty_like(self.q)
        dx = torch.empty_like(self.x)
        kk = torch.tensor(K, dtype=torch.float64, device=self.dev)
        for sl, idx, w in self._chunks():
            v = V[idx]
            z0, z1 = torch.einsum("aijk,ak->aij", v, w[2][0]), torch.einsum("aijk,ak->aij", v, w[2][1])
            y00, y10 = torch.einsum("aij,aj->ai", z0, w[1][0]), torch.einsum("aij,aj->ai", z0, w[1][1])
            y01 = torch.einsum("aij,aj->ai", z1, w[1][0])
            phi[sl] = (y00 * w[0][0]).sum(1) * self.iV
            g = torch.stack([(y00 * w[0][1]).sum(1), (y10 * w[0][0]).sum(1), (y01 * w[0][0]).sum(1)], 1)
            dx[sl] = (g * kk * (self.q[sl, None] * self.iV)) @ self.iLt.T
        return e * self.iV, vir * self.iV ** 2, dx, phi

    def box_gradient(self, vir, dx):
        """dE/dL at fixed positions, in the order of L."""
        Pi = torch.stack([vir[[0, 3, 4]], vir[[3, 1, 5]], vir[[4, 5, 2]]])
        D = -(self.iLt.T @ Pi) / self.iV - (self.x @ self.iLt).T @ dx
        return torch.stack([D[0, 0], D[1, 1], D[2, 2], D[1, 0], D[2, 0], D[2, 1]])


def _mesh_solve(case, x, q):
    m = _Mesh(case, x, q)
    return m, m.solve(case["beta"], MAX_M_FACTOR * case["beta"])


def _real_space(case, x, q):
    """The erfc pair sum within rcut (minimum image), by cells at least rcut wide."""
    L, eta, rc = _box(case), case["beta"], case["rcut"]
    iV, iLr = _inverse_box(L)
    iL = torch.tensor(iLr, dtype=torch.float64, device=x.device)
    rows = _rows(L, x)
    n = x.shape[0]
    width = 1.0 / np.linalg.norm(np.array(iLr), axis=0)
    nb = [int(w / rc) for w in width]
    nb = [b if b >= 3 else 1 for b in nb]
    s = x @ iL
    s = s - s.floor()
    cell = torch.stack([(s[:, d] * nb[d]).long().clamp(max=nb[d] - 1) for d in range(3)], 1)
    key = (cell[:, 0] * nb[1] + cell[:, 1]) * nb[2] + cell[:, 2]
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=nb[0] * nb[1] * nb[2])
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    slot = torch.arange(n, device=x.device) - start[key[order]]
    table = torch.full((len(count), cap), n, dtype=torch.long, device=x.device)
    table[key[order], slot] = order
    sp = torch.cat([s, torch.zeros((1, 3), dtype=s.dtype, device=s.device)])
    qp = torch.cat([q, torch.zeros(1, dtype=q.dtype, device=q.device)])
    ids = torch.arange(len(count), device=x.device)
    c3 = torch.stack([ids // (nb[1] * nb[2]), ids // nb[2] % nb[1], ids % nb[2]], 1)
    near = [(-1, 0, 1) if b >= 3 else (0,) for b in nb]
    dx = torch.zeros((n + 1, 3), dtype=x.dtype, device=x.device)
    E, W = torch.zeros((), dtype=x.dtype, device=x.device), torch.zeros((3, 3), dtype=x.dtype, device=x.device)
    step = max(1, (16 << 20) // (cap * cap))
    for a in range(0, len(ids), step):
        mine = table[a:a + step]
        for d0 in near[0]:
            for d1 in near[1]:
                for d2 in near[2]:
                    o = [(c3[a:a + step, d] + v) % nb[d] for d, v in enumerate((d0, d1, d2))]
                    other = table[(o[0] * nb[1] + o[1]) * nb[2] + o[2]]
                    ds = sp[mine][:, :, None] - sp[other][:, None, :]
                    r = (ds - ds.round()) @ rows
                    r2 = (r * r).sum(-1)
                    ok = (r2 < rc * rc) & (r2 > 0) & (mine < n)[:, :, None] & (other < n)[:, None, :]
                    r2 = torch.where(ok, r2, torch.ones_like(r2))
                    d = r2.sqrt()
                    qq = qp[mine][:, :, None] * qp[other][:, None, :] * ok
                    phi = torch.special.erfc(eta * d) / d
                    E += 0.5 * (qq * phi).sum()
                    t = -qq * (2 * eta / math.sqrt(math.pi) * torch.exp(-(eta * d) ** 2) + phi) / r2
                    tr = t[..., None] * r
                    dx.index_add_(0, mine.reshape(-1), tr.sum(2).reshape(-1, 3))
                    W += 0.5 * torch.einsum("abci,abcj->ij", tr, r)
    q1, q2 = q.sum(), (q * q).sum()
    net = -math.pi * q1 * q1 * iV / (2 * eta * eta)
    out = torch.stack([E, -eta / math.sqrt(math.pi) * q2, net, *(-iV * W[a, b] for a, b in
                       ((0, 0), (1, 1), (2, 2), (1, 0), (2, 0), (2, 1))), net * iV])
    return out, dx[:n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        _, (E, vir, dx, phi) = _mesh_solve(case, *_inputs(case, seed))
        return torch.cat([E[None], vir]), dx, phi
    if kind == "real":
        return _real_space(case, *_inputs(case, seed))
    if kind == "batch":
        systems = _batch_systems(case)
        got = []
        for c, (x, q) in zip(systems, _many(systems, seed)):
            m, (E, vir, dx, phi) = _mesh_solve(c, x, q)
            got.append((E, dx, phi, m.box_gradient(vir, dx)))
        E, dx, phi, dL = zip(*got)
        return torch.stack(E), torch.cat(dx), torch.cat(phi), torch.stack(dL).cpu()
    if kind == "host":
        _, (E, vir, dx, phi) = _mesh_solve(case, *_inputs(case, seed))
        return float(E), vir.cpu().numpy(), dx.cpu().numpy(), phi.cpu().numpy()
    if kind == "frames":
        S2 = sum(_Mesh(case, x, q).structure().abs() ** 2 for x, q in _frames(case, seed))
        return S2.cpu().numpy(), case["frames"]
    systems = _serve_systems(case)
    out = []
    for c, (x, q) in zip(systems, _many(systems, seed)):
        _, (E, vir, dx, phi) = _mesh_solve(c, x, q)
        out.append(torch.cat([E[None], vir, dx.reshape(-1), phi]).cpu().numpy())
    return out
