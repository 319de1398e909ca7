"""The work that a user of this framework has it do, as cases that can be timed and checked.

A case is one call sequence of a user's program: whole time steps of one run (`lcs_step`, or the Julia loop's
`lcs_timestep` + `lcs_evolve`), the statistics of an output step, an ensemble stepped as a batch, or a stream of
requests through the server.  Each pass ends with the state that the program reads back, in pinned host memory.

`exact` restates the same computation in FP64 with torch alone: the staggered 4th-order right-hand side, the
red-black HSMAC sweeps in their order (time blocking, core and faces), both forcings and the particle push.
"""

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "lcs.jl_b200"))

from lcs_b200 import Batch, Engine, Server  # noqa: E402
from lcs_b200 import config as lcfg  # noqa: E402

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # a slice of 4 steps of the smallest served run: latency and launches
        dict(name="slice32_fp32", kind="step", nx=32, ny=32, nz=32, precision="fp32-mixed", forcing="linear-power",
             nu=0.02, particles=10000, species=1, steps=4, via="step", overlap=True, itrmax=300),
        # a small FP64 run driven by the Julia loop, a timestep! and an evolve! call a step
        dict(name="loop48_fp64", kind="step", nx=48, ny=48, nz=48, precision="fp64", forcing="rc-energy", nu=0.02,
             particles=20000, species=2, steps=2, via="evolve", overlap=True, itrmax=300),
        # a box with another size along each axis, none of them a multiple of a tile, without the overlap variant
        dict(name="ragged_fp64", kind="step", nx=70, ny=34, nz=96, precision="fp64", forcing="linear-power", nu=0.02,
             particles=3001, species=1, steps=2, via="step", overlap=False, itrmax=120),
        # the largest member of the ensembles, alone
        dict(name="step96_fp32", kind="step", nx=96, ny=96, nz=96, precision="fp32-mixed", forcing="linear-power",
             nu=0.02, particles=100000, species=1, steps=1, via="step", overlap=True, itrmax=300),
        # the plain FP64 workload of the benchmark's smallest size
        dict(name="lp128_fp64", kind="step", nx=128, ny=128, nz=128, precision="fp64", forcing="linear-power", nu=0.01,
             particles=65536, species=1, steps=1, via="step", overlap=True, itrmax=300),
        # the largest grid of the served stream with its largest particle count
        dict(name="step192_fp32", kind="step", nx=192, ny=192, nz=192, precision="fp32-mixed", forcing="linear-power",
             nu=0.01, particles=1000000, species=1, steps=1, via="step", overlap=True, itrmax=300),
        # the rc-energy workload: 256^3, 16-cell box filter, 2^20 particles in 2 species
        dict(name="rc256_fp64", kind="step", nx=256, ny=256, nz=256, precision="fp64", forcing="rc-energy", nu=0.005,
             particles=2 ** 20, species=2, steps=1, via="step", overlap=True, itrmax=300),
        # the headline workload in both precision forms: 512^3, 2^24 particles in 3 species
        dict(name="lp512_fp32", kind="step", nx=512, ny=512, nz=512, precision="fp32-mixed", forcing="linear-power",
             nu=0.0025, particles=2 ** 24, species=3, steps=1, via="step", overlap=True, itrmax=300),
        dict(name="lp512_fp64", kind="step", nx=512, ny=512, nz=512, precision="fp64", forcing="linear-power",
             nu=0.0025, particles=2 ** 24, species=3, steps=1, via="step", overlap=True, itrmax=300),
        # the statistics of an output step: Flows.stat and Particles.stat with the production settings
        dict(name="stat256_fp64", kind="stat", nx=256, ny=256, nz=256, precision="fp64", particles=2 ** 20, species=1),
        # an ensemble of uneven members stepped together
        dict(name="batch12_fp32", kind="batch", sizes="32,32,32,32,48,48,48,48,64,64,96,96", particles=20000, steps=1,
             itrmax=300),
        # a burst of requests of differing size through the server
        dict(name="serve6_fp32", kind="serve", sizes="32,64,48,96,32,64", particles=20000, steps=2, itrmax=300),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["stat", "batch", "serve"])
    precision = rng.choice(["fp64", "fp32-mixed"])
    if kind == "step":
        forcing = rng.choice(["linear-power", "linear-power", "rc-energy", "no"])
        n = _log_int(rng, 32, 320)
        # every axis of its own size in half of the draws; rc-energy grids hold a whole number of coarse cells
        q = 8 if forcing == "rc-energy" else 2
        dims = [max(q * 2, q * round(n * (rng.uniform(0.5, 1.4) if rng.random() < 0.5 else 1.0) / q)) for _ in range(3)]
        if rng.random() < 0.5:
            dims = [dims[0]] * 3
        return dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2], precision=precision, forcing=forcing,
                    nu=round(rng.uniform(0.005, 0.05), 4), particles=_log_int(rng, 3000, 1000000),
                    species=rng.choice([1, 1, 2, 3]), steps=1, via=rng.choice(["step", "step", "evolve"]),
                    overlap=rng.random() < 0.8, itrmax=rng.choice([60, 120, 300, 300, 301]))
    if kind == "stat":
        n = 4 * rng.randint(12, 64)
        return dict(kind=kind, nx=n, ny=n, nz=n, precision=precision, particles=_log_int(rng, 20000, 1000000), species=1)
    sizes = [rng.choice([32, 48, 64, 96]) for _ in range(rng.randint(3, 8))]
    return dict(kind=kind, sizes=",".join(map(str, sizes)), particles=_log_int(rng, 8000, 100000),
                steps=rng.randint(1, 2), itrmax=rng.choice([120, 300]))


# ------------------------------------------------------------------ inputs
def _run_config(case, n=None):
    """The reference-format config of a single run (case) or of one member of n^3."""
    dims = [n] * 3 if n else [case["nx"], case["ny"], case["nz"]]
    species = case.get("species", 1)
    total = case["particles"]
    counts = [total // species + (1 if s < total % species else 0) for s in range(species)]
    kind = case.get("forcing", "linear-power")
    forcing = {"no": {"kind": "no"}, "linear-power": {"kind": "linear-power", "params": {"power": 0.5}},
               "rc-energy": {"kind": "rc-energy", "params": {"kmin": 1, "kmax": 2, "energy": 0.649,
                                                             "coarse_size": _coarse(dims)}}}[kind]
    d = lcfg.workload(max(dims), case.get("nu", 0.02), forcing, [0.02 * 10 ** (s % 3) for s in range(species)], counts,
                      precision=case.get("precision", "fp32-mixed"), itrmax=case.get("itrmax", 300))
    d["grid"]["dims"] = dims
    d["flow"]["couple"]["params"]["overlap"] = bool(case.get("overlap", True))
    return lcfg.from_dict(d)


def _coarse(dims):
    """Coarse grid of the rc-energy box filter: 16-cell boxes at 256, 4-cell boxes or more below."""
    g = math.gcd(math.gcd(dims[0], dims[1]), dims[2])
    return max((c for c in range(4, 17) if g % c == 0), default=1)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _flow(dims, seed):
    """Random-phase solenoidal field, E(k) ~ k^4 exp(-2 (k/4)^2), u_rms = 1, at the staggered points; [k, j, i]."""
    dev = _device()
    nx, ny, nz = dims
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    ks = [torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev) for n in dims]
    k = [ks[0][None, None, :], ks[1][None, :, None], ks[2][:, None, None]]
    kk = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    amp = kk.sqrt() * torch.exp(-kk / 16.0)
    kk[0, 0, 0] = 1.0
    a = [torch.complex(torch.randn(nz, ny, nx, generator=gen, device=dev, dtype=torch.float64),
                       torch.randn(nz, ny, nx, generator=gen, device=dev, dtype=torch.float64)) for _ in range(3)]
    dot = (k[0] * a[0] + k[1] * a[1] + k[2] * a[2]) / kk
    out = []
    for c in range(3):
        f = (a[c] - k[c] * dot) * amp
        a[c] = None
        for ax in range(3):
            shift = TWO_PI / dims[ax] * (1.0 if ax == c else 0.5)
            f = f * torch.exp(1j * k[ax] * shift)
        out.append(torch.fft.ifftn(f).real.contiguous())
    del dot, amp, kk
    rms = math.sqrt(sum(float((f * f).mean()) for f in out) / 3.0)
    return [f / rms for f in out]


def _particles(count, seed):
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    return [torch.rand(count, generator=gen, device=dev, dtype=torch.float64) * TWO_PI for _ in range(3)]


def _inputs(rc, seed):
    dims = rc.dims
    return _flow(dims, 1000003 * seed + 1), [_particles(s.nvalid, 1000003 * seed + 17 + q)
                                             for q, s in enumerate(rc.species)]


def _pinned(*shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def _to_host(t):
    h = _pinned(*t.shape)
    h.copy_(t)
    return h.numpy()


def _load(e, rc, seed):
    flow, parts = _inputs(rc, seed)
    host = [_to_host(f) for f in flow]
    e.upload_flow(*host, np.zeros(host[0].shape))
    for s, xyz in enumerate(parts):
        x, y, z = (_to_host(a) for a in xyz)
        zero = np.zeros(x.shape)
        e.upload_particles(s, np.full(x.shape, rc.species[s].diam), x, y, z, zero, zero, zero,
                           ids=np.arange(1, x.size + 1))
        e.init_particle_velocity(s)


def _buffers(rc):
    nx, ny, nz = rc.dims
    return {"flow": _pinned(4, nz, ny, nx).numpy(), "parts": [_pinned(6, s.nvalid).numpy() for s in rc.species]}


def _download(e, buf):
    """The run's state into its pinned buffers: U, V, W, P and per species x, y, z, u, v, w."""
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    e._check(e.lib.lcs_download_flow(e.handle, *(p(f) for f in buf["flow"])))
    for s, b in enumerate(buf["parts"]):
        e._check(e.lib.lcs_download_particles(e.handle, s, None, None, *(p(a) for a in b)))
    return {"U": buf["flow"][0], "V": buf["flow"][1], "W": buf["flow"][2], "P": buf["flow"][3],
            "x": [b[:3] for b in buf["parts"]], "u": [b[3:] for b in buf["parts"]]}


def _counts(logs):
    return np.array([[lg[c][f] for c in ("couple1", "couple2") for f in ("itr", "sweeps")] for lg in logs], np.int64)


# ------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "stat"):
        rc = _run_config(case)
        e = Engine(rc.abi)
        _load(e, rc, seed)
        return dict(case=case, e=e, rc=rc, buf=_buffers(rc) if kind == "step" else None)
    sizes = [int(n) for n in case["sizes"].split(",")]
    rcs = [_run_config(case, n) for n in sizes]
    if kind == "batch":
        b = Batch([rc.abi for rc in rcs])
        for q, (rc, e) in enumerate(zip(rcs, b.members)):
            _load(e, rc, seed + 100 * q)
        return dict(case=case, batch=b, rcs=rcs, bufs=[_buffers(rc) for rc in rcs])
    reqs = []
    for q, rc in enumerate(rcs):
        flow, parts = _inputs(rc, seed + 100 * q)
        sp = []
        for s, xyz in enumerate(parts):
            x, y, z = (a.cpu().numpy() for a in xyz)
            zero = np.zeros_like(x)
            sp.append(dict(diam=np.full(x.shape, rc.species[s].diam), x=x, y=y, z=z, u=zero, v=zero, w=zero))
        fl = [f.cpu().numpy() for f in flow]
        reqs.append((rc, fl + [np.zeros(fl[0].shape)], sp))
    return dict(case=case, server=Server(max_active=8, steps_per_slice=4), reqs=reqs)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        e = state["e"]
        if case["via"] == "step":
            logs = e.step(case["steps"])
        else:
            logs = [e.evolve(e.timestep()) for _ in range(case["steps"])]
        return dict(_download(e, state["buf"]), sweeps=_counts(logs))
    if kind == "stat":
        e = state["e"]
        f = e.flow_stat()
        p = e.particles_stat(0, f["tau_eta"])
        return dict(flow=np.array([f[k] for k in sorted(f)]),
                    summary=np.array([[p[a][b] for b in ("mean", "max", "min")] for a in "xyzuvw"]),
                    taup=p["taup"], St=p["St"], gr=p["rdf"]["gr"], npairs=p["rdf"]["npairs"],
                    contacts=int(p["rdf"]["npairs_contact"]), Enp=p["spectrum"]["Enp"])
    if kind == "batch":
        logs = state["batch"].step(case["steps"])
        out = []
        for e, b in zip(state["batch"].members, state["bufs"]):
            d = _download(e, b)
            out.append(dict(vel=b["flow"][:3], P=d["P"], x=d["x"][0], u=d["u"][0]))
        return {"members": out, "sweeps": np.stack([_counts(lg) for lg in logs])}
    srv = state["server"]
    tickets = [srv.submit(rc.abi, *flow, species=sp, nsteps=case["steps"]) for rc, flow, sp in state["reqs"]]
    srv.drain(120.0)
    out = []
    for t in tickets:
        r = srv.result(t)
        srv.release(t)
        out.append(dict(vel=np.stack(r["flow"][:3]), P=r["flow"][3],
                        x=np.stack([r["particles"][0][k] for k in "xyz"]),
                        u=np.stack([r["particles"][0][k] for k in "uvw"])))
    return out


def work(case):
    """Bytes: the state read once and written once a call, and its FP64 copy to the host.  Flops: what a step
    cannot do without: 17 a cell and relaxation sweep, 460 a cell and right-hand side, 350 a particle push."""
    if case["kind"] == "stat":
        cells, parts = case["nx"] * case["ny"] * case["nz"], case["particles"]
        b = 8 if case["precision"] == "fp64" else 4
        # 3 fields; 8 properties; 17 shells of up to 128 in 64 directions, a sine and a cosine each
        return {"bytes": 3 * b * cells + 8 * 8 * parts, "flops": 80.0 * cells + parts * 14 * 64 * 45.0}
    if case["kind"] == "step":
        cells, runs = case["nx"] * case["ny"] * case["nz"], 1
    else:
        sizes = [int(n) for n in case["sizes"].split(",")]
        cells, runs = sum(n ** 3 for n in sizes), len(sizes)
    b = 8 if case.get("precision") == "fp64" else 4
    steps, parts = case["steps"], case["particles"] * runs
    return {"bytes": cells * (8 * b + 32) + parts * (7 * 8 + 6 * 8 + 48),
            "flops": steps * (cells * (2 * case["itrmax"] * 17.0 + 2 * 460.0) + parts * 2 * 350.0)}


# ------------------------------------------------- the same in FP64 with torch
def _o4(a, b, c, d):
    return (9.0 * (b + c) - a - d) / 16.0


class _Exact:
    def __init__(self, rc, flow, parts):
        c = rc.abi
        self.rc, self.c = rc, c
        self.n = rc.dims
        self.dx = [TWO_PI / n for n in rc.dims]
        self.di = [1.0 / d for d in self.dx]
        self.Re = c.U0 * c.L0 / c.NU
        self.U = list(flow)
        self.P = torch.zeros_like(flow[0])
        self.parts = []
        nx, ny, nz = self.n
        ix = [torch.arange(-2, n + 4, device=flow[0].device) for n in self.n]
        par = (ix[2][:, None, None] + ix[1][None, :, None] + ix[0][None, None, :]) % 2
        self.mask = [(par == q).double() for q in (0, 1)]
        for s, (x, y, z) in enumerate(parts):
            xs = torch.stack([x, y, z])
            self.parts.append(dict(x=xs, u=self._fluid(self.U, xs)))
        self.counts = []

    @staticmethod
    def _sh(a, axis, s):  # a at index + s along axis (0: x, 1: y, 2: z), periodic
        return torch.roll(a, -s, 2 - axis)

    # trilinear interpolation of the staggered components
    def _fluid(self, U, x):
        out = []
        for a in range(3):
            idx, r = [], []
            for b in range(3):
                q = x[b] / self.dx[b] + (0.0 if a == b else 0.5)
                f = torch.floor(q)
                idx.append(f.long())
                r.append(q - f)
            n = self.n
            acc = 0.0
            for di in (0, 1):
                for dj in (0, 1):
                    for dk in (0, 1):
                        w = ((r[0] if di else 1 - r[0]) * (r[1] if dj else 1 - r[1]) * (r[2] if dk else 1 - r[2]))
                        i, j, k = ((idx[b] + d - 1) % n[b] for b, d in ((0, di), (1, dj), (2, dk)))
                        acc = acc + w * U[a].reshape(-1)[(k * n[1] + j) * n[0] + i]
            out.append(acc)
        return torch.stack(out)

    def dt(self):
        c, d = self.c, self.c.dtmax
        for a in range(3):
            u = self.U[a]
            m = float(_o4(self._sh(u, a, -2), self._sh(u, a, -1), u, self._sh(u, a, 1)).abs().max())
            d = min(d, c.cfl * self.dx[a] / (m + 1e-10))
        d = min(d, 0.5 * (self.dx[0] / 2) ** 2 * self.Re)
        for s, sp in enumerate(self.rc.species):
            d = min(d, 0.5 * c.species[s].density_ratio * self.Re * sp.diam ** 2 / 18.0)
        return d

    def rhs(self, U, comp):
        sh, A, di = self._sh, U[comp], self.di
        out = 0.0
        for a in range(3):
            out = out + di[a] ** 2 / self.Re / 12.0 * (16.0 * (sh(A, a, -1) + sh(A, a, 1)) - 30.0 * A
                                                       - sh(A, a, -2) - sh(A, a, 2))
        out -= di[comp] * (sh(self.P, comp, 1) - self.P)
        for a in range(3):
            q = U[a]
            adv = _o4(sh(q, comp, -1), q, sh(q, comp, 1), sh(q, comp, 2))
            j1 = adv * (0.5 * (A + sh(A, a, 1)))
            j3 = adv * (0.5 * (sh(A, a, -1) + sh(A, a, 2)))
            out -= di[a] * (1.125 * (j1 - sh(j1, a, -1)) - (sh(j3, a, 1) - sh(j3, a, -2)) / 24.0)
        return out

    def push(self, stage, U, dt):
        for s, p in enumerate(self.parts):
            c = self.c.species[s]
            here, other = ("x", "x2") if stage == 1 else ("x2", "x")
            off = TWO_PI * ((p[here] < 0).double() - (p[here] >= TWO_PI).double())
            p[here] = p[here] + off
            if stage == 2:
                p[other] = p[other] + off
            taup = c.density_ratio * self.Re * self.rc.species[s].diam ** 2 / 18.0
            f = (self._fluid(U, p[here]) - p["u" if stage == 1 else "u2"]) / taup
            f[0] -= c.gravity
            x, u = p["x"] + dt * p["u"], p["u"] + dt * f
            if stage == 1:
                p["x2"], p["u2"] = x, u
            else:
                p["x"], p["u"] = x, u

    def force(self, dt):
        kind = self.c.forcing
        U, sh = self.U, self._sh
        if kind == 1:  # constant-power linear forcing
            mean = [float(u.mean()) for u in U]
            e = 0.0
            for a in range(3):
                cc = 0.5 * (sh(U[a], a, -1) + U[a])
                e += 0.5 * (float((cc * cc).mean()) - mean[a] ** 2)
            A = self.c.power / (2.0 * e)
            self.U = [u + A * (u - m) * dt for u, m in zip(U, mean)]
        elif kind == 2:  # shell energies restored on the box-filtered field
            cs, n = self.c.coarse_size, self.n
            ph = (n[0] // cs) / 2.0
            dev = U[0].device
            coarse = [u.reshape(cs, n[2] // cs, cs, n[1] // cs, cs, n[0] // cs).mean(dim=(1, 3, 5)) for u in U]
            hat = [torch.fft.fftn(q) / cs ** 3 for q in coarse]
            shells = {}
            K = self.c.kmax
            for kz in range(-K, K + 1):
                for ky in range(-K, K + 1):
                    for kx in range(0, K + 1):
                        r2 = kx * kx + ky * ky + kz * kz
                        for k0 in range(self.c.kmin, K + 1):
                            if (k0 - 0.5) ** 2 <= r2 < (k0 + 0.5) ** 2:
                                shells.setdefault(k0, []).append((kx, ky, kz))
            count = lambda k: sum(1 if v[0] == 0 else 2 for v in shells[k])  # noqa: E731
            src = [torch.zeros_like(u) for u in U]
            x = [torch.arange(1, m + 1, device=dev, dtype=torch.float64) for m in n]
            for k0, ks in shells.items():
                en = sum((1.0 if k[0] == 0 else 2.0) * float(sum(abs(h[k[2], k[1], k[0]]) ** 2 for h in hat))
                         for k in ks) / 2.0
                en0 = (self.c.energy * k0 ** (-5.0 / 3.0) * (1.5 ** 3 - 0.5 ** 3)
                       / ((k0 + 0.5) ** 3 - (k0 - 0.5) ** 3) * count(k0) / count(self.c.kmin))
                r = math.sqrt(en0 / max(en, 1e-8)) - 1.0
                for k in ks:
                    if k[0] == 0 and (k[1] < 0 or (k[1] == 0 and k[2] < 0)):
                        continue  # the conjugate of a vector that is counted
                    e = [torch.exp(2j * math.pi * k[a] * (x[a] - ph) / n[a]) for a in range(3)]
                    w = e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
                    for a in range(3):
                        src[a] += 2.0 * r * (hat[a][k[2], k[1], k[0]] * w).real
            self.U = [u + q for u, q in zip(U, src)]

    # red-black HSMAC, in the order of the time-blocked loop
    def couple(self, U, dt):
        c, n = self.c, self.n
        nz, ny, nx = n[2], n[1], n[0]
        di, dti = self.di, 1.0 / dt
        dl = 0.5 / sum(d * d for d in di)
        H = [torch.zeros(nz + 6, ny + 6, nx + 6, device=U[0].device, dtype=torch.float64) for _ in range(4)]
        core = (slice(3, nz + 3), slice(3, ny + 3), slice(3, nx + 3))
        for f, q in zip(H, list(U) + [self.P]):
            f[core] = q

        def fill():
            for f in H[:3]:
                for ax, m in ((2, nx), (1, ny), (0, nz)):
                    f.narrow(ax, 0, 3).copy_(f.narrow(ax, m, 3).clone())
                    f.narrow(ax, m + 3, 3).copy_(f.narrow(ax, 3, 3).clone())

        def box(lo, hi, s=(0, 0, 0)):  # logical bounds x, y, z
            return tuple(slice(lo[a] + 2 + s[a], hi[a] + 3 + s[a]) for a in (2, 1, 0))

        def phase(lo, hi, color):
            if any(lo[a] > hi[a] for a in range(3)):
                return 0.0
            here = box(lo, hi)
            d = None
            for a in range(3):
                back = box(lo, hi, tuple(-1 if b == a else 0 for b in range(3)))
                if d is None:
                    d = (H[a][here] - H[a][back]).mul_(di[a])
                else:
                    d.add_(H[a][here], alpha=di[a]).add_(H[a][back], alpha=-di[a])
            d.mul_(self.mask[color][here])
            rlo, rhi = [max(1, q) for q in lo], [min(n[a] + 1, hi[a]) for a in range(3)]
            own = d[tuple(slice(rlo[a] - lo[a], rhi[a] - lo[a] + 1) for a in (2, 1, 0))]
            s = (own * own).sum() if all(rlo[a] <= rhi[a] for a in range(3)) else 0.0
            d.mul_(-c.omega * dl)
            H[3][here].add_(d, alpha=dti)
            for a in range(3):
                back = box(lo, hi, tuple(-1 if b == a else 0 for b in range(3)))
                H[a][here].add_(d, alpha=di[a])
                H[a][back].add_(d, alpha=-di[a])
            return s

        def sweep(lo, hi):
            return phase(lo, hi, 0) + phase(lo, hi, 1)

        def all3(v, w):
            return [v] * 3, [m + w for m in n]

        itr = sweeps = 0
        count = float((nx + 1) * (ny + 1) * (nz + 1))
        done = False
        while itr < c.itrmax and not done:
            fill()
            for b in range(3):
                lo, hi = all3(b - 1, 3 - b)
                if b == 0 and c.overlap:
                    clo, chi = all3(2, 0)
                    s = sweep(clo, chi)
                    for a in (2, 1, 0):  # z, y, x faces; an axis done before keeps its core range
                        for side in (0, 1):
                            flo, fhi = list(lo), list(hi)
                            for q in range(a + 1, 3):
                                flo[q], fhi[q] = clo[q], chi[q]
                            if side == 0:
                                fhi[a] = clo[a] - 1
                            else:
                                flo[a] = chi[a] + 1
                            s = s + sweep(flo, fhi)
                else:
                    s = sweep(lo, hi)
                sweeps += 1
                if c.itrmin <= itr and math.sqrt(float(s) / count) * min(self.dx) < c.epsp:
                    done = True
                    break
                itr += 1
        self.counts.append((itr, sweeps))
        self.P = H[3][core].clone()
        return [f[core].clone() for f in H[:3]]

    def step(self):
        dt = self.dt()
        self.counts = []
        self.push(1, self.U, 0.5 * dt)
        U2 = [self.U[a] + self.rhs(self.U, a) * (0.5 * dt) for a in range(3)]
        U2 = self.couple(U2, 0.5 * dt)
        self.push(2, U2, dt)
        new = [self.rhs(U2, a).mul_(dt).add_(self.U[a]) for a in range(3)]
        self.U = new
        self.force(dt)
        self.U = self.couple(self.U, dt)

    def state(self):
        h = lambda t: t.cpu().numpy()  # noqa: E731
        return {"U": h(self.U[0]), "V": h(self.U[1]), "W": h(self.U[2]), "P": h(self.P),
                "x": [h(p["x"]) for p in self.parts], "u": [h(p["u"]) for p in self.parts]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        rc = _run_config(case)
        m = _Exact(rc, *_inputs(rc, seed))
        for _ in range(case["steps"]):
            m.step()
        return dict(m.state(), sweeps=None)
    if kind == "stat":
        return _exact_stat(case, seed)
    out = []
    for q, n in enumerate(int(s) for s in case["sizes"].split(",")):
        rc = _run_config(case, n)
        m = _Exact(rc, *_inputs(rc, seed + 100 * q))
        for _ in range(case["steps"]):
            m.step()
        st = m.state()
        out.append(dict(vel=np.stack([st["U"], st["V"], st["W"]]), P=st["P"], x=st["x"][0], u=st["u"][0]))
    return {"members": out, "sweeps": None} if kind == "batch" else out


def _exact_stat(case, seed):
    rc = _run_config(case)
    m = _Exact(rc, *_inputs(rc, seed))
    U, sh, di = m.U, m._sh, m.di
    N = U[0].numel()

    def d1(a, axis, base):  # 4th-order half-point derivative, offsets base .. base + 3
        a0, a1, a2, a3 = (sh(a, axis, base + q) for q in range(4))
        return di[axis] / 24.0 * (a0 - 27.0 * a1 + 27.0 * a2 - a3)

    dd = [d1(U[a], a, -2) for a in range(3)]
    s12 = 0.5 * (d1(U[0], 1, -2) + d1(sh(U[1], 1, -1), 0, -1))
    s13 = 0.5 * (d1(U[0], 2, -2) + d1(sh(U[2], 2, -1), 0, -1))
    s23 = 0.5 * (d1(sh(U[1], 1, -1), 2, -1) + d1(U[2], 1, -2))
    # the dissipation and the moments of du/dx as the flow statistics define them
    return _finish_stat(case, m, N, dd, s12, s13, s23)


def _finish_stat(case, m, N, dd, s12, s13, s23):
    U, Re = m.U, m.Re
    s2 = float((2.0 * (dd[0] ** 2 + dd[1] ** 2 + dd[2] ** 2 + 2.0 * (s12 ** 2 + s13 ** 2 + s23 ** 2))).mean())
    u2 = float((U[0] ** 2 + U[1] ** 2 + U[2] ** 2).mean())
    d2, d3, d4 = (float((dd[0] ** q).mean()) for q in (2, 3, 4))
    o = {}
    for q, a in enumerate("uvw"):
        o[a + "_mean"], o[a + "_max"], o[a + "_min"] = float(U[q].mean()), float(U[q].max()), float(U[q].min())
    o["urms"] = math.sqrt(u2 / 3.0)
    o["k"] = 0.5 * (u2 - o["u_mean"] ** 2 - o["v_mean"] ** 2 - o["w_mean"] ** 2)
    o["epsilon"] = s2 / Re
    o["tau_eta"] = math.sqrt(1.0 / o["epsilon"] / Re)
    o["l_mu"] = math.sqrt(15.0 * o["urms"] ** 2 / o["epsilon"] / Re)
    l_eta = (1.0 / o["epsilon"] / Re ** 3) ** 0.25
    o["Re_lambda"] = o["l_mu"] * o["urms"] * Re
    o["k_eta"] = min(m.n) / 2.0 * l_eta
    o["skewness"] = -d3 / d2 ** 1.5
    o["flatness"] = d4 / d2 ** 2
    o["l_eta"], o["L"], o["C_epsilon"] = l_eta, 0.0, 0.0
    names = ["u_mean", "u_max", "u_min", "v_mean", "v_max", "v_min", "w_mean", "w_max", "w_min", "k", "epsilon",
             "tau_eta", "l_mu", "l_eta", "Re_lambda", "urms", "k_eta", "skewness", "flatness", "L", "C_epsilon"]
    p = m.parts[0]
    xu = torch.cat([p["x"], p["u"]])
    summary = np.array([[float(a.mean()), float(a.max()), float(a.min())] for a in xu])
    taup = m.c.species[0].density_ratio * Re * m.rc.species[0].diam ** 2 / 18.0
    return dict(flow=np.array([o[k] for k in sorted(names)]), summary=summary, taup=taup, St=taup / o["tau_eta"],
                gr=None, npairs=None, contacts=None, Enp=_exact_spectrum(p["x"]))


def _exact_spectrum(x, ns=64, max_wavenumber=128):
    """4 pi k^2 times the mean over the Fibonacci directions of |sum exp(i k.x)|^2 / N^2 - 1 / N, per shell."""
    shells = [k for k in (1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128) if k <= max_wavenumber]
    phi = math.pi * (3.0 - math.sqrt(5.0))
    N, out = x.shape[1], []
    for kk in shells:
        acc = 0.0
        for i in range(ns):
            y = 1.0 - i / (ns - 1) * 2.0
            r = math.sqrt(1.0 - y * y)
            ph = kk * math.cos(phi * i) * r * x[0] + kk * y * x[1] + kk * math.sin(phi * i) * r * x[2]
            acc += (float(ph.cos().sum()) ** 2 + float(ph.sin().sum()) ** 2) / float(N) ** 2 - 1.0 / N
        out.append(acc / ns * 4.0 * math.pi * kk * kk)
    return np.array(out)
