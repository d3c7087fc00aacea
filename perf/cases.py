"""Performance cases: the calls a user of this framework makes, over their real range.

A case is a dict of plain values.  ``listed()`` gives the named ones, ``draw``
others of the same ranges, ``prepare`` what a program has in hand before the
call (inputs from the seed, domain, sensors, transform plan, solver), ``run``
one pass through the public entry points, ``work`` the bytes and operations of
a pass and ``exact`` the same outputs in plain 64-bit torch where that is
affordable.

Kinds
  step       forward p0 -> sensor data and the gradient image of the misfit
             (the exact transpose), as a reconstruction loop calls them
  forward    the forward alone
  frame      the multiscale transform: analysis, synthesis and the Hermitian
             adjoint of the analysis
  select     the coefficients of an image and the threshold that picks beams
  reversal   time reversal of boundary data to an image
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

import beamax_b200 as bb
from beamax_b200.gb.gb_solvers import solve_hom_diag, solve_ODE_base
from beamax_b200.solvers.autograd import msgb_forward
from beamax_b200.utils.interp import make_c_function_from_grid

SPEED = 1500.0
DEVICE = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The reference's default use: host arrays, default FP64 precision, a small
        # grid with a line sensor (the smallest call: launches and latency).
        dict(name="step_64_host", kind="step", ndim=2, n=64, levels=2, thr=256, precision="fp64", medium="hom",
             sensors="row", stride=1, frozen=False, host=True),
        # The dense FP64 path (the accuracy reference, the default precision) on a
        # medium grid with sensors on all four sides.
        dict(name="step_256_fp64", kind="step", ndim=2, n=256, levels=3, thr=3000, precision="fp64", medium="hom",
             sensors="sides", stride=1, frozen=False, host=False),
        # The FP32 path on a small grid: an ordinary quick look.
        dict(name="step_128", kind="step", ndim=2, n=128, levels=3, thr=4096, precision="fp32", medium="hom",
             sensors="row", stride=1, frozen=False, host=False),
        # The 512 x 512 homogeneous benchmark workload.
        dict(name="step_512", kind="step", ndim=2, n=512, levels=4, thr=65536, precision="fp32", medium="hom",
             sensors="sides", stride=1, frozen=False, host=False),
        # One iteration of a gradient reconstruction: beam set frozen, one-sided
        # 512-point sensor.
        dict(name="iteration_512", kind="step", ndim=2, n=512, levels=4, thr=65536, precision="fp32", medium="hom",
             sensors="row", stride=1, frozen=True, host=False),
        # A circular array (the usual photoacoustic ring): sensors off the grid, no
        # straight runs.
        dict(name="ring_256", kind="forward", ndim=2, n=256, levels=3, thr=5000, precision="fp32", medium="hom",
             sensors="ring", stride=1, frozen=False, host=False),
        # Heterogeneous media.  Few beams (the chip is nearly idle during the ray
        # integration), FP64 throughout, and the 1024 x 1024 headline geometry.
        dict(name="het_128", kind="step", ndim=2, n=128, levels=3, thr=1000, precision="fp32", medium="het",
             sensors="sides", stride=1, frozen=False, host=False),
        dict(name="het_256_fp64", kind="forward", ndim=2, n=256, levels=3, thr=1500, precision="fp64", medium="het",
             sensors="sides", stride=2, frozen=False, host=False),
        dict(name="het_1024", kind="step", ndim=2, n=1024, levels=4, thr=100000, precision="fp32", medium="het",
             sensors="sides", stride=1, frozen=False, host=False),
        # 3D: planar detector on one face of a heterogeneous cube.
        dict(name="het3d_128", kind="step", ndim=3, n=128, levels=3, thr=16001, precision="fp32", medium="het",
             sensors="row", stride=1, frozen=False, host=False),
        # The transform by itself at the headline size, with the selection of beams.
        dict(name="select_1024", kind="select", ndim=2, n=1024, levels=4, thr=262144, strategy="top_n"),
        # Boundary data back to an image on every grid point.
        dict(name="reversal_256", kind="reversal", ndim=2, n=256, levels=2, thr=4000, medium="het"),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["hom64", "hom32", "hom32", "het32", "het32", "het64", "cube", "frame", "select", "reversal"])
    if kind == "hom64":
        n = rng.choice([64, 128, 256])
        return dict(kind=rng.choice(["step", "forward"]), ndim=2, n=n, levels=2 if n == 64 else 3,
                    thr=spread(101, 3000), precision="fp64", medium="hom", sensors=rng.choice(["row", "sides", "ring"]),
                    stride=rng.choice([1, 2, 3]), frozen=rng.random() < 0.3, host=rng.random() < 0.3)
    if kind == "hom32":
        n = rng.choice([128, 256, 512])
        sensors = rng.choice(["row", "sides", "ring"])
        top = 65536 if n == 512 else 16384
        return dict(kind="step", ndim=2, n=n, levels=4 if n == 512 else 3, thr=spread(301, top // 4 if sensors == "ring" else top),
                    precision="fp32", medium="hom", sensors=sensors, stride=rng.choice([1, 1, 2]),
                    frozen=rng.random() < 0.4, host=False)
    if kind == "het32":
        n = rng.choice([128, 256, 512, 1024])
        return dict(kind=rng.choice(["step", "step", "forward"]), ndim=2, n=n, levels=4 if n >= 512 else 3,
                    thr=spread(201, {128: 6000, 256: 20000, 512: 65536, 1024: 65536}[n]), precision="fp32", medium="het",
                    sensors=rng.choice(["row", "sides"]), stride=1, frozen=rng.random() < 0.3, host=False)
    if kind == "het64":
        n = rng.choice([64, 128, 256])
        return dict(kind="forward", ndim=2, n=n, levels=2 if n == 64 else 3, thr=spread(51, 1500), precision="fp64",
                    medium="het", sensors=rng.choice(["row", "sides"]), stride=rng.choice([1, 2, 4]), frozen=False,
                    host=False)
    if kind == "cube":
        n = rng.choice([64, 128])
        return dict(kind="step", ndim=3, n=n, levels=2 if n == 64 else 3, thr=spread(301, 16001), precision="fp32",
                    medium=rng.choice(["hom", "het"]), sensors="row", stride=rng.choice([1, 2]),
                    frozen=rng.random() < 0.3, host=False)
    if kind == "frame":
        ndim = rng.choice([2, 2, 3])
        n = rng.choice([64, 128, 256, 512, 1024]) if ndim == 2 else rng.choice([32, 64, 128])
        levels = {2: {64: 2, 128: 3, 256: 3}.get(n, 4), 3: {32: 1, 64: 2}.get(n, 3)}[ndim]
        return dict(kind="frame", ndim=ndim, n=n, levels=levels, noise=round(rng.uniform(0.0005, 0.05), 6))
    if kind == "select":
        n = rng.choice([128, 256, 512, 1024])
        strategy = rng.choice(["top_n", "top_n", "percentile"])
        thr = spread(255, n * n // 4) if strategy == "top_n" else round(rng.uniform(80.0, 99.0), 3)
        return dict(kind="select", ndim=2, n=n, levels={128: 3, 256: 3}.get(n, 4), thr=thr, strategy=strategy)
    n = rng.choice([64, 128, 256])
    return dict(kind="reversal", ndim=2, n=n, levels=2, thr=spread(101, 4000), medium=rng.choice(["hom", "het"]))


# ------------------------------------------------------------------ what a program holds
def _boxes(levels):
    return tuple(4 * 2 ** l for l in range(levels))


@functools.lru_cache(maxsize=8)
def _transform(N, levels, aspect):
    """A program builds the transform of its grid once and keeps it."""
    return bb.MSWPT(bb.DyadicDecomposition(levels, N, _boxes(levels), aspect), 2, "rectangular_mirror")


def _spacing(n):
    return 5e-5 if n > 512 else 1e-4


def _image(N, seed, noise=1e-3):
    """Wave packets over all scales, smooth blobs and a noise floor, max 1 (float64, on the device)."""
    gen = torch.Generator(DEVICE).manual_seed(1000003 * (seed % 1000003) + 17)
    rand = lambda *s: torch.rand(*s, generator=gen, device=DEVICE, dtype=torch.float64)
    randn = lambda *s: torch.randn(*s, generator=gen, device=DEVICE, dtype=torch.float64)
    d, low = len(N), min(N)
    axes = torch.meshgrid(*[torch.arange(m, device=DEVICE, dtype=torch.float64) for m in N], indexing="ij")
    out = noise * randn(*N)
    for i in range(48):
        centre = (0.1 + 0.8 * rand(d)) * torch.tensor(N, device=DEVICE, dtype=torch.float64)
        u = randn(d)
        u = u / u.norm()
        k = low * torch.exp2(-1.2 - 5.0 * rand(1))      # cycles over the shortest axis
        width = (0.25 + 0.75 * rand(1)) * low / (math.pi * 0.5 * k) + 1.5 if i % 6 else 0.04 * low * (0.5 + rand(1))
        r2 = sum((a - c) ** 2 for a, c in zip(axes, centre))
        ph = sum((a - c) * v for a, c, v in zip(axes, centre, u)) * (2 * math.pi * k / low if i % 6 else 0.0)
        out += randn(1) * torch.exp(-r2 / (2 * width ** 2)) * torch.cos(ph)
    return out / out.abs().max()


def _speed(N, dx, seed):
    """Smooth random sound speed, 8 % contrast in 2D and 5 % in 3D, correlation 0.04 N and 0.15 N; cubic B-spline."""
    gen = torch.Generator(DEVICE).manual_seed(7919 * (seed % 1000003) + 5)
    f = torch.fft.fftn(torch.randn(*N, generator=gen, device=DEVICE, dtype=torch.float64))
    corr = (0.04 if len(N) == 2 else 0.15) * N[0]
    for a, m in enumerate(N):
        k = torch.fft.fftfreq(m, device=DEVICE, dtype=torch.float64)
        shape = [1] * len(N)
        shape[a] = m
        f = f * torch.exp(-0.5 * (2 * math.pi * k * corr) ** 2).reshape(shape)
    g = torch.fft.ifftn(f).real
    g = (2.0 * (g - g.min()) / (g.max() - g.min()) - 1.0).cpu().numpy()
    return make_c_function_from_grid(SPEED * (1.0 + _contrast(len(N)) * g), dx, method="bspline3", boundary="clamp")


def _contrast(d):
    return 0.08 if d == 2 else 0.05


def _times(case):
    """The acquisition's time grid: one sample per CFL step (0.3) of the fastest
    sound speed until the slowest crosses the diagonal."""
    d, n = case["ndim"], case["n"]
    spread = _contrast(d) if case["medium"] == "het" else 0.0
    dt = 0.3 * _spacing(n) / (SPEED * (1.0 + spread))
    return np.arange(math.ceil(math.sqrt(d) * n / 0.3 * (1.0 + spread) / (1.0 - spread))) * dt


def _receivers(case, N, dx, dom):
    mask = np.zeros(N)
    if case["sensors"] == "ring":
        count = 2 * N[0]
        th = 2 * math.pi * np.arange(count) / count
        pos = 0.5 * N[0] * dx[0] + 0.47 * N[0] * dx[0] * np.stack([np.cos(th), np.sin(th)], -1)
        return bb.Sensor(dom, positions=pos)
    if case["sensors"] == "row":
        mask[(slice(None),) * (len(N) - 1) + (0,) if len(N) == 3 else (0, slice(None))] = 1
    else:
        mask[0, :] = mask[-1, :] = mask[:, 0] = mask[:, -1] = 1
    return bb.Sensor(dom, binary_mask=mask)


def _noise(shape, seed, dtype):
    gen = torch.Generator(DEVICE).manual_seed(104729 * (seed % 1000003) + 3)
    return torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float64).to(dtype)


def prepare(case, seed):
    d, n = case["ndim"], case["n"]
    N = (n,) * d
    dx = (_spacing(n),) * d
    kind = case["kind"]
    if kind == "frame":
        wpt = _transform(N, case["levels"], (1,) * d)
        return dict(case=case, wpt=wpt, x=_image(N, seed, case["noise"]))
    if kind == "select":
        dom = bb.Domain(N=N, dx=dx, periodic=(False,) * d, cfl=0.3, c=SPEED)
        solver = bb.MSGBSolver(case["thr"], case["strategy"], 128, "spatial", solve_hom_diag, "scan_real")
        return dict(case=case, wpt=_transform(N, case["levels"], (1,) * d), solver=solver, domain=dom, x=_image(N, seed))
    c = SPEED if case["medium"] == "hom" else _speed(N, dx, seed)
    dom = bb.Domain(N=N, dx=dx, periodic=(False,) * d, cfl=0.3, c=c)
    ts = _times(case)
    if kind == "reversal":
        Nd = (2 * n,) + N[1:]
        ddom = bb.Domain(N=Nd, dx=(float((ts[-1] - ts[0]) / (Nd[0] - 1)),) + dx[1:], periodic=(False,) * d, cfl=0.3, c=c)
        mask = np.zeros(N)
        mask[0, :] = 1
        solver = bb.MSGBSolver(case["thr"], "top_n", 128, "spatial", solve_ODE_base, "scan_real",
                               ode_config=bb.gb.gb_solvers.SolverConfig(max_steps=100000))
        return dict(case=case, solver=solver, domain=dom, ts=ts, ddom=ddom, dwpt=_transform(Nd, case["levels"], (2, 1)),
                    sources=bb.Sensor(dom, binary_mask=mask), points=bb.Sensor(dom, binary_mask=np.ones(N)),
                    x=_image(Nd, seed))
    ts = ts[::case["stride"]]
    wpt = _transform(N, case["levels"], (1,) * d)
    solver = bb.MSGBSolver(case["thr"], "top_n", 128, "spatial", solve_hom_diag if case["medium"] == "hom" else solve_ODE_base,
                           "scan_real", precision=case["precision"])
    sensors = _receivers(case, N, dx, dom)
    x = _image(N, seed)
    data = 0.05 * _noise((ts.size, sensors.positions.shape[0]), seed, torch.float64)
    selection = None
    if case["frozen"]:  # the beams were chosen once, from an earlier image
        selection = solver.select(x + 0.05 * _image(N, seed + 1), dom, wpt)
    if case["precision"] == "fp32":
        x, data = x.float(), data.float()
    if case["host"]:
        x, data = x.cpu().numpy(), data.cpu().numpy()
    return dict(case=case, solver=solver, domain=dom, sensors=sensors, ts=ts, wpt=wpt, x=x, data=data, selection=selection)


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "frame":
        wpt = state["wpt"]
        c = wpt.forward(state["x"])
        return {"coeffs": c, "image": wpt.inverse(c), "adjoint": wpt.adjoint(c, real_output=True)}
    if kind == "select":
        sel = state["solver"].select(state["x"], state["domain"], state["wpt"])
        return {"idx": sel.idx, "values": sel.values}
    if kind == "reversal":
        s = state
        return {"image": s["solver"].time_reversal(s["x"], s["domain"], s["points"], s["sources"], s["ts"], s["ddom"],
                                                   s["dwpt"])}
    solver, dom, sensors, ts, wpt = (state[k] for k in ("solver", "domain", "sensors", "ts", "wpt"))
    x, data, selection = state["x"], state["data"], state["selection"]
    if kind == "forward":
        if selection is not None:
            return {"data": solver.forward_frozen(x, dom, sensors, ts, wpt, selection)}
        return {"data": solver.forward(x, dom, sensors, ts, wpt)}
    if state["case"]["host"]:
        if selection is not None:
            y = solver.forward_frozen(x, dom, sensors, ts, wpt, selection)
            return {"data": y, "gradient": solver.adjoint(y - data, dom, sensors, ts, wpt, selection=selection)}
        y = solver.forward(x, dom, sensors, ts, wpt)
        return {"data": y, "gradient": solver.adjoint(y - data, dom, sensors, ts, wpt)}
    x = x.detach().requires_grad_()
    y = msgb_forward(x, solver, dom, sensors, ts, wpt, selection=selection)
    (g,) = torch.autograd.grad(y, x, grad_outputs=y.detach() - data)
    return {"data": y.detach(), "gradient": g}


# ------------------------------------------------------------------ cost of a pass
def _sizes(case):
    """Times and receivers of a propagation case."""
    d, n = case["ndim"], case["n"]
    nt = len(_times(case)[::case.get("stride", 1)])
    ns = {"row": n ** (d - 1), "sides": 4 * n - 4, "ring": 2 * n}[case.get("sensors", "row")]
    return nt, ns


def work(case):
    d, n, kind = case["ndim"], case["n"], case["kind"]
    total = n ** d
    fft = 5.0 * total * math.log2(total)
    frame = 2.0 ** d * total                 # redundancy 2 per axis
    if kind == "frame":
        return {"bytes": 8.0 * total + 16.0 * frame + 16.0 * total + 8.0 * total,
                "flops": 3 * (fft + 5.0 * frame * math.log2(max(2.0, frame / total)))}
    if kind == "select":
        keep = case["thr"] if case["strategy"] == "top_n" else 0.05 * frame
        return {"bytes": 8.0 * total + 24.0 * keep, "flops": fft + 5.0 * frame * 5 + 4.0 * frame}
    if kind == "reversal":
        nt = math.sqrt(2) * n / 0.3
        return {"bytes": 16.0 * total + 8.0 * total, "flops": 40.0 * case["thr"] * total + 3600.0 * case["thr"] * nt}
    nt, ns = _sizes(case)
    passes = 2.0 if kind == "step" else 1.0
    beams = 2.0 * case["thr"]
    # The FP32 path evaluates the triples within its cutoff, 16 e-folds: about 8 % of
    # all in 2D and 5 % in 3D (its own evaluation counter); the FP64 path all of them.
    share = 1.0 if case["precision"] == "fp64" else 0.08 if d == 2 else 0.05
    flops = passes * 36.0 * share * beams * nt * ns + passes * fft
    if case["medium"] == "het":
        flops += (3600.0 if d == 2 else 9700.0) * beams * nt
    size = 8.0 if case["precision"] == "fp64" else 4.0
    return {"bytes": size * (total + nt * ns) * passes, "flops": flops}


# ------------------------------------------------------------------ the same in plain 64-bit torch
class _Frame:
    """The multiscale transform, written out: overlapping Gaussian-windowed
    boxes on a dyadic lattice of the centred spectrum, one unitary FFT per box."""

    def __init__(self, N, levels, aspect):
        self.N, self.aspect, d = N, aspect, len(N)
        low, counts = min(N), _boxes(levels)
        self.levels = []
        inner = np.zeros(d)
        self.power = torch.zeros(*N, dtype=torch.float64, device=DEVICE)
        for l, count in enumerate(counts):
            length = low // (counts[-1] * 2 ** (levels - 1 - l))
            step = [length * a for a in aspect]
            per = [round(count * m / low / a) for m, a in zip(N, aspect)]
            axes = [np.arange(-(p // 2) * s + s // 2, (p // 2) * s, s) for p, s in zip(per, step)]
            centres = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, d)
            if inner.any():
                centres = centres[~np.all(np.abs(centres) < inner, axis=1)]
            inner = np.abs(centres).max(axis=0) + length // 2
            S = [2 * s for s in step]
            j = [torch.arange(m, device=DEVICE, dtype=torch.float64) - m / 2 for m in S]
            grid = torch.meshgrid(*j, indexing="ij")
            g = torch.exp(-sum((v / ((length // 2) * a)) ** 2 for v, a in zip(grid, aspect)))
            for v, s in zip(grid, step):
                g = g * (v.abs() < s)
            roll = np.stack([(1 - 2 * (((centres[:, a] + N[a]) // step[a]) & 1)) * (step[a] // 2) for a in range(d)], -1)
            # flat spectrum index of every element of every box, in the order of the box FFT's input
            flat = torch.zeros(len(centres), *S, dtype=torch.int64, device=DEVICE)
            gi = torch.zeros(len(centres), *S, dtype=torch.int64, device=DEVICE)
            for a in range(d):
                q = np.arange(S[a])
                jj = (q[None, :] + S[a] // 2 - roll[:, a:a + 1]) % S[a]
                k = (centres[:, a:a + 1] + N[a] // 2 - S[a] // 2 + jj) % N[a]
                shape = [len(centres)] + [1] * d
                shape[a + 1] = S[a]
                flat = flat * N[a] + torch.from_numpy(k).to(DEVICE).reshape(shape)
                gi = gi * S[a] + torch.from_numpy(jj).to(DEVICE).reshape(shape)
            gbox = g.reshape(-1)[gi]
            self.power.view(-1).index_add_(0, flat.reshape(-1), (gbox * gbox).reshape(-1))
            self.levels.append((length, centres, S, flat, gbox))

    def analysis(self, x):
        d = len(self.N)
        X = torch.fft.fftshift(torch.fft.fftn(x.to(torch.complex128), norm="ortho")) / self.power
        X = X.reshape(-1)
        return torch.cat([torch.fft.ifftn(X[flat] * g, dim=tuple(range(1, d + 1)), norm="ortho").reshape(-1)
                          for _, _, _, flat, g in self.levels])

    def adjoint(self, c):
        x = torch.zeros(*self.N, dtype=torch.float64, device=DEVICE, requires_grad=True)
        w = self.analysis(x)
        (g,) = torch.autograd.grad((torch.view_as_real(w) * torch.view_as_real(c)).sum(), x)
        return g

    def half(self):
        """Which coefficients a real image's beams come from: the first half of each level's boxes."""
        return torch.cat([torch.arange(f.numel(), device=DEVICE) < f.numel() // 2 for _, _, _, f, _ in self.levels])

    def beams(self, idx, L):
        """x0, p, alpha (imaginary part), unit amplitude and frequency of the beams of coefficients ``idx``."""
        d = len(self.N)
        out = [torch.zeros(len(idx), d, dtype=torch.float64, device=DEVICE) for _ in range(3)]
        amp = torch.zeros(len(idx), dtype=torch.complex128, device=DEVICE)
        om = torch.zeros(len(idx), dtype=torch.float64, device=DEVICE)
        start = 0
        for length, centres, S, flat, _ in self.levels:
            pick = (idx >= start) & (idx < start + flat.numel())
            loc = idx[pick] - start
            start += flat.numel()
            P = math.prod(S)
            cen = torch.from_numpy(centres).to(DEVICE)[loc // P]
            rem = loc % P
            k = torch.stack([(rem // math.prod(S[a + 1:])) % S[a] for a in range(d)], -1).double()
            f = cen.double() / torch.tensor(L, dtype=torch.float64, device=DEVICE)
            w = f.norm(dim=1)
            a0, cycles = 1.0, 0.0
            for a in range(d):
                width = length * self.aspect[a] / L[a]
                a0 *= math.sqrt(math.pi * L[a] / (2 * width * self.N[a])) * width / 2
                half = S[a] // 2
                roll = (1 - 2 * ((torch.div(cen[:, a] + self.N[a] // 2, half, rounding_mode="floor")) & 1)) * (half // 2)
                cycles = cycles + (cen[:, a] - roll) * k[:, a] / S[a]
                out[0][pick, a] = k[:, a] * L[a] / S[a]
                out[2][pick, a] = 2 * (math.pi * width / 2) ** 2 / w
            out[1][pick] = 2 * math.pi * f / w[:, None]
            amp[pick] = a0 * torch.exp(2j * math.pi * (cycles % 1.0))
            om[pick] = w
        return out[0], out[1], out[2], amp, om


def _dense(frame, idx, values, L, ts, pos, residual):
    """Data of the beams with coefficients ``values``, and per beam the sum of
    2 (data - residual) conj(beam) over times, receivers and both directions."""
    x0, p, al, unit, om = frame.beams(idx, L)
    eye = torch.eye(x0.shape[1], dtype=torch.complex128, device=DEVICE)
    speed = p.norm(dim=1)
    u = p / speed[:, None]
    H = (eye.real - u[:, :, None] * u[:, None, :]) / speed[:, None, None]
    M0 = torch.diag_embed(1j * al)
    y = torch.zeros(len(ts), len(pos), dtype=torch.float64, device=DEVICE)
    block = max(1, int(2e7 // len(pos)))

    def shapes(t):
        for c in (SPEED, -SPEED):
            for b in range(0, len(idx), block):
                s = slice(b, b + block)
                T = eye + c * t * (H[s].to(torch.complex128) @ M0[s])
                M = M0[s] @ torch.linalg.inv(T)
                A = 1.0 / torch.sqrt(torch.linalg.det(T))
                D = pos[None] - (x0[s] + c * t * u[s])[:, None, :]
                ph = (D * p[s][:, None, :]).sum(-1).to(torch.complex128)
                for i in range(D.shape[-1]):
                    for k in range(D.shape[-1]):
                        ph = ph + 0.5 * M[:, i, k, None] * (D[..., i] * D[..., k])
                yield s, A[:, None] * torch.exp(1j * om[s][:, None] * ph)

    for i, t in enumerate(ts):
        for s, K in shapes(float(t)):
            y[i] += 2 * ((unit[s] * values[s])[:, None] * K).sum(0).real
    if residual is None:
        return y, None
    r = (y - residual).to(torch.complex128)
    g = torch.zeros(len(idx), dtype=torch.complex128, device=DEVICE)
    for i, t in enumerate(ts):
        for s, K in shapes(float(t)):
            g[s] += 2 * torch.conj(unit[s]) * (torch.conj(K) @ r[i])
    return y, g


def exact(case, seed):
    d, n, kind = case["ndim"], case["n"], case["kind"]
    N, aspect = (n,) * d, (1,) * d
    if kind == "reversal":
        return None
    if kind == "frame":
        frame, x = _Frame(N, case["levels"], aspect), _image(N, seed, case["noise"])
        c = frame.analysis(x)
        return {"coeffs": c, "image": x.to(torch.complex128), "adjoint": frame.adjoint(c)}
    if kind == "select":
        frame = _Frame(N, case["levels"], aspect)
        if case["strategy"] != "top_n":
            return None
        c = 0.5 * frame.analysis(_image(N, seed)) * frame.half()
        keep = min(int(case["thr"]), int(frame.half().sum()))
        order = torch.sort(c.abs(), stable=True).indices[-keep:]
        return {"idx": None, "values": c[order]}
    nt, ns = _sizes(case)
    if case["medium"] != "hom" or (2 if kind == "step" else 1) * 2.0 * case["thr"] * nt * ns > 2.5e10:
        return None  # minutes of plain torch
    state = prepare(dict(case, host=False), seed)
    frame = _Frame(N, case["levels"], aspect)
    half = frame.half()
    c = 0.5 * frame.analysis(state["x"].double()) * half
    keep = min(int(case["thr"]), int(half.sum()))
    if case["frozen"]:
        chosen = 0.5 * frame.analysis(_image(N, seed) + 0.05 * _image(N, seed + 1)) * half
    else:
        chosen = c
    idx = torch.sort(chosen.abs(), stable=True).indices[-keep:]
    L = [n * _spacing(n)] * d
    pos = torch.from_numpy(np.ascontiguousarray(state["sensors"].positions)).to(DEVICE)
    y, g = _dense(frame, idx, c[idx], L, state["ts"], pos, state["data"].double() if kind == "step" else None)
    if kind == "forward":
        return {"data": y}
    G = torch.zeros_like(c)
    G[idx] = 0.5 * g
    return {"data": y, "gradient": frame.adjoint(G)}
