"""Performance cases of rdcu_b200: the calls its users make, through the Python binding.

Every case is one kind of call on one problem size:

* ``rhs``      one evaluation of the pseudospectral right-hand side (a user's own stepper);
* ``solve``    adaptive DP45 from a state to output times, dense output delivered at each
               (the CLI's ``-t``/``-d`` runs and the parameter studies of 2D patterns);
* ``advance``  a fixed number of DP45 attempts (long 3D runs between outputs);
* ``bdf``      the stiff path: finite differences and variable-order BDF to output times;
* ``adjoint``  a gradient through fixed DP45 steps (``rdcu_b200.adjoint``): forward, backward;
* ``ensemble`` many independent 2D problems of uneven size stepped together;
* ``lines``    defect lines of two consecutive 3D frames and their correlation.

Sizes are those of the benchmark workloads, the notebook runs and the tests; initial
states are band-limited random fields of unit amplitude, which is what the equations
settle to after their first transient, not white noise.
"""
from __future__ import annotations

import math
from typing import Dict, List

import numpy as np
import torch

import rdcu_b200 as R
from rdcu_b200 import adjoint as radj
from rdcu_b200.lines import Lines
from rdcu_b200.problems import brusselator_coupling_lines, cgle_coupling_lines

# Grid spacings of the standard runs: L = 100 on 128 or 256 points, 200 on 256, 200 on 8192.
ENSEMBLE_SIZES = (64, 96, 128, 192, 256)
LINE_EDGES, LINE_COMPONENTS = 32768, 512  # room for the lines of one frame


def listed() -> List[dict]:
    return [
        # one right-hand side of a small 2D grid: launches and latency
        {"name": "rhs_2d_64x48", "kind": "rhs", "shape": "64x48", "dx": 0.78},
        # the standard 2D run (L = 100, outputs along the way)
        {"name": "solve_2d_128", "kind": "solve", "shape": "128x128", "dx": 0.78125, "T": 0.5, "outputs": 2},
        # the notebook's 2D run at 256^2
        {"name": "solve_2d_256", "kind": "solve", "shape": "256x256", "dx": 0.390625, "T": 0.25, "outputs": 2},
        # a domain whose sides are no powers of two (radices 2, 3, 5)
        {"name": "solve_2d_250x180", "kind": "solve", "shape": "250x180", "dx": 0.5, "T": 0.3, "outputs": 1},
        # 3D turbulence, the benchmark's sizes; the larger one is its default workload
        {"name": "advance_3d_128", "kind": "advance", "shape": "128x128x128", "dx": 1.5625, "attempts": 6,
         "fixed": False, "h": 0.04},
        {"name": "advance_3d_256", "kind": "advance", "shape": "256x256x256", "dx": 0.78125, "attempts": 4,
         "fixed": False, "h": 0.015},
        # a 3D box of unequal sides at a fixed step (-F)
        {"name": "advance_3d_100x96x80", "kind": "advance", "shape": "100x96x80", "dx": 0.78125, "attempts": 8,
         "fixed": True, "h": 0.01},
        # the stiff path: the Brusselator benchmark and the notebook's 1D run
        {"name": "bdf_brusselator_256", "kind": "bdf", "problem": "brusselator", "shape": "256x256", "dx": 0.25,
         "T": 1.5},
        {"name": "bdf_cgle_1d_8192", "kind": "bdf", "problem": "cgle", "shape": "8192", "dx": 0.0244140625, "T": 0.25},
        # gradients of a 2D run with respect to its start and its coefficients
        {"name": "adjoint_2d_256", "kind": "adjoint", "shape": "256x256", "dx": 0.78125, "steps": 100, "K": 50},
        # a parameter study: 512 members of five sizes
        {"name": "ensemble_512", "kind": "ensemble", "members": 512, "T": 0.2},
        # two frames of a 3D run at the line tracker's default grid
        {"name": "lines_128", "kind": "lines", "shape": "128x128x128", "terms": 8},
    ]


# ------------------------------------------------------------------------------ ranges


def _smooth(n: int) -> bool:
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo: int, hi: int) -> int:
    """A length the transforms take, log-uniform in [lo, hi], odd ones among them."""
    n = max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    while not _smooth(n):
        n -= 1
    return n


def _shape(rng, ndim: int, lo: int, hi: int) -> str:
    return "x".join(str(_size(rng, lo, hi)) for _ in range(ndim))


def draw(rng) -> dict:
    kind = rng.choice(["rhs", "solve", "solve", "advance", "advance", "bdf", "adjoint", "ensemble", "lines"])
    dx = round(rng.uniform(0.4, 1.0), 4)
    if kind == "rhs":
        ndim = rng.choice([1, 2, 2, 3])
        lo, hi = {1: (16, 4096), 2: (16, 512), 3: (12, 160)}[ndim]
        return {"kind": kind, "shape": _shape(rng, ndim, lo, hi), "dx": dx}
    if kind == "solve":
        return {"kind": kind, "shape": _shape(rng, 2, 24, 512), "dx": dx, "T": round(rng.uniform(0.1, 0.4), 3),
                "outputs": rng.randint(1, 3)}
    if kind == "advance":
        return {"kind": kind, "shape": _shape(rng, 3, 32, 224), "dx": dx, "attempts": rng.randint(2, 4),
                "fixed": rng.random() < 0.3, "h": round(0.02 * dx * dx, 5)}
    if kind == "bdf":
        if rng.random() < 0.3:
            return {"kind": kind, "problem": "cgle", "shape": str(_size(rng, 512, 8192)),
                    "dx": round(rng.uniform(0.025, 0.1), 4), "T": round(rng.uniform(0.1, 0.2), 3)}
        return {"kind": kind, "problem": "brusselator", "shape": _shape(rng, 2, 32, 256),
                "dx": round(rng.uniform(0.25, 0.5), 4), "T": round(rng.uniform(0.5, 1.5), 3)}
    if kind == "adjoint":
        return {"kind": kind, "shape": _shape(rng, 2, 32, 256), "dx": dx, "steps": rng.randint(20, 100),
                "K": rng.choice([10, 25, 50])}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(16, 256), "T": round(rng.uniform(0.1, 0.2), 3)}
    return {"kind": kind, "shape": _shape(rng, 3, 32, 160), "terms": rng.randint(3, 8)}


# ------------------------------------------------------------------------------ inputs


def _dims(case: dict):
    return tuple(int(v) for v in case["shape"].split("x"))


def _device() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _field(shape, dx: float, gen: torch.Generator, batch: int = 1) -> torch.Tensor:
    """(batch, 2, *shape) real fields, band-limited (correlation length about 4 units),
    root-mean-square amplitude 0.7 each."""
    dev = _device()
    white = torch.randn((batch, 2) + tuple(shape), dtype=torch.float64, device=dev, generator=gen)
    axes = list(range(2, 2 + len(shape)))
    spec = torch.fft.fftn(white, dim=axes)
    for a, n in zip(axes, shape):
        k = 2 * math.pi * torch.fft.fftfreq(n, d=dx, dtype=torch.float64, device=dev)
        spec = spec * torch.exp(-(1.2 * k) ** 2).reshape([-1 if b == a else 1 for b in range(2 + len(shape))])
    y = torch.fft.ifftn(spec, dim=axes).real
    rms = y.reshape(batch, -1).square().mean(dim=1).sqrt().reshape([batch] + [1] * (1 + len(shape)))
    return (0.7 * y / rms).contiguous()


def _terms(lines):
    return R.parse_terms(lines)


def _cgle_solver(case: dict, fixed: bool = False) -> R.Solver:
    shape = _dims(case)
    return R.Solver(2, shape, tuple(n * case["dx"] for n in shape), _terms(cgle_coupling_lines(len(shape))),
                    fixed=fixed)


def _output_times(case: dict) -> List[float]:
    m = case.get("outputs", 1)
    return [case["T"] * (j + 1) / m for j in range(m)]


def _first_step(dx: float) -> float:
    """A first step inside DP45's stability range: what a run has settled to after its start."""
    return 0.02 * dx * dx / 0.61


def _ensemble_members(case: dict, seed: int):
    m = case["members"]
    order = np.random.default_rng(3)
    sizes = order.choice(ENSEMBLE_SIZES, size=m)
    par = np.random.default_rng(int(seed))
    bs, cs = par.uniform(0.5, 3.0, size=m), par.uniform(-2.0, 0.0, size=m)
    return [int(n) for n in sizes], [float(b) for b in bs], [float(c) for c in cs]


def _ensemble_states(sizes, seed: int) -> List[torch.Tensor]:
    gen = _generator(seed)
    ys: List[torch.Tensor] = [None] * len(sizes)
    for n in sorted(set(sizes)):
        at = [i for i, s in enumerate(sizes) if s == n]
        batch = _field((n, n), 0.78, gen, len(at))
        for j, i in enumerate(at):
            ys[i] = batch[j].reshape(-1)
    return ys


def _frames(case: dict, seed: int) -> List[torch.Tensor]:
    """Two consecutive frames of a state with vortex lines: every term adds four periodic
    lines along one axis, which wobble along it and drift between the frames; the phase
    carries 0.1 of noise."""
    shape = _dims(case)
    dev = _device()
    rng = np.random.default_rng(int(seed))
    gen = _generator(seed)
    grid = torch.meshgrid(*[torch.arange(n, dtype=torch.float64, device=dev) for n in shape], indexing="ij")
    terms = []
    for _ in range(case["terms"]):
        ax = int(rng.integers(3))
        a, b = [x for x in range(3) if x != ax]
        terms.append((ax, a, b, rng.uniform(0, shape[a]), rng.uniform(0, shape[b]), *(0.7 * rng.normal(size=2)),
                      rng.uniform(0, 2.5), rng.uniform(0, 2 * np.pi)))
    out = []
    for k in range(2):
        th = torch.zeros(shape, dtype=torch.float64, device=dev)
        for ax, a, b, p0, q0, vp, vq, amp, ph in terms:
            s = 2 * np.pi * grid[ax] / shape[ax] + ph
            p, q = p0 + vp * k + amp * torch.sin(s), q0 + vq * k + amp * torch.cos(s)
            th += torch.atan2(torch.sin(2 * np.pi * (grid[b] - q) / shape[b]),
                              torch.sin(2 * np.pi * (grid[a] - p) / shape[a]))
        th += 0.1 * torch.randn(shape, dtype=torch.float64, device=dev, generator=gen)
        r = 1.0 + 0.2 * torch.rand(shape, dtype=torch.float64, device=dev, generator=gen)
        out.append(torch.cat([(r * torch.cos(th)).reshape(-1), (r * torch.sin(th)).reshape(-1)]))
    return out


def _bdf_state(case: dict, seed: int) -> torch.Tensor:
    shape = _dims(case)
    gen = _generator(seed)
    if case["problem"] == "cgle":
        return _field(shape, case["dx"], gen)[0].reshape(-1)
    y = 0.1 * (2 * torch.rand((2,) + shape, dtype=torch.float64, device=_device(), generator=gen) - 1)
    y[0] += 1.0
    y[1] += 3.0
    return y.reshape(-1)


def prepare(case: dict, seed: int) -> Dict:
    kind = case["kind"]
    st: Dict = {"kind": kind}
    if kind in ("rhs", "solve", "advance"):
        shape = _dims(case)
        st["solver"] = _cgle_solver(case, fixed=bool(case.get("fixed", False)))
        st["y0"] = _field(shape, case["dx"], _generator(seed))[0].reshape(-1)
        if kind == "rhs":
            st["out"] = torch.empty_like(st["y0"])
        elif kind == "advance":
            st["attempts"], st["h"] = case["attempts"], case["h"]
            st["out"] = torch.empty_like(st["y0"])
        else:
            st["times"], st["h"] = _output_times(case), _first_step(case["dx"])
            st["out"] = torch.empty((len(st["times"]), st["y0"].numel()), dtype=torch.float64, device="cuda")
    elif kind == "bdf":
        shape = _dims(case)
        lines = cgle_coupling_lines(len(shape)) if case["problem"] == "cgle" else brusselator_coupling_lines()
        st["solver"] = R.Solver(2, shape, tuple(n * case["dx"] for n in shape), _terms(lines), method=R.METHOD_BDF,
                                rtol=1e-6, atol=1e-6)
        st["y0"] = _bdf_state(case, seed)
        st["times"], st["h"] = _output_times(case), 1e-3
        st["out"] = torch.empty((len(st["times"]), st["y0"].numel()), dtype=torch.float64, device="cuda")
    elif kind == "adjoint":
        shape = _dims(case)
        gen = _generator(seed)
        st["solver"] = _cgle_solver(case, fixed=True)
        st["y0"] = _field(shape, case["dx"], gen)[0].reshape(-1)
        st["C"] = torch.tensor([c for c, _ in _terms(cgle_coupling_lines(len(shape)))], dtype=torch.float64)
        st["w"] = torch.randn(st["y0"].shape, dtype=torch.float64, device="cuda", generator=gen)
        st["hs"], st["K"] = [1e-3] * case["steps"], case["K"]
    elif kind == "ensemble":
        sizes, bs, cs = _ensemble_members(case, seed)
        members = [dict(n=2, Ns=(n, n), Ls=(0.78 * n, 0.78 * n), terms=_terms(cgle_coupling_lines(2, b, c)))
                   for n, b, c in zip(sizes, bs, cs)]
        st["ensemble"] = R.Ensemble(members)
        st["y0"] = _ensemble_states(sizes, seed)
        st["out"] = [torch.empty_like(y) for y in st["y0"]]
        st["all"] = torch.empty(sum(y.numel() for y in st["y0"]), dtype=torch.float64, device="cuda")
        at = 0
        for i, y in enumerate(st["y0"]):
            st["out"][i] = st["all"][at:at + y.numel()]
            at += y.numel()
        st["T"] = case["T"]
    else:
        shape = _dims(case)
        st["frames"] = _frames(case, seed)
        Ls = tuple(0.4 * n for n in shape)
        st["handles"] = [Lines(shape, Ls), Lines(shape, Ls)]
        # where a program that follows the lines keeps them: grown in steps, zero past the end
        st["edges"] = [np.zeros((LINE_EDGES, 2, 3)), np.zeros((LINE_EDGES, 2, 3))]
        st["offsets"] = [np.zeros(LINE_COMPONENTS + 1, np.int64), np.zeros(LINE_COMPONENTS + 1, np.int64)]
        st["distances"] = np.zeros((LINE_COMPONENTS, LINE_COMPONENTS), np.int64)
        st["filled"] = [0, 0, 0, 0]
    return st


# -------------------------------------------------------------------------------- pass


def _solve_to_outputs(st: Dict) -> torch.Tensor:
    s, out = st["solver"], st["out"]
    nbytes = out.shape[1] * 8

    def deliver(ev):
        if ev.kind == R.EV_EVAL:
            s.memcpy(out[ev.eval_index].data_ptr(), ev.y, nbytes)
        return 0

    s.set_state(0.0, st["h"], st["y0"])
    s.solve(st["times"][-1], st["times"], callback=deliver)
    return out


def _keep(buffer: np.ndarray, values: np.ndarray, filled: List[int], i: int) -> None:
    """`values` at the front of `buffer`, zeros after them."""
    buffer[:len(values)] = values
    if filled[i] > len(values):
        buffer[len(values):filled[i]] = 0
    filled[i] = len(values)


def run(st: Dict):
    kind = st["kind"]
    if kind == "rhs":
        st["solver"].rhs(st["y0"], st["out"])
        return st["out"]
    if kind in ("solve", "bdf"):
        return _solve_to_outputs(st)
    if kind == "advance":
        s = st["solver"]
        s.set_state(0.0, st["h"], st["y0"])
        s.advance(st["attempts"])
        t, _, _ = s.get_state(st["out"])
        return {"y": st["out"], "t": t}
    if kind == "adjoint":
        y0 = st["y0"].detach().requires_grad_(True)
        C = st["C"].detach().requires_grad_(True)
        yT = radj.integrate(st["solver"], y0, C, st["hs"], st["K"])
        (yT * st["w"]).sum().backward()
        return {"yT": yT.detach(), "y0": y0.grad, "C": C.grad}
    if kind == "ensemble":
        e = st["ensemble"]
        for i, y in enumerate(st["y0"]):
            e.set_state(i, 0.0, 0.01, y)
        e.solve(st["T"])
        ts = np.empty(len(st["out"]))
        for i, y in enumerate(st["out"]):
            ts[i], _ = e.get_state(i, y)
        return {"y": st["all"], "t": ts}
    for i, (handle, frame) in enumerate(zip(st["handles"], st["frames"])):
        handle.find(frame)
        xyz, off = handle.edges()
        _keep(st["edges"][i], xyz, st["filled"], i)
        _keep(st["offsets"][i], off, st["filled"], 2 + i)
    d = st["handles"][1].correlate(st["handles"][0])
    if st.get("corner") not in (None, d.shape):
        st["distances"][:] = 0
    st["distances"][:d.shape[0], :d.shape[1]] = d
    st["corner"] = d.shape
    return {"edges": st["edges"], "offsets": st["offsets"], "distances": st["distances"]}


# -------------------------------------------------------------------------------- work


def _attempts(T: float, dx: float, ndim: int) -> float:
    """Steps of an adaptive CGLE run to T: DP45's stability limit (3.3 over the largest
    symbol sqrt(5) ndim (pi/dx)^2), or about 0.03 where accuracy limits it."""
    return T / min(0.03, 3.3 / (math.sqrt(5.0) * ndim * (math.pi / dx) ** 2))


def _dp45_work(N: float, ndim: int, attempts: float) -> Dict[str, float]:
    """41 state-sized arrays per accepted step, and in 3D the spectra of the strided
    axes; six right-hand sides of two forward and two inverse real transforms."""
    per_point = 656.0 if ndim < 3 else 1040.0
    fft = 6 * 4 * 2.5 * math.log2(max(2.0, N))
    return {"bytes": per_point * N * attempts, "flops": (fft + 6 * 40 + 150) * N * attempts}


def work(case: dict) -> Dict[str, float]:
    kind = case["kind"]
    if kind == "ensemble":
        sizes, _, _ = _ensemble_members(case, 0)
        return _dp45_work(float(sum(n * n for n in sizes)), 2, _attempts(case["T"], 0.78, 2))
    shape = _dims(case)
    N = float(np.prod(shape))
    if kind == "rhs":
        return {"bytes": 32.0 * N, "flops": (4 * 2.5 * math.log2(N) + 40) * N}
    if kind == "solve":
        return _dp45_work(N, 2, _attempts(case["T"], case["dx"], 2))
    if kind == "advance":
        return _dp45_work(N, 3, float(case["attempts"]))
    if kind == "bdf":
        # about 40 steps of three Newton iterations; each solves with about ten products
        # and as many basis vectors of two fields
        return {"bytes": 40 * 3 * 10 * 12 * 16.0 * N, "flops": 40 * 3 * 10 * 120.0 * N}
    if kind == "adjoint":
        return _dp45_work(N, 2, 3.0 * case["steps"])
    return {"bytes": 2 * 16.0 * N, "flops": 2 * 120.0 * N}


# ------------------------------------------------------------- the same in plain torch

_A = [[], [1.0 / 5], [3.0 / 40, 9.0 / 40], [44.0 / 45, -56.0 / 15, 32.0 / 9],
      [19372.0 / 6561, -25360.0 / 2187, 64448.0 / 6561, -212.0 / 729],
      [9017.0 / 3168, -355.0 / 33, 46732.0 / 5247, 49.0 / 176, -5103.0 / 18656],
      [35.0 / 384, 0.0, 500.0 / 1113, 125.0 / 192, -2187.0 / 6784, 11.0 / 84]]
_E = [-71.0 / 57600, 0.0, 71.0 / 16695, -71.0 / 1920, 17253.0 / 339200, -22.0 / 525, 1.0 / 40]
_P = [[1.0, -8048581381.0 / 2820520608, 8663915743.0 / 2820520608, -12715105075.0 / 11282082432],
      [0, 0, 0, 0],
      [0, 131558114200.0 / 32700410799, -68118460800.0 / 10900136933, 87487479700.0 / 32700410799],
      [0, -1754552775.0 / 470086768, 14199869525.0 / 1410260304, -10690763975.0 / 1880347072],
      [0, 127303824393.0 / 49829197408, -318862633887.0 / 49829197408, 701980252875.0 / 199316789632],
      [0, -282668133.0 / 205662961, 2019193451.0 / 616988883, -1453857185.0 / 822651844],
      [0, 40617522.0 / 29380423, -110615467.0 / 29380423, 69997945.0 / 29380423]]


def _combine(ks, weights):
    out = None
    for k, w in zip(ks, weights):
        if w != 0:
            out = w * k if out is None else out + w * k
    return out


class _Cgle:
    """The CGLE right-hand side on (batch, 2, *shape) fields, pseudospectral."""

    def __init__(self, shape, dx: float, b, c):
        dev = _device()
        self.axes = list(range(2, 2 + len(shape)))
        col = [-1] + [1] * len(shape)
        self.b = torch.as_tensor(b, dtype=torch.float64, device=dev).reshape(col)
        self.c = torch.as_tensor(c, dtype=torch.float64, device=dev).reshape(col)
        self.lap = torch.zeros((1, 1) + tuple(shape), dtype=torch.float64, device=dev)
        for a, n in zip(self.axes, shape):
            na = torch.arange(n, dtype=torch.float64, device=dev)
            k = 2 * math.pi / (n * dx) * torch.where(na < n // 2, na, na - n)
            self.lap = self.lap - (k * k).reshape([-1 if d == a else 1 for d in range(2 + len(shape))])

    def __call__(self, y: torch.Tensor) -> torch.Tensor:
        d = torch.fft.ifftn(self.lap * torch.fft.fftn(y, dim=self.axes), dim=self.axes).real
        u, v, du, dv = y[:, 0], y[:, 1], d[:, 0], d[:, 1]
        r = u * u + v * v
        return torch.stack([u + du - self.b * dv - r * (u + self.c * v),
                            v + dv + self.b * du - r * (v - self.c * u)], dim=1)


def _column(h: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
    return h.reshape([-1] + [1] * (y.dim() - 1))


def _stages(f, y, h, k1):
    ks = [k1]
    for s in range(1, 6):
        ks.append(f(y + h * _combine(ks, _A[s])))
    yn = y + h * _combine(ks, _A[6])
    ks.append(f(yn))
    return yn, ks


def _dp45(f, y, h0: float, attempts=None, T=None, times=(), fixed=False, rtol=1e-8, atol=1e-8):
    """Adaptive DP45 of every batch member by its own steps: `attempts` of them, or until
    its first accepted step at or past T.  Returns (y, t, values at `times`)."""
    B = y.shape[0]
    h = torch.full((B,), h0, dtype=torch.float64, device=y.device)
    t = torch.zeros_like(h)
    n = y[0].numel()
    k1 = f(y)
    outs, done, i = [], 0, 0
    while i < attempts if attempts is not None else bool((t < T).any()):
        i += 1
        live = torch.ones_like(t, dtype=torch.bool) if T is None else t < T
        H = _column(h, y)
        yn, ks = _stages(f, y, H, k1)
        if fixed:
            ok, factor = live, torch.ones_like(h)
        else:
            e = H * _combine(ks, _E) / (atol + rtol * torch.maximum(y.abs(), yn.abs()))
            norm = (e.reshape(B, -1).square().sum(dim=1) / n).sqrt()
            factor = 0.9 * norm ** -0.2
            good = norm < 1
            ok = live & good
            factor = torch.where(good, factor.clamp(max=10.0), factor.clamp(min=0.2, max=1.0))
        if bool(ok.all()) and done < len(times):  # dense output: single problems only
            t1 = float(t[0] + h[0])
            while done < len(times) and t1 >= times[done]:
                x = (times[done] - float(t[0])) / (t1 - float(t[0]))
                w = [sum(p * x ** (j + 1) for j, p in enumerate(row)) for row in _P]
                outs.append((y + (t1 - float(t[0])) * _combine(ks, w)).reshape(-1))
                done += 1
        m = _column(ok, y)
        y, k1 = torch.where(m, yn, y), torch.where(m, ks[6], k1)
        t = torch.where(ok, t + h, t)
        h = torch.where(live, h * factor, h)
    return y, t, outs


def _fd_rhs(case: dict):
    """The finite-difference right-hand side of the stiff problems."""
    dx = case["dx"]

    def lap(u):
        d = torch.zeros_like(u)
        for a in range(u.dim()):
            d = d + (torch.roll(u, 1, a) - 2 * u + torch.roll(u, -1, a)) / (dx * dx)
        return d

    def brusselator(y):
        u, v = y[0, 0], y[0, 1]
        r = u * u * v
        return torch.stack([1 - 4 * u + r + lap(u), 3 * u - r + 8 * lap(v)])[None]

    def cgle(y):
        u, v = y[0, 0], y[0, 1]
        r, du, dv = u * u + v * v, lap(u), lap(v)
        return torch.stack([u + du - 2.0 * dv - r * (u + 0.8 * v), v + dv + 2.0 * du - r * (v - 0.8 * u)])[None]

    return cgle if case["problem"] == "cgle" else brusselator


def _line_edges(y: torch.Tensor, shape) -> torch.Tensor:
    """The scaled edges of a frame's line components, component by component."""
    dev = y.device
    n = int(np.prod(shape))
    th = (torch.atan2(y[n:], y[:n]) + math.pi).reshape(shape)

    def wrap(x):
        return torch.remainder(x + math.pi, 2 * math.pi) - math.pi

    def wound(a, b):
        t1, t3 = torch.roll(th, -1, a), torch.roll(th, -1, b)
        t2 = torch.roll(t1, -1, b)
        return torch.round((wrap(t1 - th) + wrap(t2 - t1) + wrap(t3 - t2) + wrap(th - t3)) / (2 * math.pi)) != 0

    mark = torch.zeros(shape, dtype=torch.bool, device=dev)
    for a, b, c in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        w = wound(a, b)
        mark |= w | torch.roll(w, -1, c)
    label = torch.where(mark, torch.arange(n, device=dev).reshape(shape), n)
    while True:  # every cube takes the smallest index of its component
        new = label
        for a in range(3):
            for s in (1, -1):
                new = torch.where(mark, torch.minimum(new, torch.roll(new, s, a)), n)
        if torch.equal(new, label):
            break
        label = new
    cube = torch.nonzero(mark.reshape(-1)).reshape(-1)
    at = torch.stack([cube // (shape[1] * shape[2]), cube // shape[2] % shape[1], cube % shape[2]], dim=1)
    sizes = torch.tensor(shape, device=dev)
    us, vs = [], []
    for a in range(3):
        for s in (1, -1):
            other = at.clone()
            other[:, a] = (other[:, a] + s) % shape[a]
            idx = (other[:, 0] * shape[1] + other[:, 1]) * shape[2] + other[:, 2]
            keep = mark.reshape(-1)[idx] & (idx > cube)
            us.append(cube[keep])
            vs.append(idx[keep])
    pairs = torch.unique(torch.cat(us) * n + torch.cat(vs))  # ascending (u, v), each once
    u, v = pairs // n, pairs % n
    order = torch.argsort(label.reshape(-1)[u], stable=True)
    e = torch.stack([u[order], v[order]], dim=1)
    xyz = torch.stack([e // (shape[1] * shape[2]), e // shape[2] % shape[1], e % shape[2]], dim=2).double()
    L = torch.tensor([0.4 * m for m in shape], dtype=torch.float64, device=dev)
    return xyz * L / (sizes - 1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "ensemble":
        sizes, bs, cs = _ensemble_members(case, seed)
        ys = _ensemble_states(sizes, seed)
        ts = np.empty(len(sizes))
        for n in sorted(set(sizes)):
            at = [i for i, s in enumerate(sizes) if s == n]
            f = _Cgle((n, n), 0.78, [float("%f" % bs[i]) for i in at], [float("%f" % cs[i]) for i in at])
            y, t, _ = _dp45(f, torch.stack([ys[i].reshape(2, n, n) for i in at]), 0.01, T=case["T"])
            for j, i in enumerate(at):
                ys[i], ts[i] = y[j].reshape(-1), float(t[j])
        return {"y": torch.cat(ys), "t": ts}
    shape = _dims(case)
    if kind == "lines":
        edges = [torch.zeros((LINE_EDGES, 2, 3), dtype=torch.float64) for _ in range(2)]
        for kept, frame in zip(edges, _frames(case, seed)):
            xyz = _line_edges(frame, shape).cpu()
            kept[:len(xyz)] = xyz
        return {"edges": edges, "offsets": [None, None], "distances": None}
    if kind == "bdf":
        # the solution itself, by explicit steps far inside their tolerance
        y = _bdf_state(case, seed).reshape((1, 2) + shape)
        big = (8.0 if case["problem"] == "brusselator" else math.sqrt(5.0)) * 4 * len(shape) / case["dx"] ** 2
        steps = math.ceil(case["T"] * big / 2.5)
        if steps > 8000:
            return None
        f, h = _fd_rhs(case), case["T"] / steps
        k1 = f(y)
        for _ in range(steps):
            y, ks = _stages(f, y, h, k1)
            k1 = ks[6]
        return y.reshape(1, -1)
    gen = _generator(seed)
    y = _field(shape, case["dx"], gen)
    f = _Cgle(shape, case["dx"], 2.0, 0.8)
    if kind == "rhs":
        return f(y).reshape(-1)
    if kind == "solve":
        times = _output_times(case)
        _, _, outs = _dp45(f, y, _first_step(case["dx"]), T=times[-1], times=times)
        return torch.stack(outs)
    if kind == "advance":
        y, t, _ = _dp45(f, y, case["h"], attempts=case["attempts"], fixed=bool(case["fixed"]))
        return {"y": y.reshape(-1), "t": float(t[0])}
    # adjoint: torch's own gradient of the same steps
    w = torch.randn(2 * int(np.prod(shape)), dtype=torch.float64, device=_device(), generator=gen)
    C = torch.tensor([c for c, _ in _terms(cgle_coupling_lines(len(shape)))], dtype=torch.float64, device=_device(),
                     requires_grad=True)
    monomials = [ints for _, ints in _terms(cgle_coupling_lines(len(shape)))]
    y0 = y[0].reshape(-1).clone().requires_grad_(True)
    ndim = len(shape)
    seconds = []
    for a, n in enumerate(shape):
        na = torch.arange(n, dtype=torch.float64, device=_device())
        k = 2 * math.pi / (n * case["dx"]) * torch.where(na < n // 2, na, na - n)
        seconds.append(-(k * k).reshape([-1 if d == a else 1 for d in range(ndim)]))

    def rhs(s):
        u = s.reshape((2,) + shape)
        uh = [torch.fft.fftn(u[i]) for i in range(2)]
        block = {0: u[0], 1: u[1]}
        for a in range(ndim):
            for i in range(2):
                block[2 + 2 * ndim + (a * ndim + a) * 2 + i] = torch.fft.ifftn(seconds[a] * uh[i]).real
        out = [torch.zeros_like(u[0]), torch.zeros_like(u[1])]
        for q, ints in enumerate(monomials):
            m = C[q]
            for j in range(1, len(ints), 2):
                m = m * block[ints[j]] ** ints[j + 1]
            out[ints[0]] = out[ints[0]] + m
        return torch.stack(out).reshape(-1)

    s = y0
    for _ in range(case["steps"]):
        ks = [rhs(s)]
        for j in range(1, 6):
            ks.append(rhs(s + 1e-3 * _combine(ks, _A[j])))
        s = s + 1e-3 * _combine(ks, _A[6])
    (s * w).sum().backward()
    return {"yT": s.detach(), "y0": y0.grad, "C": C.grad}
