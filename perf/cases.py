"""The work that a user of vlapy_gb300 has it do, as timed cases.

Every case goes through the package's public entry points, on inputs made from
a seed.  ``listed()`` names the cases, ``draw(rng)`` gives more of the same
ranges, ``prepare`` makes what a program holds before the call, ``run`` is one
pass, ``work`` what that pass cannot do without, and ``exact`` the same result
in 64 bits by plain torch (FFTs, a row-by-row elimination, dense spline
systems), without the package.

Kinds of case:
  loop     the inner loop or the per-step closure of a single run, through
           outer_loop.get_inner_loop_stepper / core.step.get_timestep
  plan     steps of a large single run through Plan.run_steps, replayed as a graph
  sweep    steps of many FP32 runs together (sweep.Sweep)
  batch    steps of many FP64 runs together (batch.Batch64)
  apply    one learned correction of coarse rows (corrector.Corrector.apply)
  train    loss and gradients of one training batch (Corrector.gradients)

The float64 buffers of the FP32 modes hold FP32 results; they are handed back
as float32, the precision they carry.
"""

from __future__ import annotations

import math

import numpy as np
import torch

VMAX, DT = 6.0, 0.1
FIELDS = ("e", "driver", "n", "j", "T", "q", "fv4", "vN")
SERIES = ("mean_n", "mean_j", "mean_T", "mean_e2", "mean_de2", "mean_f2", "mean_flogf")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _loop(name, nx, nv, steps, precision="fp64", time="leapfrog", op="none", x_step="exponential",
          v_step="exponential", driven=False, per_step=False):
    c = dict(kind="loop", nx=nx, nv=nv, steps=steps, precision=precision, time=time, op=op, x_step=x_step,
             v_step=v_step, driven=driven, per_step=per_step)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one call of the per-step closure on the reference's default grid: the
        # smallest call a drop-in user makes, all latency and launches
        _loop("step_fp64_32x512", 32, 512, 1, per_step=True),
        # a batch of the driven-wave run in the parity mode, as the run manager
        # asks for it between two writes of its history
        _loop("driven_fp64_64x1024", 64, 1024, 20, op="dg", driven=True),
        # the same run in the throughput mode
        _loop("driven_fp32_64x1024", 64, 1024, 100, precision="fp32-deltaf", op="dg", driven=True),
        # grids that are no powers of two (the reference takes any length), with
        # the default collision operator
        _loop("ragged_fp64_48x720", 48, 720, 4, op="lb"),
        # the alternative steppers a user picks by name: the composed time step
        _loop("sl_fp64_64x1024", 64, 1024, 4, op="dg", x_step="sl", v_step="sl"),
        # the large two-stream run in the parity mode, one step
        dict(name="large_fp64_2048x4096", kind="plan", nx=2048, nv=4096, steps=1, precision="fp64"),
        # the large two-stream run at full size in the throughput mode
        dict(name="large_fp32_4096x8192", kind="plan", nx=4096, nv=8192, steps=4, precision="fp32-deltaf"),
        # the parameter sweep of the benchmark: all shapes, all runs
        dict(name="sweep_4096", kind="sweep", runs=4096, nx_lo=32, nx_hi=128, nv_lo=256, nv_hi=1024, steps=8),
        # a small scan, as when a user looks at a few dozen parameters
        dict(name="sweep_64", kind="sweep", runs=64, nx_lo=32, nx_hi=128, nv_lo=256, nv_hi=1024, steps=20),
        # the FP64 judge of a scan
        dict(name="batch_192", kind="batch", runs=192, nx_lo=32, nx_hi=128, nv_lo=256, nv_hi=1024, steps=2),
        # one learned correction of 2048 coarse runs
        dict(name="apply_2048x64", kind="apply", runs=2048, nx=64),
        # one training batch of the corrector: 128 runs of 64 rows
        dict(name="train_128x64", kind="train", runs=128, nx=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo, hi):
    return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))


def draw(rng):
    """One more case: any kind, sizes spread over its range."""
    kind = rng.choice(("loop64", "loop64", "loop32", "ragged", "alt", "plan", "sweep", "sweep", "batch", "apply",
                       "train"))
    op = rng.choice(("none", "lb", "dg", "dg"))
    time = rng.choice(("leapfrog", "leapfrog", "leapfrog", "pefrl", "h-sixth"))
    per_step = rng.random() < 0.3
    if kind == "loop64":
        return _loop(None, _pow2(rng, 8, 256), _pow2(rng, 128, 2048), 1 if per_step else rng.randint(2, 4), time=time,
                     op=op, driven=rng.random() < 0.5, per_step=per_step)
    if kind == "loop32":
        steps = _log_int(rng, 4, 60) if time == "leapfrog" else rng.randint(2, 8)
        return _loop(None, _pow2(rng, 16, 256), _pow2(rng, 128, 4096), 1 if per_step else steps,
                     precision="fp32-deltaf", time=time, op=op, driven=op != "none" and rng.random() < 0.5,
                     per_step=per_step)
    if kind == "ragged":
        return _loop(None, _log_int(rng, 12, 128), _log_int(rng, 100, 1024), 1 if per_step else rng.randint(1, 2),
                     op=op, driven=rng.random() < 0.5, per_step=per_step)
    if kind == "alt":
        x_step, v_step = rng.choice((("sl", "sl"), ("sl", "sl"), ("exponential", "cd2"), ("sl", "exponential")))
        pow2 = "exponential" in (x_step, v_step)
        nx = _pow2(rng, 16, 256) if pow2 else _log_int(rng, 16, 256)
        nv = _pow2(rng, 256, 2048) if pow2 else _log_int(rng, 200, 2000)
        return _loop(None, nx, nv, 1 if per_step else rng.randint(1, 4), op=op, x_step=x_step, v_step=v_step,
                     per_step=per_step)
    if kind == "plan":
        precision = rng.choice(("fp64", "fp32-deltaf", "fp32-deltaf"))
        hi = 2048 if precision == "fp64" else 4096
        return dict(kind="plan", nx=_pow2(rng, 256, hi), nv=_pow2(rng, 1024, 4096 if precision == "fp64" else 8192),
                    steps=1 if precision == "fp64" else rng.randint(1, 4), precision=precision)
    if kind in ("sweep", "batch"):
        nx_lo, nv_lo = _pow2(rng, 16, 64), _pow2(rng, 256, 512)
        if nx_lo == 16:
            nv_lo = 512  # the sweep's narrowest grids have wide column tiles
        nx_hi, nv_hi = min(256, nx_lo * _pow2(rng, 1, 4)), min(1024, nv_lo * _pow2(rng, 1, 4))
        if kind == "batch":
            return dict(kind="batch", runs=_log_int(rng, 6, 128), nx_lo=nx_lo, nx_hi=min(nx_hi, 128), nv_lo=nv_lo,
                        nv_hi=nv_hi, steps=rng.randint(1, 2))
        return dict(kind="sweep", runs=_log_int(rng, 16, 2048), nx_lo=nx_lo, nx_hi=nx_hi, nv_lo=nv_lo, nv_hi=nv_hi,
                    steps=rng.randint(2, 8))
    if kind == "apply":
        return dict(kind="apply", runs=_log_int(rng, 8, 2048), nx=rng.choice((32, 60, 64)))
    return dict(kind="train", runs=_log_int(rng, 8, 128), nx=rng.choice((32, 60, 64)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _x_axis(nx, k):
    """Cell-centred x grid of one wavelength, its wavenumbers and their inverses (0 for the mean)."""
    length = 2.0 * np.pi / k
    dx = length / nx
    x = np.linspace(dx / 2.0, length - dx / 2.0, nx)
    kx = np.fft.fftfreq(nx, d=dx) * 2.0 * np.pi
    inv = np.zeros(nx)
    inv[1:] = 1.0 / kx[1:]
    return dx, x, kx, inv


def _v_axis(nv, vmax):
    dv = 2.0 * vmax / nv
    v = np.linspace(-vmax + dv / 2.0, vmax - dv / 2.0, nv)
    return dv, v, np.fft.fftfreq(nv, d=dv) * 2.0 * np.pi


def _trapz(f, dv):
    return dv * (f.sum(-1) - 0.5 * (f[..., 0] + f[..., -1]))


def _single(case, seed):
    """Grids, initial f, parameters and driver of a single run: a Maxwellian
    with a weak bump on its tail (two unequal streams for the large run) and
    a density perturbation of a few modes."""
    rng = np.random.default_rng([seed, 1])
    large = case["kind"] == "plan"
    nx, nv = case["nx"], case["nv"]
    k = float(rng.uniform(0.25, 0.45))
    vmax, dt = (8.0, 0.05) if large else (VMAX, DT)
    dx, x, kx, inv = _x_axis(nx, k)
    dv, v, kv = _v_axis(nv, vmax)
    if large:
        u = rng.uniform(2.8, 3.2)
        w = rng.uniform(0.52, 0.6)
        fv = w * np.exp(-((v - u) ** 2) / 2.0) + (1.0 - w) * np.exp(-((v + u) ** 2) / 2.0)
        modes, amp = 16, 1e-3
    else:
        fv = np.exp(-(v ** 2) / 2.0) + rng.uniform(0.01, 0.04) * np.exp(-((v - 3.0) ** 2) / 0.8)
        modes, amp = 3, 10.0 ** rng.uniform(-3.7, -3.3)
    fv = fv / _trapz(fv, dv)
    pert = np.zeros(nx)
    for m in range(1, min(modes, nx // 2 - 1) + 1):
        pert += amp * rng.uniform(0.3, 1.0) * np.cos(m * k * x + rng.uniform(0.0, 2.0 * np.pi))
    op = "dg" if large else case["op"]
    nu = 0.0 if op == "none" else (1e-4 if large else float(10.0 ** rng.uniform(-4.0, -2.5)))
    steps = case["steps"]
    t0 = float(rng.uniform(10.0, 40.0))
    pulse = None
    if case.get("driven"):
        pulse = dict(k0=k, w0=float(rng.uniform(1.1, 1.3)), a0=2e-3, t_L=0.0, t_R=100.0, envelope="sin2")
    return dict(nx=nx, nv=nv, k=k, dx=dx, x=x, kx=kx, inv=inv, dv=dv, v=v, kv=kv, dt=dt, nu=nu, op=op,
                f=fv[None, :] * (1.0 + pert)[:, None], pulse=pulse, t=t0 + dt * np.arange(steps))


def _scan(case, seed):
    """The runs of a sweep or batch: the shapes belong to the case (so that its
    work does not depend on the seed), k, amplitude and nu to the seed."""
    n = case["runs"]
    shape = np.random.default_rng(20261203)
    nxs = [q for q in (16, 32, 64, 128, 256) if case["nx_lo"] <= q <= case["nx_hi"]]
    nvs = [q for q in (256, 512, 1024) if case["nv_lo"] <= q <= case["nv_hi"]]
    nx, nv = shape.choice(nxs, n), shape.choice(nvs, n)
    free = shape.random(n) < 0.25  # collisionless runs
    rng = np.random.default_rng([seed, 2])
    k = rng.uniform(0.25, 0.45, n)
    # weak enough that the FP32 f = g + f0 stays positive at the ends of the v grid, where f0 is 6e-9: its
    # entropy would be no number otherwise
    amp = 10.0 ** rng.uniform(-6.0, -3.3, n)
    nu = np.where(free, 0.0, 10.0 ** rng.uniform(-5.0, -2.0, n))
    return [dict(nx=int(a), nv=int(b), k=float(c), amplitude=float(d), nu=float(e))
            for a, b, c, d, e in zip(nx, nv, k, amp, nu)]


def _rows(case, seed):
    """Coarse rows [runs * nx][128] before and after a step, their collision
    feature, a training target and the network's parameters."""
    n, nx = case["runs"], case["nx"]
    rows = n * nx
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 3)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=torch.float32)  # noqa: E731
    v = torch.as_tensor(_v_axis(128, VMAX)[1], dtype=torch.float32, device="cuda")
    bell = torch.exp(-0.5 * v * v)
    amp = 10.0 ** (-4.0 + 2.0 * torch.rand((n, 1, 1), generator=gen, device="cuda"))
    phase = 6.2831853 * torch.arange(nx, device="cuda", dtype=torch.float32)[None, :, None] / nx
    kick = 4.0 + 20.0 * torch.rand((n, 1, 1), generator=gen, device="cuda")
    prev = amp * bell * (torch.cos(phase) + 0.4 * torch.cos(phase + kick * v) + 0.02 * rnd(n, nx, 128))
    g = amp * bell * (torch.cos(phase + 0.05 * v) + 0.4 * torch.cos(phase + kick * v + 0.05 * v)
                      + 0.02 * rnd(n, nx, 128))
    target = g + 0.03 * amp * bell * rnd(n, nx, 128)
    nu = 10.0 ** (-5.0 + 3.0 * torch.rand((n, 1), generator=gen, device="cuda", dtype=torch.float64))
    feat = (torch.log10(1.0 + nu / 1e-5) / 3.0).expand(n, nx).reshape(rows).float().contiguous()
    flat = lambda a: a.reshape(rows, 128).contiguous()  # noqa: E731
    rng = np.random.default_rng([seed, 3])
    shapes = [((64, 16, 5), 20), ((64,), 20), ((64, 64, 5), 320), ((64,), 320), ((64, 64, 5), 320), ((64,), 320),
              ((1, 64, 5), 320), ((1,), 320)]
    parts = []
    for q, (shape, fan) in enumerate(shapes):
        w = rng.uniform(-1.0, 1.0, shape) / math.sqrt(fan)
        if q == 0:
            w[:, 4:, :] = 0.0  # the network uses four input channels
        parts.append(w.reshape(-1))
    return flat(g), flat(prev), flat(target), feat, np.concatenate(parts).astype(np.float32)


TAU, PROTECT = 0.05, 56
_side = []


def _stream():
    """The one side stream of this program: the graph-replaying calls need a stream of their own."""
    if not _side:
        _side.append(torch.cuda.Stream())
    return _side[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loop":
        return _prepare_loop(case, seed)
    if kind == "plan":
        return _prepare_plan(case, seed)
    if kind == "sweep":
        from vlapy_gb300.sweep import Sweep
        sw = Sweep(_scan(case, seed), vmax=VMAX, dt=DT, collision="dg")
        sw.reset()
        eh, sh = sw.history(case["steps"])
        torch.cuda.synchronize()
        return dict(case=case, sweep=sw, eh=eh, sh=sh)
    if kind == "batch":
        from vlapy_gb300.batch import Batch64
        b = Batch64(_scan(case, seed), vmax=VMAX, dt=DT, collision="dg")
        f, e = b.initial_state()
        eh, sh = b.history(case["steps"])
        torch.cuda.synchronize()
        return dict(case=case, batch=b, f=f, e=e, eh=eh, sh=sh)
    from vlapy_gb300.corrector import Corrector
    g, prev, target, feat, params = _rows(case, seed)
    corr = Corrector(g.shape[0], params=params, vmax=VMAX, tau=TAU, protect_modes=PROTECT)
    return dict(case=case, corr=corr, g=g, prev=prev, target=target, feat=feat, out=torch.empty_like(g))


def _params(case, w):
    return {"nu": w["nu"], "fokker-planck": {"type": w["op"] if w["op"] != "none" else "lb",
                                             "solver": "batched_tridiagonal"},
            "vlasov-poisson": {"time": case["time"], "vdfdx": case["x_step"], "edfdv": case["v_step"],
                               "poisson": "spectral"},
            "backend": {"core": "gb300", "precision": case["precision"]}}


def _prepare_loop(case, seed):
    from vlapy_gb300 import field_driver, outer_loop
    from vlapy_gb300.core import step
    w = _single(case, seed)
    nx, nv = w["nx"], w["nv"]
    drv = field_driver.get_driver_function(w["x"], {"p": w["pulse"]} if w["pulse"] else {})
    d_host = field_driver.make_driver_array(drv, w["x"], w["t"])
    rules = {"time": "first-last", "space": ["k0", "k1"]}
    stuff = {"nx": nx, "nv": nv, "x": w["x"], "v": w["v"], "kx": w["kx"], "kv": w["kv"], "one_over_kx": w["inv"],
             "dv": w["dv"], "dt": w["dt"], "nu": w["nu"], "driver_function": drv, "rules_to_store_f": rules,
             "f": w["f"], "e": np.zeros(nx)}
    params = _params(case, w)
    state = dict(case=case, t=w["t"], d=d_host)
    if case["per_step"]:
        state["step"] = step.get_timestep(params, stuff)
        sc = outer_loop.get_arrays_for_inner_loop(stuff, case["steps"], rules)
        sc["time_batch"] = torch.as_tensor(w["t"], device="cuda")
        sc["driver_array_batch"] = torch.as_tensor(d_host, device="cuda")
        state["sc"] = sc
    else:
        state["sc"], state["inner"] = outer_loop.get_sim_config_and_inner_loop_step(params, stuff, case["steps"], rules)
    return state


def _prepare_plan(case, seed):
    from vlapy_gb300.plan import Plan, history_struct
    w = _single(case, seed)
    nx, nv, nt = w["nx"], w["nv"], case["steps"]
    fp32 = case["precision"] != "fp64"
    bg = w["f"].mean(axis=0) if fp32 else None
    plan = Plan(nx, nv, w["x"], w["v"], w["kx"], w["kv"], w["inv"], w["dx"], w["dv"], dt=w["dt"], nu=w["nu"],
                collision=w["op"], precision=case["precision"], f_background=bg)
    dev = torch.device("cuda")
    f = torch.as_tensor((w["f"] - bg[None, :]).astype(np.float32) if fp32 else w["f"], device=dev).contiguous()
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
    storage = {"stored_f": torch.zeros((nt, 2, nv), dtype=torch.complex64, device=dev),
               "fields": {q: z(nt, nx) for q in FIELDS}, "series": {q: z(nt) for q in SERIES}}
    state = dict(case=case, plan=plan, f=f, e=z(nx), storage=storage, hist=history_struct(storage, nx, 2),
                 tb=torch.as_tensor(w["t"], device=dev), db=z(nt, nx))
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _stored(f, e, sc, single):
    out = {"f": f, "e": e, "stored_f": sc["stored_f"], "fields": {q: sc["fields"][q] for q in FIELDS},
           "series": {q: sc["series"][q] for q in SERIES}}
    if single:  # an FP32 mode: its float64 buffers hold FP32 results
        low = lambda a: a.float() if a.dtype == torch.float64 else a  # noqa: E731
        out = {q: ({p: low(b) for p, b in a.items()} if isinstance(a, dict) else low(a)) for q, a in out.items()}
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loop":
        if case["per_step"]:
            sc = state["sc"]
            for i in range(case["steps"]):
                sc, _ = state["step"](sc, i)
        else:
            sc = state["inner"](state["t"], state["d"], state["sc"])
        state["sc"] = sc
        return _stored(sc["f"], sc["e"], sc, case["precision"] != "fp64")
    if kind in ("plan", "sweep", "batch"):
        stream = _stream()
        with torch.cuda.stream(stream):
            if kind == "plan":
                state["plan"].run_steps(state["f"], state["e"], state["hist"], state["tb"], state["db"], 0,
                                        case["steps"], use_graph=True, stream=stream)
                return _stored(state["f"], state["e"], state["storage"], case["precision"] != "fp64")
            if kind == "sweep":
                state["sweep"].run_steps(case["steps"], state["eh"], state["sh"], use_graph=True, stream=stream)
                return {"g": state["sweep"].state_view(), "e": state["eh"].float(), "series": state["sh"].float()}
            state["batch"].run_steps(state["f"], state["e"], case["steps"], state["eh"], state["sh"], use_graph=True,
                                     stream=stream)
            return {"f": state["f"], "e": state["e"], "e_hist": state["eh"], "series": state["sh"]}
    corr, nx = state["corr"], case["nx"]
    if kind == "apply":
        return corr.apply(state["g"], state["prev"], state["feat"], out=state["out"], group_rows=nx)
    loss, grad = corr.gradients(state["g"], state["target"], state["prev"], state["feat"], group_rows=nx)
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _step_flops(nx, nv, op, time):
    """One time step: forward and inverse transforms with a phase per cell
    (two real lines share a complex transform), the elimination of the
    collision step and the moments."""
    cells = nx * nv
    fft_v, fft_x = 5.0 * math.log2(nv) + 6.0, 5.0 * math.log2(nx) + 6.0
    kicks, drifts = {"leapfrog": (2, 1), "pefrl": (4, 5), "h-sixth": (6, 5)}[time]
    return cells * (kicks * fft_v + drifts * fft_x + (20.0 if op != "none" else 0.0) + 20.0 + 2.0 * drifts)


def work(case):
    kind = case["kind"]
    if kind in ("loop", "plan"):
        nx, nv, n = case["nx"], case["nv"], case["steps"]
        size = 8 if case["precision"] == "fp64" else 4
        held = 8 if kind == "loop" else size  # what the caller's f is held in
        return {"bytes": 2.0 * held * nx * nv + n * (8.0 * 10 * nx + 2 * 8.0 * nv),
                "flops": n * _step_flops(nx, nv, case.get("op", "dg"), case.get("time", "leapfrog"))}
    if kind in ("sweep", "batch"):
        size = 4 if kind == "sweep" else 8
        bytes_, flops = 0.0, 0.0
        for r in _scan(case, 0):
            bytes_ += 2.0 * size * r["nx"] * r["nv"] + case["steps"] * 8.0 * (r["nx"] + 7)
            flops += case["steps"] * _step_flops(r["nx"], r["nv"], "dg" if r["nu"] > 0 else "none", "leapfrog")
        return {"bytes": bytes_, "flops": flops}
    rows = case["runs"] * case["nx"]
    net = 2.0 * rows * 128 * 5 * (4 * 64 + 64 * 64 + 64 * 64 + 64)
    if kind == "apply":
        return {"bytes": rows * (3.0 * 512 + 4), "flops": net}
    return {"bytes": rows * (3.0 * 512 + 4) + 4.0 * 46593, "flops": 3.0 * net}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

class _Runs64:
    """A set of runs of one shape, f[B][nx][nv] in float64 on the GPU, with the
    reference's operators written in plain torch."""

    def __init__(self, f, x, kx, inv, v, kv, dv, dt, nu, op, x_step="exponential", v_step="exponential", pulse=None):
        t = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")  # noqa: E731
        self.f = f
        self.nb, self.nx, self.nv = f.shape
        self.x, self.kx, self.inv = t(x), t(kx), t(inv)  # [B][nx]
        self.v, self.kv, self.dv, self.dt = t(v), t(kv), float(dv), float(dt)
        self.nu, self.op = t(nu), op  # [B]
        self.x_step, self.v_step, self.pulse = x_step, v_step, pulse
        self.e = torch.zeros((self.nb, self.nx), dtype=torch.float64, device="cuda")

    def kick(self, dt):
        f, e = self.f, self.e
        if self.v_step == "exponential":
            ph = torch.exp(-1j * (self.kv * dt)[None, None, :] * e[:, :, None])
            self.f = torch.fft.ifft(torch.fft.fft(f, dim=2) * ph, dim=2).real
        elif self.v_step == "cd2":
            g = torch.gradient(f, spacing=self.dv, dim=2, edge_order=2)[0]
            self.f = f - (e[:, :, None] * g) * dt
        else:
            self.f = _spline_shift(f[0], self.v, self.v[None, :] - e[0][:, None] * dt)[None]

    def drift(self, dt):
        if self.x_step == "exponential":
            for b in range(0, self.nb, 256):
                ph = torch.exp(-1j * (self.kx[b:b + 256] * dt)[:, :, None] * self.v[None, None, :])
                self.f[b:b + 256] = torch.fft.ifft(torch.fft.fft(self.f[b:b + 256], dim=1) * ph, dim=1).real
        else:
            lines = self.f[0].T.contiguous()
            self.f = _spline_shift(lines, self.x[0], self.x[0][None, :] - self.v[:, None] * dt).T.contiguous()[None]

    def field(self, time):
        n = _trapz(self.f, self.dv)
        self.e = torch.fft.ifft(1j * self.inv * torch.fft.fft(1.0 - n, dim=1), dim=1).real + self.driver(time)

    def driver(self, time):
        p = self.pulse
        if p is None or time < 0.0 or time > p["t_R"]:
            return 0.0
        env = p["a0"] * math.sin(math.pi * time / p["t_R"]) ** 2
        return env * torch.sin(p["k0"] * self.x - p["w0"] * time)

    def collide(self):
        if self.op == "none":
            return
        f = self.f.reshape(-1, self.nv)
        nudt = (self.nu * self.dt)[:, None].expand(self.nb, self.nx).reshape(-1)
        v = self.v
        dg = self.op == "dg"
        vbar = _trapz(f * v, self.dv) if dg else torch.zeros_like(nudt)
        vth = _trapz(f * (v - vbar[:, None]) ** 2, self.dv)
        a0 = vth / self.dv ** 2
        drift = ((v[:, None] - vbar[None, :]) if dg else v[:, None].expand(-1, f.shape[0])) * 0.5 / self.dv
        b = 1.0 + nudt * 2.0 * a0
        low, up = nudt * (-a0 + drift[:-1]), nudt * (-a0 - drift[1:])  # of rows j + 1 and j
        d = f.T.contiguous()
        piv = torch.empty_like(d)
        piv[0] = b
        for j in range(1, self.nv):
            m = low[j - 1] / piv[j - 1]
            piv[j] = b - m * up[j - 1]
            d[j] -= m * d[j - 1]
        d[-1] /= piv[-1]
        for j in range(self.nv - 2, -1, -1):
            d[j] = (d[j] - up[j] * d[j + 1]) / piv[j]
        self.f = torch.where((nudt > 0)[:, None], d.T, f).reshape(self.f.shape).contiguous()

    def step(self, t, time):
        dt = self.dt
        if time == "leapfrog":
            self.kick(0.5 * dt)
            self.drift(dt)
            self.field(t + dt)
            self.kick(0.5 * dt)
        elif time == "pefrl":
            xsi, lam, chi = 0.1786178958448091, -0.2123418310626054, -0.6626458266981849e-1
            xs = [xsi, chi, 1.0 - 2.0 * (chi + xsi), chi, xsi]
            ks = [0.5 * (1.0 - 2.0 * lam), lam, lam, 0.5 * (1.0 - 2.0 * lam)]
            at = t
            for q in range(5):
                self.drift(xs[q] * dt)
                at += xs[q] * dt
                self.field(at)
                if q < 4:
                    self.kick(ks[q] * dt)
        else:
            a1, a2, a3 = 0.168735950563437422448196, 0.377851589220928303880766, -0.093175079568731452657924
            b1, b2, b3 = 0.049086460976116245491441, 0.264177609888976700200146, 0.186735929134907054308413
            c1, c2, c3 = -0.000069728715055305084099, -0.000625704827430047189169, -0.002213085124045325561636
            d2, d3, e3 = -2.916600457689847816445691e-6, 3.048480261700038788680723e-5, 4.985549387875068121593988e-7
            k1 = b1 + 2.0 * c1 * dt ** 2
            k2 = b2 + 2.0 * c2 * dt ** 2 + 4.0 * d2 * dt ** 4
            k3 = b3 + 2.0 * c3 * dt ** 2 + 4.0 * d3 * dt ** 4 - 8.0 * e3 * dt ** 6
            self.kick(k1 * dt)
            for a, kk in ((a1, k2), (a2, k3), (a3, k3), (a2, k2), (a1, k1)):
                self.drift(a * dt)
                self.field(t + a * dt)
                self.kick(kk * dt)
        self.collide()

    def moments(self):
        """n, j, T, q, the 4th and 5th moments, trapz f^2 and trapz f log f, each [B][nx]."""
        f, v = self.f, self.v
        return [_trapz(f * v ** p, self.dv) for p in range(6)] + [_trapz(f * f, self.dv),
                                                                  _trapz(f * torch.log(f), self.dv)]


def _spline_shift(y, g, at):
    """The not-a-knot cubic spline of every line y[L][N] over the grid g
    extended by one periodic cell at each end, at the points at[L][N]
    (clamped to the extended grid)."""
    n = y.shape[1]
    h = float(g[2] - g[1])
    p = torch.cat([y[:, -1:], y, y[:, :1]], dim=1)
    r = (p[:, :-2] - 2.0 * p[:, 1:-1] + p[:, 2:]) * (6.0 / h ** 2)  # equations of the nodes 1 .. n
    a = 4.0 * torch.eye(n, dtype=torch.float64, device=y.device)
    a += torch.diag(torch.ones(n - 1, dtype=torch.float64, device=y.device), 1)
    a += torch.diag(torch.ones(n - 1, dtype=torch.float64, device=y.device), -1)
    a[0, 0] = a[-1, -1] = 6.0  # not-a-knot: 2 M_1 = M_0 + M_2 and its mirror
    a[0, 1] = a[-1, -2] = 0.0
    m = torch.linalg.solve(a, r.T).T
    m = torch.cat([2.0 * m[:, :1] - m[:, 1:2], m, 2.0 * m[:, -1:] - m[:, -2:-1]], dim=1)
    lo = float(g[0]) - h
    u = (at.clamp(lo, float(g[-1]) + h) - lo) / h
    k = u.floor().clamp(0, n).long()
    t = u - k
    s = 1.0 - t
    pick = lambda q, i: torch.gather(q, 1, i)  # noqa: E731
    return (s * pick(p, k) + t * pick(p, k + 1)
            + h * h / 6.0 * ((s ** 3 - s) * pick(m, k) + (t ** 3 - t) * pick(m, k + 1)))


def _exact_single(case, seed):
    w = _single(case, seed)
    r = _Runs64(torch.as_tensor(w["f"], device="cuda")[None].clone(), w["x"][None], w["kx"][None], w["inv"][None],
                w["v"], w["kv"], w["dv"], w["dt"], [w["nu"]], w["op"], case.get("x_step", "exponential"),
                case.get("v_step", "exponential"), w["pulse"])
    nt, nx, nv = case["steps"], w["nx"], w["nv"]
    fields = {q: torch.zeros((nt, nx), dtype=torch.float64, device="cuda") for q in FIELDS}
    series = {q: torch.zeros(nt, dtype=torch.float64, device="cuda") for q in SERIES}
    stored = torch.zeros((nt, 2, nv), dtype=torch.complex128, device="cuda")
    for i in range(nt):
        r.step(float(w["t"][i]), case.get("time", "leapfrog"))
        de = r.driver(float(w["t"][i]))
        de = de[0] if isinstance(de, torch.Tensor) else torch.zeros(nx, dtype=torch.float64, device="cuda")
        mom = [m[0] for m in r.moments()]
        for q, val in zip(FIELDS, [r.e[0], de] + mom[:6]):
            fields[q][i] = val
        for q, val in zip(SERIES, mom[:3] + [r.e[0] ** 2, de ** 2] + mom[6:]):
            series[q][i] = val.mean()
        stored[i] = torch.fft.fft(r.f[0], dim=0)[:2]
    f = r.f[0]
    if case["kind"] == "plan" and case["precision"] != "fp64":
        f = f - torch.as_tensor(w["f"].mean(axis=0), device="cuda")[None, :]
    return {"f": f, "e": r.e[0], "stored_f": stored, "fields": fields, "series": series}


def _exact_scan(case, seed):
    runs = _scan(case, seed)
    batch = case["kind"] == "batch"
    n, steps = len(runs), case["steps"]
    order = sorted(range(n), key=lambda i: (runs[i]["nv"], i)) if batch else list(range(n))
    x_at, f_at, at, cell = {}, {}, 0, 0
    for i in order:
        x_at[i], f_at[i] = at, cell
        at += runs[i]["nx"]
        cell += runs[i]["nx"] * runs[i]["nv"]
    slot = {i: s for s, i in enumerate(order)}
    state = torch.zeros(cell, dtype=torch.float64, device="cuda")
    eh = torch.zeros((steps, at), dtype=torch.float64, device="cuda")
    sh = torch.zeros((steps, n, 7), dtype=torch.float64, device="cuda")
    for nx, nv in sorted({(r["nx"], r["nv"]) for r in runs}):
        ids = [i for i in range(n) if (runs[i]["nx"], runs[i]["nv"]) == (nx, nv)]
        dv, v, kv = _v_axis(nv, VMAX)
        m = np.exp(-(v ** 2) / 2.0)
        m = m / _trapz(m, dv)
        ax = [_x_axis(nx, runs[i]["k"]) for i in ids]
        pert = np.stack([1.0 + runs[i]["amplitude"] * np.cos(runs[i]["k"] * a[1]) for i, a in zip(ids, ax)])
        f = torch.as_tensor(pert, device="cuda")[:, :, None] * torch.as_tensor(m, device="cuda")[None, None, :]
        r = _Runs64(f, np.stack([a[1] for a in ax]), np.stack([a[2] for a in ax]), np.stack([a[3] for a in ax]), v, kv,
                    dv, DT, [runs[i]["nu"] for i in ids], "dg")
        xi = (torch.tensor([x_at[i] for i in ids], device="cuda")[:, None] + torch.arange(nx, device="cuda")).reshape(-1)
        si = torch.tensor([slot[i] for i in ids], device="cuda")
        for s in range(steps):
            r.step(s * DT, "leapfrog")
            mom = r.moments()
            eh[s, xi] = r.e.reshape(-1)
            for q, val in enumerate(mom[:3] + [r.e ** 2, None] + mom[6:]):
                if val is not None:
                    sh[s, si, q] = val.mean(dim=1)
        fi = torch.tensor([f_at[i] for i in ids], device="cuda")[:, None] + torch.arange(nx * nv, device="cuda")
        held = r.f.reshape(len(ids), -1)
        state[fi] = held if batch else held - torch.as_tensor(np.tile(m, nx), device="cuda")[None, :]
    if batch:
        return {"f": state, "e": eh[-1].clone(), "e_hist": eh, "series": sh}
    return {"g": state, "e": eh, "series": sh}


def _exact_rows(case, seed):
    g, prev, target, feat, params = _rows(case, seed)
    n, nx = case["runs"], case["nx"]
    dev = lambda a: (a.double().view(n, nx, 128) - a.double().view(n, nx, 128).mean(1, keepdim=True))  # noqa: E731
    d, dp = dev(g).reshape(-1, 128), dev(prev).reshape(-1, 128)
    mean = g.double() - d
    sizes = [(64, 16, 5), (64,), (64, 64, 5), (64,), (64, 64, 5), (64,), (1, 64, 5), (1,)]
    p, at = [], 0
    for s in sizes:
        q = int(np.prod(s))
        p.append(torch.as_tensor(params[at:at + q].astype(np.float64), device="cuda").view(s))
        at += q
    v = torch.as_tensor(_v_axis(128, VMAX)[1], device="cuda") / VMAX
    out = torch.empty_like(d)
    lost = 0.0
    mode = torch.fft.fftfreq(128, 1.0 / 128, device="cuda").abs()
    high = lambda a: torch.fft.ifft(torch.fft.fft(a, dim=1) * (mode >= PROTECT), dim=1).real  # noqa: E731
    for b in range(0, d.shape[0], 8192):
        x, y = d[b:b + 8192], dp[b:b + 8192]
        s = x.square().mean(1, keepdim=True).sqrt()
        ch = torch.stack([x / s, v[None, :].expand_as(x), feat[b:b + 8192].double()[:, None].expand_as(x), y / s], 1)
        h = torch.relu(torch.nn.functional.conv1d(ch, p[0][:, :4], p[1], padding=2))
        h = torch.relu(torch.nn.functional.conv1d(h, p[2], p[3], padding=2))
        h = torch.relu(torch.nn.functional.conv1d(h, p[4], p[5], padding=2))
        net = torch.nn.functional.conv1d(h, p[6], p[7], padding=2)[:, 0]
        if case["kind"] == "train":
            want = (dev(target).reshape(-1, 128)[b:b + 8192] - x) / (s * TAU)
            lost += float(high(net - want).square().sum())
            continue
        c = high(s * TAU * net)
        pd = high(x)
        nrm = lambda a: a.square().sum(1, keepdim=True).sqrt()  # noqa: E731
        cap = torch.clamp(nrm(pd) / nrm(pd + c), max=1.0)
        out[b:b + 8192] = mean[b:b + 8192] + (x - pd) + (pd + c) * cap
    if case["kind"] == "apply":
        return out
    # the gradients pass through BF16 activations: 64-bit gradients of the same network say nothing about them
    return {"loss": lost / d.numel(), "grad": None}


def exact(case, seed):
    if case["kind"] in ("loop", "plan"):
        return _exact_single(case, seed)
    if case["kind"] in ("sweep", "batch"):
        return _exact_scan(case, seed)
    return _exact_rows(case, seed)
