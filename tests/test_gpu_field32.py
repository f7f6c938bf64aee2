"""The FP32 plan's field solve, driver and storage at the edges of their launches.

Shapes around the rules: the field kernel adds the density partials itself (few
of them) or a launch of its own does (many, or long x axes); its CTA is wider
than the transform or as wide; the storage has one or several CTAs of rows.
Pulses: none, silent ones among live ones, and more than one batch of envelopes.
The field is compared with the FP64 plan's on the same inputs: the FP32 state follows
that to TOL_STEP of the perturbation's size (the FP32 mode's bar for a few steps), and
the field, an integral of the density over a wavelength 2 pi / k, to that / k.  The
storage of the last step is compared with sums in FP64 over the state handed back,
which is the state it was taken from: what is left is FP32 rounding, u = 2^-24 for
each of at most 32 additions in a row, each factor of a product and each rounded
constant, of the sum of absolute values.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
TOL_STEP = 5e-5
AMP = 1e-2


def pulses_of(n):
    out = []
    for i in range(n):
        if i % 3 == 1:   # over before the step, or not yet begun
            out.append(dict(k0=0.3, w0=1.1, a0=1e-2, t_L=0.0, t_R=0.5, envelope="sin2"))
        elif i % 3 == 2:
            out.append(dict(k0=0.6, w0=1.4, a0=2e-3, t_L=0.0, t_R=9.0, envelope="sin2"))
        else:
            out.append(dict(k0=0.3, w0=1.2 + 0.01 * i, a0=3e-3, t_L=1.0, t_R=8.0, t_wL=0.7, t_wR=0.9, envelope="tanh"))
    return out


def run(precision, nx, nv, pulses, f, f0, axes, nsteps):
    from vlapy_gb300 import _lib
    from vlapy_gb300.plan import Plan, history_struct
    x, v, kx, kv, inv, dx, dv = axes
    env = {"sin2": _lib.VG_ENV_SIN2, "tanh": _lib.VG_ENV_TANH}
    ps = [dict(p, envelope=env[p["envelope"]]) for p in pulses]
    fp32 = precision != "fp64"
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1, pulses=ps, precision=precision,
             f_background=f0 if fp32 else None)
    dev = torch.device("cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
    st = {"stored_f": torch.zeros((nsteps, 2, nv), dtype=torch.complex64, device=dev),
          "fields": {kk: z(nsteps, nx) for kk in vo.FIELD_KEYS}, "series": {kk: z(nsteps) for kk in vo.SERIES_KEYS}}
    g = (torch.as_tensor((f - f0[None, :]).astype(np.float32), device=dev) if fp32
         else torch.as_tensor(f.copy(), device=dev))
    e = z(nx)
    tb = torch.as_tensor(4.0 + 0.1 * np.arange(nsteps), device=dev)
    p.run_steps(g, e, history_struct(st, nx, 2), tb, None, 0, nsteps)
    torch.cuda.synchronize()
    return e.cpu().numpy(), {k: t.cpu().numpy() for k, t in {**st["fields"], **st["series"]}.items()}, \
        st["stored_f"].cpu().numpy().astype(np.complex128), g.double().cpu().numpy()


@pytest.mark.parametrize("n_pulses", [0, 3, 70])
@pytest.mark.parametrize("nx,nv", [(4, 64), (8, 8192), (64, 1024), (256, 4096), (512, 64), (1024, 2048), (2048, 128)])
def test_field_and_storage_follow_the_fp64_plan(nx, nv, n_pulses):
    k, nsteps = 0.3, 2
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / k, nx)
    dv, v, kv = vo.velocity_axis(6.0, nv)
    fv = np.exp(-v ** 2 / 2.0)
    fv /= np.trapezoid(fv, dx=dv)
    f = fv[None, :] * (1.0 + AMP * np.cos(k * x + 0.4))[:, None]
    f0 = f.mean(axis=0)
    axes = (x, v, kx, kv, inv, dx, dv)
    e64, h64, _, _ = run("fp64", nx, nv, pulses_of(n_pulses), f, f0, axes, nsteps)
    e32, h32, m32, g = run("fp32-deltaf", nx, nv, pulses_of(n_pulses), f, f0, axes, nsteps)
    pert = AMP + 0.1 * nsteps * np.abs(h64["e"]).max()
    field = TOL_STEP * (pert / k + np.abs(h64["driver"]).max())
    np.testing.assert_allclose(e32, e64, rtol=0, atol=field)
    np.testing.assert_allclose(h32["e"], h64["e"], rtol=0, atol=field)
    np.testing.assert_allclose(h32["driver"], h64["driver"], rtol=0, atol=0)

    u = 2.0 ** -24
    w = np.full(nv, dv)
    w[[0, -1]] *= 0.5
    last = lambda key: h32[key][-1]  # noqa: E731
    for p, (key, mean) in enumerate((("n", "mean_n"), ("j", "mean_j"), ("T", "mean_T"), ("q", None), ("fv4", None),
                                     ("vN", None))):
        ref = g @ (w * v ** p) + f0 @ (w * v ** p)
        bound = (40 + 2 * p) * u * (np.abs(g) @ (w * np.abs(v) ** p)) + 1e-12
        assert (np.abs(last(key) - ref) <= bound).all(), key
        if mean:
            assert abs(last(mean) - ref.mean()) <= bound.mean(), mean
    assert abs(last("mean_e2") - (h32["e"][-1] ** 2).mean()) <= 1e-12 * (h32["e"][-1] ** 2).mean()
    assert last("mean_de2") == 0.0
    full = g + f0
    assert abs(last("mean_f2") - (full ** 2 @ w).mean()) <= 44 * u * ((g ** 2 + 2 * np.abs(g) * f0) @ w).mean() + 1e-12
    with np.errstate(invalid="ignore"):
        logs = full * np.log(full)
        bound = 48 * u * ((np.abs(logs) + np.abs(full)) @ w).mean()
    np.testing.assert_allclose(last("mean_flogf"), (logs @ w).mean(), rtol=0, atol=np.nan_to_num(bound))
    # a stored mode is a sum over x, in FP32 for the rows of a CTA
    for m in range(2):
        ref = np.exp(-2j * np.pi * m * np.arange(nx) / nx) @ g + (nx * f0 if m == 0 else 0.0)
        bound = (nx + 8) * u * 1.5 * np.abs(g).sum(0) + 2 * u * np.abs(ref) + 1e-30
        assert (np.abs(m32[-1, m] - ref) <= bound).all(), m
