"""A pulse whose amplitude is no number: the field is NaN where its sine is formed and
the status word says so, in both precision modes and at every block size of the FP32
field kernel; a pulse that is silent (a sin^2 envelope outside its interval) still adds
nothing, whatever its other values are."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
NAN = float("nan")


def _run(precision, nx, pulses, t=0.0):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from vlapy_gb300.plan import Plan
    nv, k, dt = 64, 0.3, 0.1
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / k, nx)
    dv, v, kv = vo.velocity_axis(6.4, nv)
    f = vo.maxwellian(nx, nv, 6.4) * (1.0 + 1e-3 * np.cos(k * x))[:, None]
    bg = vo.maxwellian(1, nv, 6.4)[0] if precision == "fp32-deltaf" else None
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=dt, precision=precision, f_background=bg, pulses=pulses)
    s = f if bg is None else (f - bg[None, :]).astype(np.float32)
    state = torch.as_tensor(s, device="cuda")
    e = torch.zeros(nx, dtype=torch.float64, device="cuda")
    p.run_steps(state, e, None, torch.as_tensor([t], dtype=torch.float64, device="cuda"), None, 0, 1)
    return p, e.cpu().numpy()


def _pulse(**kw):
    from vlapy_gb300._lib import VG_ENV_TANH
    return dict(dict(k0=0.3, w0=1.2, a0=1e-3, t_L=5.0, t_R=20.0, t_wL=1.0, t_wR=1.0, envelope=VG_ENV_TANH), **kw)


# the field of the step from t = 0 is taken at t = 0.1
BAD = [dict(a0=NAN), dict(k0=NAN), dict(t_wL=0.0, t_L=0.1), dict(t_wR=0.0, t_R=0.1), dict(w0=NAN)]


@pytest.mark.parametrize("bad", range(len(BAD)))
@pytest.mark.parametrize("nx", [16, 1024, 2048])
@pytest.mark.parametrize("precision", ["fp64", "fp32-deltaf"])
def test_amplitude_that_is_nan_reaches_the_field(precision, nx, bad):
    from vlapy_gb300._lib import VG_ERR_NUMERIC, VlagpuError
    # beyond the first 32 pulses as well
    for n_good in (0, 33):
        p, e = _run(precision, nx, [_pulse()] * n_good + [_pulse(**BAD[bad])])
        assert np.isnan(e).all()
        with pytest.raises(VlagpuError) as err:
            p.status()
        assert err.value.status == VG_ERR_NUMERIC


@pytest.mark.parametrize("precision", ["fp64", "fp32-deltaf"])
def test_silent_pulse_adds_nothing(precision):
    from vlapy_gb300._lib import VG_ENV_SIN2
    _, e0 = _run(precision, 64, [_pulse()])
    p, e1 = _run(precision, 64, [_pulse(), _pulse(envelope=VG_ENV_SIN2, t_R=0.05, a0=NAN)])
    assert np.array_equal(e0, e1) and p.status() == 0
    # a sin^2 pulse of zero length at t = 0: 0 / 0
    p, e2 = _run(precision, 64, [_pulse(), _pulse(envelope=VG_ENV_SIN2, t_R=0.0)], t=-0.1)
    assert np.isnan(e2).all()
