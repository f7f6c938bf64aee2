"""The Poisson solve by its Green's function against an extended-precision
transform: fewer points than warps, a last tile of points that is not full, odd
lengths, the longest length and the ones on the other side of the limit (which go
through transforms), charges far from order one, a driver, and non-finite charges.

Bound: a transform in doubles errs by about 2e-16 log2(N) of the field's largest
contribution, max|rho| sum|G|; the sum errs by G's rounding, a few 2^-53 of it."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e200])
@pytest.mark.parametrize("nx", [2, 3, 5, 7, 8, 9, 31, 32, 33, 48, 64, 100, 255, 256, 1000, 1024, 2048, 4095, 4096, 8192])
def test_poisson(nx, scale):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import scipy.fft as sf
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.0, 16)
    rng = np.random.default_rng(nx)
    rho = scale * (rng.standard_normal(nx) + np.cos(0.3 * x))
    p = Plan(nx, 16, x, v, kx, kv, inv, dx, dv, dt=0.1)
    out = torch.empty(nx, dtype=torch.float64, device="cuda")
    p.poisson(torch.as_tensor(rho, device="cuda"), out)
    ref = sf.ifft(1j * inv.astype(LD) * sf.fft(rho.astype(LD))).real
    green = np.abs(np.fft.ifft(1j * inv).real).sum()
    bound = 2.2e-16 * (1.0 + np.log2(nx)) * np.abs(rho).max() * max(green, 1e-300)
    assert (np.abs(out.cpu().numpy() - ref) <= bound).all(), np.abs(out.cpu().numpy() - ref).max() / bound


@pytest.mark.parametrize("nx", [3, 33, 64, 300])
def test_driver_and_non_finite_charge(nx):
    from vlapy_gb300._lib import VlagpuError
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.0, 32)
    p = Plan(nx, 32, x, v, kx, kv, inv, dx, dv, dt=0.1)
    f = vo.maxwellian(nx, 32, 6.0) * (1.0 + 0.1 * np.cos(0.3 * x))[:, None]
    drv = np.linspace(-1.0, 1.0, nx)
    out = torch.empty(nx, dtype=torch.float64, device="cuda")
    g = torch.as_tensor(f, device="cuda")
    p.field_solve(g, torch.as_tensor(drv, device="cuda"), out)
    n = vo.charge_density(f, dv)
    ref = drv + np.fft.ifft(1j * inv * np.fft.fft(1.0 - n)).real
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-14
    assert p.status() == 0
    g[nx // 2, 3] = float("nan")
    p.field_solve(g, None, out)
    assert torch.isnan(out).all()
    with pytest.raises(VlagpuError):
        p.status()
