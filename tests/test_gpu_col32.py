"""The FP32 x-drift at the edges of its tile shapes, against the FP64 oracle.

nx on both sides of every change of radix or CTA width (8, 16; 128, 256; 512, 1024), the
longest x axis, rows shorter than a tile, and a state that is only 4-byte aligned.  The bar
is the FP32 mode's for one operator: 2e-5 of the perturbation.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
TOL_OP = 2e-5


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("nx,nv", [(8, 64), (16, 32), (128, 16), (256, 128), (512, 32), (1024, 64), (2048, 16),
                                   (8192, 16)])
def test_col32_tiles_match_oracle(nx, nv, offset):
    from vlapy_gb300.plan import Plan
    k = 0.3
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / k, nx)
    dv, v, kv = vo.velocity_axis(6.0, nv)
    fv = np.exp(-v ** 2 / 2)
    fv /= np.trapezoid(fv, dx=dv)
    f = fv[None, :] * (1.0 + 1e-3 * (np.cos(k * x) + 0.5 * np.sin(3 * k * x)))[:, None]
    f0 = f.mean(axis=0)
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1, precision="fp32-deltaf", f_background=f0)
    buf = torch.empty(nx * nv + offset, dtype=torch.float32, device="cuda")
    g = buf[offset:].view(nx, nv)
    g.copy_(torch.as_tensor(f - f0[None, :], device="cuda"))
    p.vdfdx(g, 0.1)
    got = g.double().cpu().numpy() + f0[None, :]
    ref = vo.vdfdx_exponential(f, kx, v, 0.1)
    assert np.linalg.norm(got - ref) <= TOL_OP * np.linalg.norm(ref - f0[None, :])
