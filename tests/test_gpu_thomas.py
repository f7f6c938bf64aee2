"""The chunked tridiagonal solve against the oracle's serial Thomas order, bit
for bit, at the sizes where its dispatch and its chunks change: rows that fit a
warp's lanes and rows over several warps, chunks of 8, 16 and 32, lengths that
leave a partial or a single-element last chunk, rows whose diagonals go through
the scratch array, the one-thread-per-row sizes on both sides, and strong
collisions (slow contraction, so many sweeps)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["dg", "lb"])
@pytest.mark.parametrize("nx,nv,nu", [
    (5, 15, 1e-2), (5, 16, 1e-2), (3, 17, 1e-2), (9, 33, 1e-2), (33, 256, 1e-3), (7, 257, 1e-3), (48, 720, 1e-3),
    (64, 1024, 1e-2), (2, 4096, 1e-4), (3, 4095, 1e-3), (3, 4097, 1e-3), (2, 8192, 1e-4), (2, 8193, 1e-4),
    (700, 600, 1e-3), (640, 1024, 1e-3), (130, 5000, 1e-4), (12287, 40, 1e-3), (12288, 40, 1e-3), (4, 512, 1.0),
    (4, 1024, 0.0)])
def test_collision_step_bit_exact(op, nx, nv, nu):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.4, nv)
    rng = np.random.default_rng(nx * 10007 + nv)
    f = vo.maxwellian(nx, nv, 6.4) * (1.0 + 0.1 * rng.standard_normal((nx, 1)) + 0.05 * np.cos(2.0 * v + rng.uniform(
        0, 6, (nx, 1))))
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1, nu=nu, collision=op)
    g = torch.as_tensor(f, device="cuda").contiguous()
    p.collision_step(g)
    np.testing.assert_array_equal(g.cpu().numpy(), vo.collision_step(f, v, nu, 0.1, dv, op))
