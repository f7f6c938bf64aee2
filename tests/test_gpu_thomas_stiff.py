"""Strong collisions in the FP64 tridiagonal solve: launches on both sides of the line
from which one thread solves a row, with rows of very different collisionality, bit for
bit the oracle's serial order, rows of collisionless runs left alone; and the time of such a solve, which must not grow with the collisionality as the
sweeps of the chunked solve do (45 ms against 1.3 at 2048 x 4096; one thread a row takes
6.8)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _plan(nx, nv, c, op):
    """nu so that c = nu dt vth / dv^2 for vth = 1."""
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.4, nv)
    nu = c * dv * dv / 0.1
    return Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1, nu=nu, collision=op), v, dv, nu


@pytest.mark.parametrize("op", ["dg", "lb"])
@pytest.mark.parametrize("nx,nv,c", [(1024, 1024, 1526.0), (2048, 512, 381.0), (8192, 128, 24.0), (12287, 90, 10.6),
                                     (257, 4096, 24000.0), (3, 4096, 4e4), (2, 8192, 4e4), (1023, 1024, 1526.0),
                                     (5000, 256, 1e6), (2048, 512, 40.0), (8192, 128, 5.0), (3, 4096, 4e3),
                                     (2048, 512, 4e3), (8192, 128, 500.0), (3, 4096, 4e5), (64, 8192, 4e5)])
def test_bit_exact(op, nx, nv, c):
    p, v, dv, nu = _plan(nx, nv, c, op)
    rng = np.random.default_rng(nx + nv)
    vth = rng.uniform(0.5, 1.6, (nx, 1))  # vth^2 spreads c by ten
    f = np.exp(-v ** 2 / (2.0 * vth ** 2)) / (vth * np.sqrt(2.0 * np.pi)) * (1.0 + 0.05 * np.cos(2.0 * v))
    g = torch.as_tensor(f, device="cuda").contiguous()
    p.collision_step(g)
    np.testing.assert_array_equal(g.cpu().numpy(), vo.collision_step(f, v, nu, 0.1, dv, op))


@pytest.mark.parametrize("nu", [1e-4, 30.0])
def test_collisionless_runs_of_a_batch(nu):
    """A class of 2^20 cells, every third run without collisions: the others as single plans (few rows: in chunks)."""
    from vlapy_gb300.batch import Batch64
    runs = [dict(nx=64, nv=1024, k=0.3, amplitude=1e-2 * (1 + i), nu=0.0 if i % 3 == 1 else nu) for i in range(16)]
    b = Batch64(runs)
    f, e = b.initial_state()
    f0 = f.clone()
    b.run_steps(f, e, 1)
    for i in (0, 1, 14, 15):
        one = Batch64([runs[i]])
        g, q = b.f_of(f0, i).reshape(-1).clone(), torch.zeros(64, dtype=torch.float64, device="cuda")
        one.run_steps(g, q, 1)
        assert torch.equal(b.f_of(f, i).reshape(-1), g), i


@pytest.mark.parametrize("nx,nv,most", [(2048, 4096, 12.0), (8192, 1024, 4.0)])
def test_time_is_bounded(nx, nv, most):
    times = []
    for c in (3.0, 1e5):
        p, v, dv, nu = _plan(nx, nv, c, "dg")
        f = torch.as_tensor(np.repeat(np.exp(-v ** 2 / 2.0)[None, :] / 2.5066, nx, axis=0), device="cuda")
        p.collision_step(f)
        torch.cuda.synchronize()
        best = float("inf")
        for _ in range(4):
            b, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            b.record()
            p.collision_step(f)
            e.record()
            torch.cuda.synchronize()
            best = min(best, b.elapsed_time(e))
        times.append(best)
    assert times[1] <= most * times[0], times
