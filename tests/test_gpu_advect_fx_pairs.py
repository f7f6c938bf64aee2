"""Line pairs of the FP64 advection that its fixed-point transform turns away: such
a pair is transformed in doubles, and each of its two lines has to come out as if
it were alone, whatever the scale of the other.

Bound: that of tests/test_gpu_advect_fx.py, plus one step of the subnormal grid
for the last rounding of a line that lies on it."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_advect_fx import LD, advected, plan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _within(got, ref, bound, axis):
    assert np.isfinite(got).all()
    err = np.sqrt(np.mean((got.astype(LD) - ref) ** 2, axis=axis))
    assert (err <= bound.astype(LD) + LD(5e-324)).all(), (err, bound)


@pytest.mark.parametrize("tiny", [1e-310, 4e-320, 5e-324])
@pytest.mark.parametrize("n", [2048, 4096, 8192])
def test_subnormal_line_beside_a_spike(n, tiny):
    """Row pairs (subnormal, spike) and (spike, subnormal); the spike sends them to doubles."""
    p, x, v, kx, kv = plan(4, n)
    f = np.zeros((4, n))
    f[0] = tiny * np.exp(-v ** 2 / 8.0)
    f[3] = f[0]
    f[1, n // 3] = f[2, n // 5] = 1.0
    e = np.array([0.03, -0.05, 0.05, -0.02])
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    got = g.cpu().numpy()
    for r in range(4):
        _within(got[r:r + 1], ref[r:r + 1], bound[r:r + 1], 1)


@pytest.mark.parametrize("tiny", [1e-310, 1e-307])
@pytest.mark.parametrize("nx", [2048, 4096])
def test_subnormal_columns_beside_a_spike(nx, tiny):
    """The same for columns: the spike's partner, and pairs of subnormal columns in its tile."""
    nv = 16
    p, x, v, kx, kv = plan(nx, nv)
    f = np.repeat(tiny * (1.0 + 0.5 * np.cos(0.3 * x))[:, None], nv, axis=1)
    f[:, 5] = 0.0
    f[nx // 3, 5] = 1.0
    g = torch.as_tensor(f, device="cuda")
    p.vdfdx(g, 0.1)
    ref, bound = advected(f, kx, v, 0.1, 0)
    got = g.cpu().numpy()
    for c in range(nv):
        _within(got[:, c:c + 1], ref[:, c:c + 1], bound[c:c + 1], 0)


@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e6, 1e-307, 1e290])
@pytest.mark.parametrize("n", [2048, 4096, 8192])
def test_spike_beside_a_smooth_line(n, scale):
    """A line in doubles beside one of far more of its maximum in its RMS: each errs by its own RMS only."""
    p, x, v, kx, kv = plan(4, n)
    f = np.zeros((4, n))
    f[0] = scale * np.exp(-v ** 2 / 2.0)
    f[3] = f[0]
    f[1, n // 3] = f[2, n // 5] = 1.0
    e = np.array([0.03, -0.05, 0.05, -0.02])
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    got = g.cpu().numpy()
    for r in range(4):
        _within(got[r:r + 1], ref[r:r + 1], bound[r:r + 1], 1)


@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e6, 1e-307, 1e290])
@pytest.mark.parametrize("nx", [1024, 4096, 8192])
def test_spiked_column_beside_a_smooth_one(nx, scale):
    nv = 6
    p, x, v, kx, kv = plan(nx, nv)
    f = np.repeat(scale * (1.0 + 0.5 * np.cos(0.3 * x))[:, None], nv, axis=1)
    f[:, 2:5] = 0.0
    f[nx // 3, 2] = f[nx // 7, 4] = 1.0
    g = torch.as_tensor(f, device="cuda")
    p.vdfdx(g, 0.1)
    ref, bound = advected(f, kx, v, 0.1, 0)
    got = g.cpu().numpy()
    for c in range(nv):
        _within(got[:, c:c + 1], ref[:, c:c + 1], bound[c:c + 1], 0)
