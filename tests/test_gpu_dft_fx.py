"""The fixed-point DFTs of lengths that are not powers of two against
extended-precision FFTs: primes and composites, one bin or point past a CTA's 32,
the longest length, an odd number of lines, columns, and the inputs of the
power-of-two tests (with their bound, which a transform in doubles sets)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402
from test_gpu_advect_fx import advected, lines, plan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("kind", ["smooth", "noise", "spike", "scales"])
@pytest.mark.parametrize("n,count", [(3, 5), (5, 2), (7, 1), (30, 3), (62, 3), (63, 4), (65, 3), (97, 5), (127, 2), (720, 5),
                                     (1000, 3), (1021, 2), (2049, 3), (4095, 3)])
def test_edfdv(n, count, kind):
    rng = np.random.default_rng(n)
    nx = max(count, 2)
    p, x, v, kx, kv = plan(nx, n)
    f = lines(kind, n, nx, rng, v)
    e = 0.05 * rng.standard_normal(nx)
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    err = np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=1)).astype(np.float64)
    assert (err <= bound).all(), (err / np.where(bound > 0, bound, 1)).max()


@pytest.mark.parametrize("kind", ["smooth", "noise", "spike", "scales"])
@pytest.mark.parametrize("nx,nv", [(3, 40), (48, 720), (65, 33), (97, 5), (1000, 7), (2047, 4), (4095, 3)])
def test_vdfdx(nx, nv, kind):
    rng = np.random.default_rng(nx + nv)
    p, x, v, kx, kv = plan(nx, nv)
    f = lines(kind, nx, nv, rng, np.linspace(-6, 6, nx)).T.copy()
    g = torch.as_tensor(f, device="cuda")
    p.vdfdx(g, 0.1)
    ref, bound = advected(f, kx, v, 0.1, 0)
    err = np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=0)).astype(np.float64)
    assert (err <= bound).all(), (err / np.where(bound > 0, bound, 1)).max()


def test_non_finite_lines_and_a_grid_that_is_not_uniform():
    p, x, v, kx, kv = plan(6, 90)
    f = np.exp(-v ** 2 / 2.0)[None, :] * np.arange(1.0, 7.0)[:, None]
    e = torch.as_tensor(np.linspace(-0.1, 0.1, 6), device="cuda")
    clean = torch.as_tensor(f, device="cuda")
    p.edfdv(clean, e, 0.05)
    f[2, 30], f[5, 0] = np.nan, np.inf
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, e, 0.05)
    assert torch.isnan(g[2]).all() and torch.isnan(g[5]).all()
    assert torch.equal(g[[0, 1, 3, 4]], clean[[0, 1, 3, 4]])
    rng = np.random.default_rng(3)
    dv, v, kv = vo.velocity_axis(6.4, 90)
    kv = kv * (1.0 + 1e-3 * rng.standard_normal(90))
    kv[46:] = -kv[44:0:-1]
    p, x, v, kx, kv = plan(4, 90, kv)
    f = lines("smooth", 90, 4, rng, v)
    e = 0.05 * rng.standard_normal(4)
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    # a direct DFT in doubles: sqrt(N) roundings instead of log N
    assert (np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=1)) <= 4 * bound).all()
