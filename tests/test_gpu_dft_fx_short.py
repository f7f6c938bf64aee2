"""Lengths that are not powers of two and short enough for one launch both ways: around
the lengths where the CTA's shape changes (16, 64), odd numbers of lines, rows and
columns, with the bound of tests/test_gpu_dft_fx.py; and a call's time, which is that of
one launch (two took 12 to 14 us where the transforms in doubles had taken 8)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_advect_fx import advected, lines, plan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("kind", ["smooth", "noise", "spike", "scales"])
@pytest.mark.parametrize("n,count", [(3, 2), (6, 3), (9, 7), (14, 3), (15, 4), (17, 3), (31, 5), (33, 2), (62, 3), (63, 9),
                                     (66, 3)])
def test_rows_and_columns(n, count, kind):
    rng = np.random.default_rng(n)
    p, x, v, kx, kv = plan(count, n)
    f = lines(kind, n, count, rng, v)
    e = 0.05 * rng.standard_normal(count)
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    assert (np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=1)) <= bound).all()
    p, x, v, kx, kv = plan(n, count)
    f = lines(kind, n, count, rng, np.linspace(-6, 6, n)).T.copy()
    g = torch.as_tensor(f, device="cuda")
    p.vdfdx(g, 0.1)
    ref, bound = advected(f, kx, v, 0.1, 0)
    assert (np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=0)) <= bound).all()


def _time(fn):
    best = float("inf")
    for _ in range(6):
        b, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        b.record()
        for _ in range(200):
            fn()
        e.record()
        torch.cuda.synchronize()
        best = min(best, b.elapsed_time(e))
    return best


def test_time_of_one_launch():
    p, x, v, kx, kv = plan(64, 9)
    f = torch.rand((64, 9), dtype=torch.float64, device="cuda")
    n = torch.zeros(64, dtype=torch.float64, device="cuda")
    one, kick = _time(lambda: p.charge_density(f, n)), _time(lambda: p.edfdv(f, n, 0.05))
    assert kick <= 1.6 * one, (kick, one)
