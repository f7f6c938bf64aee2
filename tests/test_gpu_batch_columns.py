"""A run of an FP64 batch against the same run by a single plan, bit for bit, where the
x-drift could make a column depend on what else is advanced with it: a spiked column
(transformed in doubles) in tiles whose width follows the number of columns of all
runs, and a run whose wavenumbers are not a uniform grid beside one whose are."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from vlapy_gb300 import initializers as I  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _single(r, f, kx=None, vmax=6.4, dt=0.1):
    from vlapy_gb300.plan import Plan
    dx, x, kx0, inv = I.initialize_spatial_quantities(0.0, 2.0 * np.pi / r["k"], r["nx"])
    dv, v, kv = I.initialize_velocity_quantities(vmax, r["nv"])
    p = Plan(r["nx"], r["nv"], x, v, kx0 if kx is None else kx, kv, inv, dx, dv, dt=dt, nu=r["nu"],
             collision="dg" if r["nu"] > 0 else "none")
    g, e = f.clone(), torch.zeros(r["nx"], dtype=torch.float64, device="cuda")
    p.run_steps(g, e, None, torch.zeros(1, dtype=torch.float64, device="cuda"), None, 0, 1)
    return g, e


@pytest.mark.parametrize("nx,nv,n", [(1024, 256, 8), (1024, 64, 24), (512, 128, 24), (256, 128, 40)])
def test_spiked_column(nx, nv, n):
    from vlapy_gb300.batch import Batch64
    runs = [dict(nx=nx, nv=nv, k=0.3 + 0.005 * i, amplitude=1e-3, nu=0.0) for i in range(n)]
    b = Batch64(runs)
    f, e = b.initial_state()
    for i in range(n):
        g = b.f_of(f, i)
        for c in (3, nv // 2, nv - 6):
            g[:, c] *= 1e-12
            g[nx // 3 + i, c] = 0.4
    f0 = f.clone()
    b.run_steps(f, e, 1)
    for i in range(n):
        pf, pe = _single(runs[i], b.f_of(f0, i).clone())
        assert torch.equal(b.f_of(f, i), pf) and torch.equal(b.e_of(e, i), pe), i


def test_run_with_its_own_wavenumbers(monkeypatch):
    from vlapy_gb300 import batch
    runs = [dict(nx=64, nv=128, k=0.3, amplitude=1e-2, nu=0.0), dict(nx=64, nv=128, k=0.4, amplitude=1e-2, nu=1e-3)]
    make = I.initialize_spatial_quantities
    own = make(0.0, 2.0 * np.pi / 0.4, 64)[2].copy()
    own[1:32] *= 1.0 + 1e-3 * np.random.default_rng(1).standard_normal(31)
    own[33:] = -own[31:0:-1]

    def quantities(x0, x1, nx):
        dx, x, kx, inv = make(x0, x1, nx)
        return (dx, x, own, inv) if abs(x1 - 2.0 * np.pi / 0.4) < 1e-12 else (dx, x, kx, inv)

    monkeypatch.setattr(batch.initializers, "initialize_spatial_quantities", quantities)
    b = batch.Batch64(runs)
    monkeypatch.undo()
    f, e = b.initial_state()
    f0 = f.clone()
    b.run_steps(f, e, 1)
    for i in range(2):
        pf, pe = _single(runs[i], b.f_of(f0, i).clone(), own if i else None)
        assert torch.equal(b.f_of(f, i), pf) and torch.equal(b.e_of(e, i), pe), i
