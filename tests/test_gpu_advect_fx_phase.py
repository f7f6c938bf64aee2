"""The phases of the fixed-point advection: they step along the wavenumber grid, and a
step's own rounding taken m times must not add to what the doubles ((-k) dt) c carry.
Columns with all wavenumbers in them, over a drift of many cells, against extended
precision; the bound is the error of those doubles in an otherwise exact transform,
plus that of a transform in doubles, 1e-16 (1 + log2(N) / 5)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_gpu_advect_fx import LD, advected, plan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["noise", "spike"])
@pytest.mark.parametrize("nx", [512, 1000, 1024, 2047, 2048])
def test_phase_of_high_wavenumbers(nx, kind):
    import scipy.fft as sf
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(nx)
    nv, dt = 24, 0.1
    p, x, v, kx, kv = plan(nx, nv)
    f = rng.random((nx, nv))
    if kind == "spike":
        f = 1e-12 * f
        f[rng.integers(0, nx, nv), np.arange(nv)] = 1.0
    g = torch.as_tensor(f, device="cuda")
    p.vdfdx(g, dt)
    ref, _ = advected(f, kx, v, dt, 0)
    th = ((-kx * dt)[:, None] * v[None, :]).astype(LD)  # as doubles round it
    doubles = sf.ifft(sf.fft(f.astype(LD), axis=0) * (np.cos(th) + 1j * np.sin(th)), axis=0).real

    def err(a):
        rel = np.sqrt(np.mean((a - ref) ** 2, axis=0) / np.mean(ref ** 2, axis=0))
        return float(np.sqrt(np.mean(rel ** 2)))

    got = err(g.cpu().numpy().astype(LD))
    assert got <= err(doubles) + 1e-16 * (1.0 + 0.2 * np.log2(nx)), (got, err(doubles))
