"""The fixed-point transforms of the FP64 advection against extended-precision
FFTs, at every power of two they take, on the inputs that choose their branches:
smooth lines (fixed point), noise and spikes (long ones go through doubles), an
odd number of lines, a last column without a partner, columns that are not
16-byte aligned, lines of zeros, extreme scales, NaN and infinity, and a
wavenumber grid that is not uniform.

Bound: the transform in doubles errs by about 1e-16 (1 + log2(N) / 5) of a line's
RMS; twice that, plus the rounding of the phases ((-k) dt) c (two products and
k's own rounding: 3 x 2^-53 of the largest phase)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def plan(nx, nv, kv=None):
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv0 = vo.velocity_axis(6.4, nv)
    kv = kv0 if kv is None else kv
    return Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1), x, v, kx, kv


def advected(f, k, c, dt, axis):
    """Re IFFT(exp(-i k dt c) FFT f) along axis in extended precision, and the bound of the line errors."""
    import scipy.fft as sf
    ph = -(k.astype(LD) * LD(dt))
    th = ph[None, :] * c.astype(LD)[:, None] if axis == 1 else ph[:, None] * c.astype(LD)[None, :]
    out = sf.ifft(sf.fft(f.astype(LD), axis=axis) * (np.cos(th) + 1j * np.sin(th)), axis=axis).real
    n = f.shape[axis]
    rms = np.sqrt(np.mean(f.astype(LD) ** 2, axis=axis))
    eps = 2e-16 * (1 + 0.2 * np.log2(n)) + 3.4e-16 * np.abs(th).max(axis=axis)
    return out, np.asarray(eps * rms, dtype=np.float64)


def lines(kind, n, count, rng, axis_grid):
    if kind == "smooth":
        g = np.exp(-axis_grid ** 2 / 2.0)[None, :] * (1.0 + 0.3 * rng.standard_normal((count, 1)))
    elif kind == "noise":
        g = rng.standard_normal((count, n))
    elif kind == "spike":
        g = np.zeros((count, n))
        g[np.arange(count), rng.integers(0, n, count)] = rng.uniform(0.1, 1.0, count)
    else:  # zeros beside smooth lines, and scales far apart
        g = np.exp(-axis_grid ** 2 / 2.0)[None, :] * 10.0 ** rng.integers(-280, 280, (count, 1)).astype(float)
        g[1] = 0.0
    return g


@pytest.mark.parametrize("kind", ["smooth", "noise", "spike", "scales"])
@pytest.mark.parametrize("n", [2 ** q for q in range(1, 14)])
def test_edfdv_against_extended_precision(n, kind):
    rng = np.random.default_rng(n)
    nx = 7  # an odd row
    p, x, v, kx, kv = plan(nx, n)
    f = lines(kind, n, nx, rng, v)
    e = 0.05 * rng.standard_normal(nx)
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    err = np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=1)).astype(np.float64)
    assert (err <= bound).all(), (err / np.where(bound > 0, bound, 1)).max()


@pytest.mark.parametrize("kind", ["smooth", "noise", "spike", "scales"])
@pytest.mark.parametrize("nx,nv,shift", [(2 ** q, 8, 0) for q in range(1, 14)] + [(64, 37, 0), (64, 300, 0), (64, 300, 1),
                                                                              (2048, 5, 0), (4096, 3, 1)])
def test_vdfdx_against_extended_precision(nx, nv, shift, kind):
    rng = np.random.default_rng(nx + nv)
    p, x, v, kx, kv = plan(nx, nv)
    f = lines(kind, nx, nv, rng, np.linspace(-6, 6, nx)).T
    # a buffer that starts 8 bytes past a 16-byte boundary when shift is 1
    buf = torch.zeros(nx * nv + shift, dtype=torch.float64, device="cuda")
    g = buf[shift:].view(nx, nv)
    g.copy_(torch.as_tensor(f, device="cuda"))
    p.vdfdx(g, 0.1)
    ref, bound = advected(f, kx, v, 0.1, 0)
    err = np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=0)).astype(np.float64)
    assert (err <= bound).all(), (err / np.where(bound > 0, bound, 1)).max()
    if shift:
        assert float(buf[0]) == 0.0


@pytest.mark.parametrize("n", [16, 1024, 4096])
def test_non_finite_lines(n):
    """A line with a NaN or infinity comes out as NaN, the others of its launch as without it."""
    p, x, v, kx, kv = plan(8, n)
    f = np.exp(-v ** 2 / 2.0)[None, :] * np.arange(1.0, 9.0)[:, None]
    e = torch.as_tensor(np.linspace(-0.1, 0.1, 8), device="cuda")
    clean = torch.as_tensor(f, device="cuda")
    p.edfdv(clean, e, 0.05)
    f[2, n // 3], f[5, 0] = np.nan, np.inf
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, e, 0.05)
    bad = torch.isnan(g)
    assert bad[2].all() and bad[5].all()
    keep = [0, 1, 6, 7]
    assert torch.equal(g[keep], clean[keep])


def test_grid_that_is_not_uniform():
    """Any wavenumber array is taken: one that is not k[1] times the index goes through doubles."""
    rng = np.random.default_rng(3)
    dv, v, kv = vo.velocity_axis(6.4, 256)
    kv = kv * (1.0 + 1e-3 * rng.standard_normal(256))
    kv[129:] = -kv[127:0:-1]
    p, x, v, kx, kv = plan(6, 256, kv)
    f = lines("smooth", 256, 6, rng, v)
    e = 0.05 * rng.standard_normal(6)
    g = torch.as_tensor(f, device="cuda")
    p.edfdv(g, torch.as_tensor(e, device="cuda"), 0.05)
    ref, bound = advected(f, kv, e, 0.05, 1)
    assert (np.sqrt(np.mean((g.cpu().numpy() - ref) ** 2, axis=1)) <= bound).all()
