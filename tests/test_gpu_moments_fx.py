"""The fixed-point storage moments against extended-precision sums: every
block size and the lengths around it, long rows, subnormal and huge scales, values down to and past the
scale's last place, and rows with zeros, negative values, infinities and NaN.

Bound: a product rounds at 2^-60.5 of the row's maximum times the power's, so a
sum of n of them errs by less than n 2^-60 of max f max|v^p| dv, and by a few
2^-53 of the result (its conversion and the multiplication by dv)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
LD = np.longdouble


def trapz(y, dv):
    return LD(dv) * (y.sum(axis=1) - (y[:, 0] + y[:, -1]) / 2)


def stored(f, nv, vmax=6.0):
    from vlapy_gb300.plan import Plan, history_struct
    nx = f.shape[0]
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(vmax, nv)
    dev = torch.device("cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
    st = {"stored_f": torch.zeros((1, 1, nv), dtype=torch.complex64, device=dev),
          "fields": {k: z(1, nx) for k in vo.FIELD_KEYS}, "series": {k: z(1) for k in vo.SERIES_KEYS}}
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1)
    p.storage_step(torch.as_tensor(f, device=dev), z(nx), z(nx), history_struct(st, nx, 1), 0)
    out = [st["fields"][k][0].cpu().numpy() for k in vo.FIELD_KEYS[2:]]
    return out, {k: float(st["series"][k][0]) for k in vo.SERIES_KEYS}, dv, v


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("scale", [1.0, 1e-300, 1e280, 3e-310])
@pytest.mark.parametrize("nv", [2, 3, 31, 64, 511, 512, 1023, 1024, 4096, 8191, 8192, 8193])
def test_moments(nv, scale):
    rng = np.random.default_rng(nv)
    v0 = vo.velocity_axis(6.0, nv)[1]
    f = np.exp(-v0 ** 2 / 2.0)[None, :] * rng.uniform(0.5, 1.5, (5, nv))
    f[3] *= np.exp(-4.0 * v0 ** 2)  # down to 1e-70 of its maximum
    f *= scale
    f[f == 0.0] = 5e-324
    got, series, dv, v = stored(f, nv)
    F = f.astype(LD)
    for p in range(6):
        w = v if p == 1 else v ** p  # as NumPy forms the powers the plan holds
        ref = trapz(F * w.astype(LD)[None, :], dv)
        top = f.max(axis=1) * (np.abs(w).max() if p else 1.0)
        bound = nv * 2.0 ** -60 * top * dv + 8e-16 * np.abs(ref) + 3 * 5e-324
        bound = bound + 2e-16 * np.asarray(trapz(F * np.abs(w).astype(LD), dv), float) * (nv > 8192)
        assert (np.abs(got[p] - ref) <= bound).all(), (p, np.abs(got[p] - ref), bound)
    if scale == 1.0:
        f2, fl = trapz(F * F, dv), trapz(F * np.log(F), dv)
        size = float(trapz(np.abs(F * np.log(F)), dv).max())
        assert abs(series["mean_f2"] - float(f2.mean())) <= 1e-15 * float(f2.max()) + nv * 2.0 ** -54 * dv * f.max() ** 2
        assert abs(series["mean_flogf"] - float(fl.mean())) <= 1e-15 * size + nv * 2.0 ** -54 * dv * f.max()


@pytest.mark.parametrize("nv", [40, 1024])
def test_values_without_a_logarithm_and_non_finite_rows(nv):
    f = np.full((6, nv), 0.25)
    clean = stored(f, nv)[0]
    for bad in (0.0, -1e-30):
        g = f.copy()
        g[2, nv // 2] = bad
        got, series, dv, v = stored(g, nv)
        assert np.isnan(series["mean_flogf"]) and np.isfinite(series["mean_f2"])
        for p in range(6):
            assert np.array_equal(got[p][[0, 1, 3, 4, 5]], clean[p][[0, 1, 3, 4, 5]])
            assert np.isfinite(got[p]).all()
    g = f.copy()
    g[1, 3], g[4, 5] = np.inf, np.nan
    got, series, dv, v = stored(g, nv)
    assert got[0][1] == np.inf and got[2][1] == np.inf and np.isnan(got[0][4])
    assert all(np.array_equal(got[p][[0, 2, 3, 5]], clean[p][[0, 2, 3, 5]]) for p in range(6))
