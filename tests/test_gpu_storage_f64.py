"""The FP64 storage step against the oracle at the sizes where its kernels
change: fewer rows than a leaf's eight accumulators, several leaves and their
tails, columns on both sides of the angle table's limit, a last CTA of
columns that is not full, one mode broadcast into several slots and several
modes."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nv,modes,slots", [
    (2, 64, 1, 1), (7, 33, 2, 2), (9, 100, 3, 3), (64, 1024, 2, 2), (130, 31, 5, 5), (300, 257, 1, 3), (1024, 8, 2, 2),
    (4096, 5, 2, 2), (4097, 5, 2, 2), (8192, 3, 3, 3), (48, 720, 2, 2), (3, 8192, 2, 2)])
def test_storage_step(nx, nv, modes, slots):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from vlapy_gb300.plan import Plan, history_struct
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.0, nv)
    rng = np.random.default_rng(nx + nv)
    f = (np.exp(-v ** 2 / 2.0) + 0.05 * np.exp(-(v - 2.0) ** 2))[None, :] * rng.uniform(0.5, 1.5, (nx, nv))
    f /= np.trapezoid(f, dx=dv, axis=1).mean()
    e, de = rng.standard_normal(nx), rng.standard_normal(nx)
    dev = torch.device("cuda")
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)  # noqa: E731
    st = {"stored_f": torch.zeros((2, slots, nv), dtype=torch.complex64, device=dev),
          "fields": {k: z(2, nx) for k in vo.FIELD_KEYS}, "series": {k: z(2) for k in vo.SERIES_KEYS}}
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1)
    t = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    p.storage_step(t(f), t(e), t(de), history_struct(st, nx, modes), 1)
    pw = [np.ones(nv), v, v ** 2, v ** 3, v ** 4, v ** 5]
    mom = [vo.trapz(f * w[None, :], dv, 1) for w in pw]
    want = dict(zip(vo.FIELD_KEYS, [e, de] + mom))
    for k in vo.FIELD_KEYS:
        # a sum of nv terms of a positive f: 1e-14 of the integrand's scale holds for any order of summation
        scale = np.abs(e).max() if k == "e" else np.abs(de).max() if k == "driver" else \
            vo.trapz(f * np.abs(pw[vo.FIELD_KEYS.index(k) - 2])[None, :], dv, 1).max()
        np.testing.assert_allclose(st["fields"][k][1].cpu().numpy(), want[k], rtol=0, atol=1e-14 * scale, err_msg=k)
        assert not st["fields"][k][0].any()
    f2, fl = vo.trapz(f * f, dv, 1), vo.trapz(f * np.log(f), dv, 1)
    series = [mom[0], mom[1], mom[2], e * e, de * de, f2, fl]
    for k, s in zip(vo.SERIES_KEYS, series):
        scale = vo.trapz(np.abs(f * np.log(f)), dv, 1).max() if k == "mean_flogf" else np.abs(s).max() + 1.0
        np.testing.assert_allclose(float(st["series"][k][1]), s.mean(), rtol=0, atol=2e-14 * scale, err_msg=k)
    F = np.fft.fft(f, axis=0)[:modes]
    got = st["stored_f"][1].cpu().numpy()
    for s in range(slots):
        ref = F[0 if modes == 1 else s]
        # complex64 of a sum of nx terms: half a unit of each component's last place, and the sum's own rounding
        assert (np.abs(got[s] - ref) <= 1.2e-7 * np.abs(ref) + 1e-12 * nx * np.abs(f).max()).all()
