"""The sweep's stored series carry the background's moments as doubles: a collisionless run
without a perturbation stays at its background, whose moments are the sums a host makes."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


def test_series_of_the_background():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from vlapy_gb300.sweep import Sweep
    runs = [dict(nx=nx, nv=nv, k=0.3, amplitude=0.0, nu=0.0) for nv in (256, 512, 1024, 2048) for nx in (32, 64, 128)]
    sw = Sweep(runs)
    sw.reset()
    eh, sh = sw.history(2)
    sw.run_steps(2, eh, sh)
    torch.cuda.synchronize()
    for i, r in enumerate(runs):
        f, e = (t.cpu().numpy() for t in sw.read_run(i))
        f0 = f[0]
        assert np.array_equal(f, np.repeat(f0[None, :], r["nx"], axis=0)) and not e.any()
        dv, v, kv = vo.velocity_axis(6.4, r["nv"])
        w = np.ones(r["nv"])
        w[0] = w[-1] = 0.5
        got = sh[:, i].cpu().numpy()
        # one after the other, as the host adds them up: n and f^2 to the bit
        for q, terms in ((0, w * f0), (5, w * f0 * f0)):
            assert (got[:, q] == np.add.accumulate(terms)[-1] * dv).all(), (i, q)
        t = np.add.accumulate(w * f0 * (v * v))[-1] * dv
        np.testing.assert_allclose(got[:, 2], t, rtol=1e-15, atol=0)
