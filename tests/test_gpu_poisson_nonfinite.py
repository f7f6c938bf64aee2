"""A 1 / kx table with an entry that is no number (the caller kept 1 / 0 for the mean, for
instance): the field is NaN and the status word says so, whichever entry it is, as the
reference's product with the spectrum gives it."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("nx,entry", [(64, 0), (64, 32), (64, 5), (64, 63), (49, 0), (49, 24), (48, 24), (2, 0), (2, 1)])
def test_entry_that_is_no_number(nx, entry, value):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from vlapy_gb300._lib import VG_ERR_NUMERIC, VlagpuError
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    dv, v, kv = vo.velocity_axis(6.4, 32)
    inv = inv.copy()
    inv[entry] = value
    p = Plan(nx, 32, x, v, kx, kv, inv, dx, dv, dt=0.1)
    rho = torch.as_tensor(1e-3 * np.cos(0.3 * x) + 1e-4 * np.sin(0.6 * x), device="cuda")
    e = torch.zeros(nx, dtype=torch.float64, device="cuda")
    p.poisson(rho, e)
    assert torch.isnan(e).all()
    with pytest.raises(VlagpuError) as err:
        p.status()
    assert err.value.status == VG_ERR_NUMERIC
