"""The density's trapz with its tree added level by level: NumPy's bits.

Lengths around the tree's changes of shape: one leaf, leaves shorter than eight terms'
multiples, two to sixty-four leaves, odd splits.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [2, 3, 9, 100, 129, 130, 131, 257, 386, 1000, 1025, 4096, 8191, 8192])
def test_density_has_numpys_bits(nv):
    from vlapy_gb300.plan import Plan
    nx = 5
    dx, x, kx, inv = vo.spatial_axis(0.0, 20.0, nx)
    dv, v, kv = vo.velocity_axis(6.0, nv)
    f = np.random.default_rng(nv).standard_normal((nx, nv)) ** 3
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1)
    n = torch.empty(nx, dtype=torch.float64, device="cuda")
    p.charge_density(torch.as_tensor(f, device="cuda"), n)
    np.testing.assert_array_equal(n.cpu().numpy(), np.trapezoid(f, dx=dv, axis=1))
