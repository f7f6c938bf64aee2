"""The semi-Lagrangian solves at the edges of their splits, against the oracle.

Around the rules: nx on both sides of 32 (x step: eight chunks of a column's unknowns,
the last one short or empty, a short last block of columns), nv on both sides of 256
and 512 (v step: one, two or four warps a row).  The bar is that of
the steps themselves, a relative L2 of 1e-12: the splits reassociate a contracting
recurrence (factors below 0.27), which moves a result by a few roundings.
"""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402

pytestmark = pytest.mark.gpu
TOL_SL = 1e-12


@pytest.mark.parametrize("nx,nv", [(31, 255), (32, 256), (33, 33), (35, 511), (40, 512), (64, 513), (257, 100)])
def test_sl_splits_match_oracle(nx, nv):
    from vlapy_gb300.plan import Plan
    k, vmax = 0.3, 6.0
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / k, nx)
    dv, v, kv = vo.velocity_axis(vmax, nv)
    rng = np.random.default_rng(nx * 7919 + nv)
    f = np.exp(-v ** 2 / 2)[None, :] * (1.0 + 0.1 * np.cos(k * x))[:, None] + 1e-3 * rng.standard_normal((nx, nv))
    e = 0.2 * np.sin(k * x) + 0.05
    p = Plan(nx, nv, x, v, kx, kv, inv, dx, dv, dt=0.1)
    fin = torch.as_tensor(f, device="cuda")
    gx = p.vdfdx_sl(fin, torch.empty_like(fin), 0.1).cpu().numpy()
    gv = p.edfdv_sl(fin, torch.as_tensor(e, device="cuda"), torch.empty_like(fin), 0.1).cpu().numpy()
    for got, ref in ((gx, vo.vdfdx_sl(f, x, v, 0.1)), (gv, vo.edfdv_sl(f, e, x, v, 0.1))):
        assert np.linalg.norm(got - ref) <= TOL_SL * np.linalg.norm(ref)


@pytest.mark.parametrize("nx", [32, 61])
def test_sl_x_split_matches_a_thread_a_column(nx):
    """nv = 4864 takes the split x solve, 4865 a thread a column; the columns they share
    (values and velocities) agree to the reassociation of a recurrence of factors below
    0.27, a few 2^-53 of the second differences: 1e-14 of the values."""
    from vlapy_gb300.plan import Plan
    dx, x, kx, inv = vo.spatial_axis(0.0, 2 * np.pi / 0.3, nx)
    v = -6.0 + 12.0 / 4864 * (np.arange(4865) + 0.5)
    rng = np.random.default_rng(nx)
    f = np.exp(-v ** 2 / 2)[None, :] * (1.0 + 0.1 * np.cos(0.3 * x))[:, None] + 1e-3 * rng.standard_normal((nx, 4865))
    out = []
    for nv in (4864, 4865):
        p = Plan(nx, nv, x, v[:nv], kx, np.fft.fftfreq(nv), inv, dx, 12.0 / 4864, dt=0.1)
        fin = torch.as_tensor(np.ascontiguousarray(f[:, :nv]), device="cuda")
        out.append(p.vdfdx_sl(fin, torch.empty_like(fin), 0.1).cpu().numpy()[:, :4864])
    assert np.linalg.norm(out[0] - out[1]) <= 1e-14 * np.linalg.norm(out[1])
    assert not np.array_equal(out[0], f[:, :4864])
