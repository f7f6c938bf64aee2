"""The storage moments of the FP64 mode over wide, narrow and drifting distributions,
spikes, noise, values over many decades, rows close to one and mantissas at the ends of
their range, against extended-precision sums.

Bounds, relative to the sum of the terms' moduli S (no term may be known to less than a
double is): the sum's conversion and its product with dv, 3e-16 S; n terms, each rounded
twice at up to 2^-58 of the largest one, six standard deviations of their sum, 4 sqrt(n)
2^-58 max |f v^p| dv; the entropy's logarithms 2^-55.4 of each f, at most 8.6e-17 of S
where the sum of f |log f| is a quarter of that of f, where it is less they are doubles."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import vlapy_oracle as vo  # noqa: E402
from test_gpu_moments_fx import LD, stored, trapz  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def bell(vth, drift):
    return lambda v, rng: np.exp(-(v - drift) ** 2 / (2.0 * vth * vth)) * rng.uniform(0.3, 1.5)


def spike(v, rng):
    f = 1e-12 * rng.random(v.size) + 1e-14
    f[rng.integers(v.size)] = rng.uniform(0.3, 1.3)
    return f


ROWS = {
    "vmax 6": (6.0, bell(1.0, 0.0)), "vth 0.3": (6.4, bell(0.3, 0.0)), "vth 0.3 drifting": (6.4, bell(0.3, 0.06)),
    "vth 0.24": (16.0, bell(0.24, 0.0)), "vmax 12": (12.0, bell(1.0, 0.2)), "vmax 24": (24.0, bell(1.0, 0.3)),
    "vmax 40": (40.0, bell(1.0, 0.3)), "filaments": (6.4, lambda v, rng: np.exp(-v ** 2 / 2) * (
        1 + 0.5 * np.cos(60 * v + rng.uniform(0, 6)) + 0.3 * np.cos(140 * v))),
    "spike": (6.4, spike), "noise": (6.4, lambda v, rng: rng.random(v.size) + 1e-9),
    "decades": (6.4, lambda v, rng: np.exp(8.0 * rng.standard_normal(v.size))),
    "one to 1e-3": (6.4, lambda v, rng: 1.0 + 1e-3 * rng.standard_normal(v.size)),
    "one to 1e-6": (6.4, lambda v, rng: 1.0 + 1e-6 * rng.standard_normal(v.size)),
    "one to 0.3": (6.4, lambda v, rng: np.abs(1.0 + 0.3 * rng.standard_normal(v.size)) + 0.05),
    "mantissas of ones": (6.4, lambda v, rng: (2.0 - 2.0 ** -rng.integers(20, 53, v.size)) * 2.0 ** -rng.integers(0, 3, v.size)),
    "1e5": (6.4, lambda v, rng: 1e5 * np.exp(-v ** 2 / 2)), "1e30": (6.4, lambda v, rng: 1e30 * np.exp(-v ** 2 / 2)),
}


@pytest.mark.parametrize("kind", list(ROWS))
@pytest.mark.parametrize("nv", [64, 511, 1024, 4096, 8192])
def test_moments(nv, kind):
    vmax, row = ROWS[kind]
    rng = np.random.default_rng(nv)
    v = vo.velocity_axis(vmax, nv)[1]
    for _ in range(3):
        f = np.repeat(np.maximum(row(v, rng), 1e-290)[None, :], 2, axis=0)
        got, series, dv, v = stored(f, nv, vmax)
        F = f[:1].astype(LD)
        many = 4.0 * np.sqrt(nv) * 2.0 ** -58 * dv

        def check(value, terms, name):
            ref, size = trapz(terms, dv)[0], trapz(np.abs(terms), dv)[0]
            bound = LD(3e-16) * size + LD(many) * np.abs(terms).max()
            assert abs(LD(value) - ref) <= bound, (name, float(abs(LD(value) - ref) / size), float(bound / size))

        for p in range(6):
            w = v if p == 1 else v ** p  # as NumPy forms the powers the plan holds
            check(got[p][0], F * w.astype(LD)[None, :], p)
        check(series["mean_f2"], F * F, "f2")
        check(series["mean_flogf"], F * np.log(F), "f log f")
