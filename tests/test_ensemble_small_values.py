"""Statistics of float rows: means where values differ by more than 27 binades
(the small ones count with all their bits), and counts beside NaN."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from geosgs import ensemble  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [2, 30, 100, 128, 300, 512])
@pytest.mark.parametrize("binades", [20, 26, 27, 28, 29, 34, 45, 60, 120, 140])
def test_means_with_small_values(geosgs_lib, r, binades):
    rng = np.random.default_rng(r + binades)
    n = 70
    small = np.float32(2.0**-binades) * (1 + rng.uniform(size=(n, 1)).astype(np.float32))
    x = np.repeat(small, r, axis=1).astype(np.float32)
    x[np.arange(n), rng.integers(0, r, n)] = np.float32(1.0)
    x[::7, 0] = 0.0
    x[3::7] *= -1.0
    mean, var = (t.cpu().numpy() for t in ensemble.mean_var(torch.from_numpy(x).cuda(), r, r))
    want = np.array([math.fsum(map(float, row)) / r for row in x])
    size = np.array([math.fsum(map(float, np.abs(row))) / r for row in x])
    # exact sums, or FP64 sums of a lane's values and of the 8 or 32 lanes that
    # share a row: each addition rounds to half an ulp of the magnitudes' sum
    lanes = 8 if r <= 128 else 32
    steps = -(-r // lanes) + int(math.log2(lanes)) + 1
    assert np.all(np.abs(mean - want) <= steps * 2.0**-53 * size)
    y = x.astype(np.longdouble)
    exact = ((y - y.mean(axis=1)[:, None]) ** 2).sum(axis=1) / (r - 1)
    # the same sums of squares, each value's difference from the mean rounded
    # (to 2^-53 of numbers up to 1, twice where the mean is, too)
    assert np.all(np.abs(var - exact) <= (steps + 8) * 2.0**-53 * np.abs(exact) + 4 * r * 2.0**-53 * 2.0**-53)


def test_counts_of_rows_with_nan(geosgs_lib):
    x = np.random.default_rng(0).standard_normal((40, 24)).astype(np.float32)
    x[::5, 3] = np.nan
    v = torch.from_numpy(x).cuda()
    for complement in (False, True):
        got = ensemble.cdf(v, 24, [0.5, -1.0], 24, complement=complement).cpu().numpy()
        with np.errstate(invalid="ignore"):
            hit = x[:, :, None] > np.float32([0.5, -1.0]) if complement else x[:, :, None] <= np.float32([0.5, -1.0])
        assert np.array_equal(got, hit.sum(axis=1) / 24)
