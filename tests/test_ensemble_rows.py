"""Ensemble statistics of float rows where their forms change: row lengths
around a lane's, a group's and a warp's values, strides above the row, node
counts that leave lanes over, offsets, thresholds on and beside the values,
and rows of zeros, of one value, of infinities, of NaN, of very large, very
small and very different magnitudes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from geosgs import ensemble  # noqa: E402

pytestmark = pytest.mark.gpu


def rows(n, r, stride, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, stride)).astype(np.float32)
    x[1] = 0.0
    x[2] = np.float32(1.7)
    x[3] *= np.float32(1e25)
    x[4] *= np.float32(1e-30)
    x[5] = np.float32(1000.0) + np.float32(2.0**-14) * rng.integers(0, 3, stride)
    x[6, : max(1, r // 2)] *= np.float32(2.0**-40)
    x[7, 0] = np.inf
    x[8, r - 1] = -np.inf
    return x


@pytest.mark.parametrize("offset", [0.0, 3.25])
@pytest.mark.parametrize("r", [1, 2, 7, 8, 9, 31, 32, 33, 64, 65, 100, 127, 128, 129, 255, 256, 257, 512, 513, 1000, 1024])
def test_float_rows(geosgs_lib, r, offset):
    n, stride = 77, r + r % 3
    x = rows(n, r, stride, r)
    v = torch.from_numpy(x).cuda()
    y = x[:, :r].astype(np.float64) + offset
    mean, var = (t.cpu().numpy() for t in ensemble.mean_var(v, r, stride, offset))
    ok = np.isfinite(y).all(axis=1)
    top = np.abs(y).max(axis=1)
    # sums of r terms in 53 bits, in any order: r units in the last place of
    # the largest term at most, and so for the squares about the mean
    with np.errstate(all="ignore"):
        want_mean, want_var = y.mean(axis=1), y.var(axis=1, ddof=1) if r > 1 else np.full(n, np.nan)
    assert np.all(np.abs(mean - want_mean)[ok] <= r * 2.0**-52 * top[ok])
    if r > 1:
        spread = np.abs(y - want_mean[:, None]).max(axis=1)
        bound = r * 2.0**-50 * (spread**2 + 2.0**-52 * top * spread) + (r * 2.0**-52 * top) ** 2
        assert np.all(np.abs(var - want_var)[ok] <= bound[ok])
    else:
        assert np.isnan(var).all()
    assert not np.isfinite(mean[~ok]).any()
    if r > 1:
        assert np.isnan(var[~ok]).all()

    p = [0.0, 0.1, 1 / 3, 0.5, 0.999, 1.0]
    got = ensemble.quantile(v, r, p, stride, offset).cpu().numpy()
    s = np.sort(y, axis=1)
    for i, pi in enumerate(p):
        h = (r - 1) * pi
        lo = min(int(np.floor(h)), r - 1)
        hi = min(lo + 1, r - 1)
        with np.errstate(all="ignore"):
            want = s[:, lo] + (h - np.floor(h)) * (s[:, hi] - s[:, lo])
        fin = np.isfinite(want)
        # one product and one sum, fused or not
        assert np.all(np.abs(got[fin, i] - want[fin]) <= 2.0**-51 * (np.abs(s[fin, lo]) + np.abs(s[fin, hi])))
        assert np.array_equal(np.isnan(got[:, i]), np.isnan(want))

    pick = y[9, : min(r, 3)]
    thr = np.concatenate([pick, np.nextafter(pick, np.inf), np.nextafter(pick, -np.inf), [-1.0, offset, np.inf, -np.inf, np.nan]])
    for t in (thr, thr[:3]):
        for comp in (False, True):
            got = ensemble.cdf(v, r, t, stride, offset, complement=comp).cpu().numpy()
            cmp = y[:, :, None] > t if comp else y[:, :, None] <= t
            assert np.array_equal(got, cmp.sum(axis=1) / r)


def test_rows_with_nan(geosgs_lib):
    x = np.random.default_rng(0).standard_normal((40, 24)).astype(np.float32)
    x[::5, 3] = np.nan
    v = torch.from_numpy(x).cuda()
    mean, var = (t.cpu().numpy() for t in ensemble.mean_var(v, 24, 24))
    assert np.array_equal(np.isnan(mean), np.isnan(x).any(axis=1))
    assert np.array_equal(np.isnan(var), np.isnan(x).any(axis=1))
    with np.errstate(invalid="ignore"):
        want = (x <= np.float32(0.5)).sum(axis=1) / 24
    assert np.array_equal(ensemble.cdf(v, 24, [0.5], 24).cpu().numpy()[:, 0], want)
