"""FP64 results at their own rounding: the deviations of small systems against
extended precision, and the factor of a multivariate prior against correctly
rounded roots and quotients."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def deviation(cov, lags, own):
    """sqrt(1 - w'c) of a stack of systems by Cholesky, in the lags' precision."""
    K, c = cov(lags), cov(own)
    n = c.shape[1]
    L, y, w = np.zeros_like(K), np.zeros_like(c), np.zeros_like(c)
    for j in range(n):
        L[:, j, j] = np.sqrt(K[:, j, j] - (L[:, j, :j] ** 2).sum(1))
        for i in range(j + 1, n):
            L[:, i, j] = (K[:, i, j] - (L[:, i, :j] * L[:, j, :j]).sum(1)) / L[:, j, j]
        y[:, j] = (c[:, j] - (L[:, j, :j] * y[:, :j]).sum(1)) / L[:, j, j]
    for j in range(n - 1, -1, -1):
        w[:, j] = (y[:, j] - (L[:, j + 1 :, j] * w[:, j + 1 :]).sum(1)) / L[:, j, j]
    return np.sqrt(1 - (w * c).sum(1))


@pytest.mark.parametrize("k", [4, 8, 10, 16])
def test_deviations_of_small_systems(geosgs_lib, k):
    n, rng = 48, np.random.default_rng(k)
    at = rng.uniform(size=(40, 2)) * n
    data = geosgs.georef({"Z": rng.standard_normal(40)}, at)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=k, precision="fp64")
    process = geosgs.GaussianProcess(geosgs.SphericalVariogram(range=20.0, sill=1.0, nugget=0.0), 0.0)
    p, keep = geosgs.build_problem(process, geosgs.CartesianGrid((n, n)), data, method)
    plan = geosgs.Plan(p, keep).prepare()
    _, sigma, status = plan.weights()
    idx, cnt = plan.neighbors()
    plan.close()
    g = np.nonzero((status == 0) & (cnt == k))[0]
    x = np.arange(n * n)
    points = np.concatenate([np.stack([x % n + 0.5, x // n + 0.5], axis=1), at])

    def cov(lag):
        h = np.sqrt((lag**2).sum(-1)) / 20
        return np.where(h < 1, 1 - (1.5 * h - 0.5 * h**3), 0)

    P = points[idx[g]]
    lags = P[:, :, None] - P[:, None], P - points[g][:, None]
    want = deviation(cov, *(v.astype(np.longdouble) for v in lags))

    def rms(s):
        return np.sqrt(float(((s - want) ** 2).mean()))

    # no further off than a plain FP64 Cholesky of the same systems
    assert rms(sigma[g]) <= rms(deviation(cov, *lags))


def test_factor_of_a_multivariate_prior(geosgs_lib):
    rng = np.random.default_rng(0)
    L = 8
    for _ in range(40):
        B = rng.standard_normal((L, L))
        A = B @ B.T + 0.1 * np.eye(L)
        A = 0.5 * (A + A.T)
        method = geosgs.GPUSEQSIM(path=geosgs.LinearPath(), maxneighbors=1, precision="fp64")
        process = geosgs.GaussianProcess(geosgs.SphericalVariogram(range=2.0, sill=1.0, nugget=0.0), 0.0)
        p, keep = geosgs.build_problem(process, geosgs.CartesianGrid((2, 1)), None, method)
        plan = geosgs.Plan(p, keep).set_multivariate(np.zeros(L), A[None]).prepare()
        z = np.zeros((1, L, 2))
        z[0, 0] = 1.0
        got = plan.simulate_multivariate(1, z=z)[0, :, 0]  # the first node: the factor's first column
        plan.close()
        assert np.array_equal(got, np.r_[np.sqrt(A[0, 0]), A[1:, 0] / np.sqrt(A[0, 0])])
