"""Models whose sills lie near the ends of FP64's range: weights and statuses do
not depend on the sill's scale, deviations and values scale with its root."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu

SILL = 0.9137
# an even power of two scales every covariance, pivot and deviation exactly
SCALES = [-1016, -1000, -930, 800, 1020]


def problem(sill, k, precision):
    rng = np.random.default_rng(k)
    data = geosgs.georef({"Z": rng.standard_normal(30)}, rng.uniform(size=(30, 2)) * [24, 20])
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(3), maxneighbors=k, precision=precision)
    model = geosgs.ExponentialVariogram(range=6.0, sill=sill, nugget=0.03125 * sill)
    process = geosgs.GaussianProcess(model, 0.0)
    return process, geosgs.CartesianGrid((24, 20)), data, method


@pytest.mark.parametrize("e", SCALES)
@pytest.mark.parametrize("precision,k", [("fp64", 6), ("fp64", 10), ("fp64", 16), ("fp64", 40), ("fp32", 12)])
def test_weights(geosgs_lib, precision, k, e):
    out = []
    for sill in (SILL, SILL * 2.0**e):
        p, keep = geosgs.build_problem(*problem(sill, k, precision))
        plan = geosgs.Plan(p, keep).prepare()
        out.append(plan.weights())
        plan.close()
    (w, s, st), (w1, s1, st1) = out
    assert np.array_equal(st, st1) and (st == 0).any()
    np.testing.assert_array_equal(w1, w)
    if precision == "fp64":
        np.testing.assert_array_equal(s1 * 2.0 ** (-e // 2), s)


@pytest.mark.parametrize("e", SCALES)
def test_posterior(geosgs_lib, e):
    out = []
    for sill in (SILL, SILL * 2.0**e):
        process, grid, data, _ = problem(sill, 8, "fp64")
        out.append(geosgs.posterior(process, grid, data, maxneighbors=8))
    np.testing.assert_array_equal(out[1][0], out[0][0])
    # small variances, the squares of deviations, may be below the smallest
    # normal number
    np.testing.assert_allclose(out[1][1] * 2.0**-e, out[0][1], rtol=0, atol=2.0 ** (-1074 - e) if e < 0 else 0)


@pytest.mark.parametrize("e,of", [(-1000, "coef"), (-1000, "sill"), (960, "coef"), (960, "sill")])
def test_multivariate(geosgs_lib, e, of):
    A = np.array([[1.0, 0.4], [0.4, 0.7]])
    z = np.random.default_rng(0).standard_normal((3, 2, 24 * 20))
    out = []
    for scale in (1.0, 2.0**e):
        method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(3), maxneighbors=9, precision="fp64")
        sill = scale * SILL if of == "sill" else SILL
        model = geosgs.ExponentialVariogram(range=6.0, sill=sill, nugget=0.03125 * sill)
        p, keep = geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid((24, 20)), None, method)
        plan = geosgs.Plan(p, keep)
        plan.set_multivariate(np.zeros(2), (A * scale if of == "coef" else A)[None]).prepare()
        out.append(plan.simulate_multivariate(3, z=z))
        plan.close()
    np.testing.assert_array_equal(out[1] * 2.0 ** (-e // 2), out[0])
