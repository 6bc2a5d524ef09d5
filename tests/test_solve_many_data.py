"""FP32 systems made of data: a covariance each for the pairs, which the lag
table does not hold, spread over a block's threads without idle ones."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def make(precision, k, dims, ndata, model, seed=1):
    rng = np.random.default_rng(seed)
    data = geosgs.georef({"Z": rng.standard_normal(ndata)}, rng.uniform(size=(ndata, len(dims))) * dims)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(2), maxneighbors=k, precision=precision)
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(dims), data, method)


def test_solves_of_data_take_less_than_in_fp64(geosgs_lib):
    # four data a cell: the same covariances are evaluated for both, and FP64
    # eliminates 40 x 40 systems besides (5.6 ms; FP32 took 6.5 with half of
    # its threads idle)
    model = geosgs.SphericalVariogram(range=30.0, sill=1.0, nugget=0.1)
    best = {}
    for precision in ("fp32", "fp64"):
        plan = geosgs.Plan(*make(precision, 40, (200, 200), 160000, model))
        times = []
        for _ in range(4):
            plan.prepare()
            times.append(plan.info().ms_solve)
        plan.close()
        best[precision] = min(times)
    assert best["fp32"] <= 0.9 * best["fp64"]


@pytest.mark.parametrize("k", [1, 8, 15, 16, 17, 31, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("density", [0.05, 0.5, 6.0])
@pytest.mark.parametrize("nested", [False, True])
def test_mixed_systems_match_fp64(geosgs_lib, k, density, nested):
    # rows of a block's chunk with no, some and only data; blocks whose last
    # systems are missing
    dims = (23, 17)
    model = geosgs.ExponentialVariogram(ranges=(12.0, 5.0), rotation=geosgs.RotZ(30.0), sill=1.0, nugget=0.1)
    if nested:
        model = model + geosgs.SphericalVariogram(range=9.0, sill=0.5, nugget=0.05)
    out = []
    for precision in ("fp32", "fp64"):
        plan = geosgs.Plan(*make(precision, k, dims, int(density * dims[0] * dims[1]), model, seed=k)).prepare()
        out.append(plan.weights() + plan.neighbors())
        plan.close()
    (w, s, st, idx, cnt), (w1, s1, st1, idx1, cnt1) = out
    assert np.array_equal(idx, idx1) and np.array_equal(cnt, cnt1) and np.array_equal(st, st1)
    # the solve accepts weights whose estimated error is below 1e-9 of weights below 1
    np.testing.assert_allclose(w, w1, rtol=0, atol=1e-8)
    np.testing.assert_allclose(s * s, s1 * s1, rtol=0, atol=1e-8)
