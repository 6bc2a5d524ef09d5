"""The k nearest data of nodes that lie far from all of them: rings of buckets
around such a node stay empty, which must not cost more than testing every
datum would."""
import time

import numpy as np
import pytest

import geosgs
from geosgs import simulation

pytestmark = pytest.mark.gpu


def problem(dims, points):
    rng = np.random.default_rng(1)
    data = geosgs.georef({"Z": rng.standard_normal(len(points))}, points)
    model = geosgs.ExponentialVariogram(range=float(max(dims)), sill=1.0, nugget=0.1)
    return geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(dims), data


def best_time(process, grid, data):
    t = []
    for _ in range(4):
        t0 = time.perf_counter()
        geosgs.posterior(process, grid, data, maxneighbors=10)
        t.append(time.perf_counter() - t0)
    return min(t)


def test_clustered_data_cost_no_more_than_all_of_them(geosgs_lib):
    # a million nodes on 16,384 buckets in a row: some 8,000 rings to a cluster
    # at one end when each is looked at (940 ms), and testing all 100 data
    # takes three times what the nearest of 100 spread ones take
    dims = (131072, 8)
    u = np.random.default_rng(0).uniform(size=(100, 2))
    spread = best_time(*problem(dims, u * np.array(dims)))
    clustered = best_time(*problem(dims, u * 8.0))
    assert clustered <= 4.0 * spread + 0.02


@pytest.mark.parametrize("dims,ndata", [((4096, 8), 100), ((2048, 16), 70), ((600, 8, 8), 150)])
def test_clustered_data_match_oracle(geosgs_lib, oracle_mod, dims, ndata):
    rng = np.random.default_rng(ndata)
    process, grid, data = problem(dims, rng.uniform(size=(ndata, len(dims))) * 8.0)
    opts = simulation._KrigingOptions(maxneighbors=10, minneighbors=1, neighborhood=None, precision="fp64")
    p, keep = geosgs.build_problem(process, grid, data, opts)
    mean, var = geosgs.posterior(process, grid, data, maxneighbors=10)
    want_mean, want_var = oracle_mod.OraclePlan(p, keep).krige()
    # the same neighbours solved in FP64, nugget a tenth of the sill; one other
    # neighbour moves the values by 1e-6 and more
    np.testing.assert_allclose(mean, want_mean, rtol=0, atol=1e-10)
    np.testing.assert_allclose(var, want_var, rtol=0, atol=1e-10)


@pytest.mark.parametrize("scale", [1e-25, 1e-23, 1e-19, 1e-15, 1e15, 1e19, 1e25])
@pytest.mark.parametrize("radius", [None, 30.0])
def test_lengths_whose_squares_leave_fp32(geosgs_lib, scale, radius):
    rng = np.random.default_rng(3)
    z = rng.standard_normal(300)
    u = rng.uniform(size=(300, 2)) * 64.0

    def mean(s):
        process = geosgs.GaussianProcess(geosgs.ExponentialVariogram(range=20.0 * s, sill=1.0, nugget=0.1), 0.0)
        grid = geosgs.CartesianGrid((64, 64), spacing=(s, s))
        ball = None if radius is None else geosgs.MetricBall(radius * s)
        return geosgs.posterior(process, grid, geosgs.georef({"Z": z}, u * s), maxneighbors=10, neighborhood=ball)[0]

    # the same neighbours: lags rounded at another scale, systems of condition
    # below 1e3; other neighbours move the values by 1e-3 and more
    np.testing.assert_allclose(mean(scale), mean(1.0), rtol=0, atol=1e-10)
