"""The k nearest of many data where the ring of buckets that bounds them can
go wrong: clusters, data outside the grid (kept in its edge buckets) and
nothing but those, fewer data than the ring starts with, exactly k data, balls
smaller and larger than the ring, and uneven cells."""
import numpy as np
import pytest

import geosgs
from geosgs import simulation

pytestmark = pytest.mark.gpu


def points(kind, dim, n, size, rng):
    if kind == "spread":
        return rng.uniform(0.0, 1.0, (n, dim)) * size
    if kind == "clustered":
        return 0.05 * size * rng.standard_normal((n, dim)) + 0.3 * size
    if kind == "outside":
        return (rng.uniform(-1.0, 2.0, (n, dim))) * size
    return np.array([4.0] + [1.5] * (dim - 1)) * size * (1.0 + 0.2 * rng.uniform(size=(n, dim)))  # far


CASES = [
    ("spread", (60, 50), (1.0, 1.0), 900, 10, None),
    ("spread", (33, 47), (1.0, 1.0), 65, 65 - 1, None),
    ("spread", (90, 20), (0.2, 5.0), 300, 1, None),
    ("clustered", (70, 61), (1.0, 1.0), 400, 16, None),
    ("clustered", (30, 30, 12), (1.0, 1.0, 2.0), 300, 12, None),
    ("outside", (64, 64), (1.0, 1.0), 500, 8, None),
    ("outside", (20, 17, 9), (1.0, 1.0, 1.0), 250, 32, geosgs.MetricBall(25.0)),
    ("far", (40, 40), (1.0, 1.0), 100, 9, None),
    ("spread", (60, 50), (1.0, 1.0), 900, 10, geosgs.MetricBall(3.0)),
    ("spread", (60, 50), (1.0, 1.0), 900, 10, geosgs.MetricBall(40.0)),
]


@pytest.mark.parametrize("kind,dims,spacing,ndata,k,ball", CASES)
def test_nearest_data_match_oracle(geosgs_lib, oracle_mod, kind, dims, spacing, ndata, k, ball):
    rng = np.random.default_rng(ndata + k)
    grid = geosgs.CartesianGrid(dims, spacing=spacing)
    size = np.asarray(dims) * np.asarray(spacing)
    data = geosgs.georef({"Z": rng.standard_normal(ndata)}, points(kind, len(dims), ndata, size, rng))
    process = geosgs.GaussianProcess(geosgs.ExponentialVariogram(range=float(size.max()), sill=1.0, nugget=0.1), 0.0)
    opts = simulation._KrigingOptions(maxneighbors=k, minneighbors=1, neighborhood=ball, precision="fp64")
    p, keep = geosgs.build_problem(process, grid, data, opts)
    mean, var = geosgs.posterior(process, grid, data, maxneighbors=k, neighborhood=ball)
    want_mean, want_var = oracle_mod.OraclePlan(p, keep).krige()
    # the same neighbours solved in FP64: 64 x 64 systems of condition below
    # 1e3; one other neighbour moves the values by 1e-6 and more
    np.testing.assert_allclose(mean, want_mean, rtol=0, atol=1e-10)
    np.testing.assert_allclose(var, want_var, rtol=0, atol=1e-10)
    # and beside grid neighbours, early nodes with fewer than k of them
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(1), maxneighbors=k, precision="fp64", neighborhood=ball)
    p, keep = geosgs.build_problem(process, grid, data, method)
    plan = geosgs.Plan(p, keep).prepare()
    got, gcount = plan.neighbors()
    want, wcount = oracle_mod.OraclePlan(p, keep).prepare().neighbors()
    plan.close()
    np.testing.assert_array_equal(gcount, wcount)
    np.testing.assert_array_equal(got, want)
