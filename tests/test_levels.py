"""Dependency levels where their kernel's tickets of 32 nodes begin and end:
node counts around multiples of 32, linear paths (neighbours within a
ticket), random ones, and batches of many small domains (one node, less than
a ticket, several tickets) whose order the values depend on."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def problem(dims, k, path, seed=0, ndata=0, precision="fp64"):
    rng = np.random.default_rng(seed)
    data = None
    if ndata:
        data = geosgs.georef({"Z": rng.standard_normal(ndata)}, rng.uniform(0.0, 1.0, (ndata, len(dims))) * dims)
    p = geosgs.LinearPath() if path == "linear" else geosgs.RandomPath(seed)
    method = geosgs.GPUSEQSIM(path=p, maxneighbors=k, precision=precision)
    model = geosgs.ExponentialVariogram(range=7.0, sill=1.0, nugget=0.1)
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(tuple(dims)), data, method)


@pytest.mark.parametrize("path", ["linear", "random"])
@pytest.mark.parametrize("dims,k", [((1, 1), 4), ((31, 1), 6), ((32, 1), 6), ((33, 1), 6), ((63, 1), 64), ((8, 8), 9),
                                    ((65, 1), 3), ((41, 37), 26), ((13, 9, 11), 48)])
def test_levels_follow_the_neighbours(geosgs_lib, dims, k, path):
    p, keep = problem(dims, k, path, seed=3, ndata=5 if len(dims) == 3 else 0)
    plan = geosgs.Plan(p, keep).prepare()
    nbr, cnt = plan.neighbors()
    level, nlevels = plan.levels()
    order = np.arange(plan.N) if path == "linear" else geosgs.RandomPath(3).permutation(plan.N)
    expect = np.zeros(plan.N, dtype=np.int64)
    for g in order:
        c = nbr[g, :cnt[g]]
        c = c[c < plan.N]
        expect[g] = 1 + expect[c].max() if c.size else 0
    plan.close()
    assert np.array_equal(level, expect)
    assert nlevels == expect.max() + 1


def test_levels_of_many_small_domains(geosgs_lib, oracle_mod):
    sizes = [(1, 1), (5, 5), (16, 2), (33, 1), (7, 9), (40, 30), (9, 8, 5)] * 6
    probs = [problem(d, 8, "linear" if i % 3 == 0 else "random", seed=i, ndata=i % 4) for i, d in enumerate(sizes)]
    batch = geosgs.Batch(probs).prepare()
    zs = [np.random.default_rng(d).standard_normal((2, int(n))) for d, n in enumerate(batch.sizes)]
    vals = batch.simulate(2, z=zs)
    batch.close()
    for d, (p, keep) in enumerate(probs):
        # FP64 solves and values: sums in another order, a few ulp a level
        np.testing.assert_allclose(vals[d], oracle_mod.OraclePlan(p, keep).prepare().simulate(2, zs[d]), rtol=0, atol=1e-10)
