"""Neighbour rows where the hand-out of nodes to warps changes: as many nodes
as warps, a few more, and around eight per warp (where a counter takes over),
in plans and in batches, with data and without."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def build(dims, k, ndata, seed):
    rng = np.random.default_rng(seed)
    data = geosgs.georef({"Z": rng.standard_normal(ndata)}, rng.uniform(0.0, 1.0, (ndata, 2)) * dims) if ndata else None
    model = geosgs.ExponentialVariogram(range=5.0, sill=1.0, nugget=0.1)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(seed), maxneighbors=k, precision="fp32")
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(dims), data, method)


@pytest.mark.parametrize("dims,ndata", [((1, 1), 0), ((9, 1), 3), ((97, 50), 20), ((203, 191), 0), ((204, 191), 200), ((310, 270), 50)])
def test_rows_of_a_plan(geosgs_lib, oracle_mod, dims, ndata):
    p, keep = build(dims, 6, ndata, 3)
    plan = geosgs.Plan(p, keep).prepare()
    got, gcount = plan.neighbors()
    again = geosgs.Plan(p, keep).prepare()
    np.testing.assert_array_equal(got, again.neighbors()[0])
    plan.close()
    again.close()
    want, wcount = oracle_mod.OraclePlan(p, keep).prepare().neighbors()
    np.testing.assert_array_equal(gcount, wcount)
    np.testing.assert_array_equal(got, want)


def test_values_of_a_batch(geosgs_lib, oracle_mod):
    probs = [build(d, 5, n, i) for i, (d, n) in enumerate([((150, 120), 0), ((7, 3), 2), ((160, 140), 40), ((1, 1), 0)])]
    batch = geosgs.Batch(probs).prepare()
    zs = [np.random.default_rng(d).standard_normal((1, int(n))) for d, n in enumerate(batch.sizes)]
    vals = batch.simulate(1, z=zs)
    batch.close()
    for d, (p, keep) in enumerate(probs):
        # FP32 values: a rounding per level, some tens of levels
        np.testing.assert_allclose(vals[d], oracle_mod.OraclePlan(p, keep).prepare().simulate(1, zs[d]), rtol=0, atol=2e-5)
