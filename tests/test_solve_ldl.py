"""FP64 systems of one warp where the strides, the 32-lane columns and the 4 x
8 tiles of their elimination end (17 to 64 neighbours), with and without data,
in plans and in batches of domains of different sizes."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def build(dims, k, ndata, seed):
    rng = np.random.default_rng(seed)
    data = geosgs.georef({"Z": rng.standard_normal(ndata)}, rng.uniform(0.0, 1.0, (ndata, 2)) * dims) if ndata else None
    model = geosgs.SphericalVariogram(range=14.0, sill=2.0, nugget=0.2)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(seed), maxneighbors=k, precision="fp64")
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.5), geosgs.CartesianGrid(dims), data, method)


# condition numbers below 1e4: two FP64 eliminations differ by 1e-11 and less
@pytest.mark.parametrize("k", [17, 23, 24, 25, 31, 32, 33, 39, 40, 41, 55, 56, 57, 63, 64])
@pytest.mark.parametrize("ndata", [0, 60])
def test_fp64_systems(geosgs_lib, oracle_mod, k, ndata):
    p, keep = build((21, 18), k, ndata, k)
    plan = geosgs.Plan(p, keep).prepare()
    w, s, st = plan.weights()
    plan.close()
    wo, so, sto = oracle_mod.OraclePlan(p, keep).prepare().weights()
    np.testing.assert_array_equal(st, sto)
    np.testing.assert_allclose(w, wo, rtol=0, atol=1e-10)
    np.testing.assert_allclose(s, so, rtol=0, atol=1e-10)


def test_fp64_systems_in_a_batch(geosgs_lib, oracle_mod):
    probs = [build((15 + i, 22 - i), k, 10 * (i % 2), i) for i, k in enumerate((5, 17, 33, 64, 24, 40))]
    batch = geosgs.Batch(probs).prepare()
    zs = [np.random.default_rng(d).standard_normal((2, int(n))) for d, n in enumerate(batch.sizes)]
    vals = batch.simulate(2, z=zs)
    batch.close()
    for d, (p, keep) in enumerate(probs):
        np.testing.assert_allclose(vals[d], oracle_mod.OraclePlan(p, keep).prepare().simulate(2, zs[d]), rtol=0, atol=1e-9)
