"""The FP32 kriging solve against the FP64 oracle at the edges of its tiles:
neighbour counts around multiples of 4 (block rows), 16 (rows per lane) and
the kernel's size classes, systems of data alone, of grid nodes alone and
mixed, one and several structures, data on and off cell centres, and a grid far from the
origin.  The solve accepts a system when its estimated weight error is at
most 1e-9 of the weights (below 1 here), so weights and variances are held to 1e-8."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu

TOL = 1e-8


def solve_case(k, dims, ndata, model, centres=False, origin=None, seed=0, path="random"):
    grid = geosgs.CartesianGrid(tuple(dims), origin=origin)
    rng = np.random.default_rng(seed)
    data = None
    if ndata:
        lo, ext = np.asarray(grid.origin, dtype=np.float64), np.asarray(dims, dtype=np.float64)
        if centres:
            xyz = grid.centroids()[rng.choice(grid.nelements(), ndata, replace=False)]
        else:
            xyz = lo + rng.uniform(0.0, 1.0, (ndata, len(dims))) * ext
        data = geosgs.georef({"Z": rng.standard_normal(ndata)}, xyz)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(seed), maxneighbors=k, precision="fp32")
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.3), grid, data, method)


def exp3(nugget=0.05):
    return geosgs.ExponentialVariogram(ranges=(14.0, 9.0, 4.0), rotation=geosgs.RotZ(30.0), sill=1.7, nugget=nugget)


CASES = {f"k{k}_3d": (k, (13, 11, 7), 60, exp3()) for k in (1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64)}
CASES.update({
    "k20_2d_nodata": (20, (31, 29), 0, geosgs.SphericalVariogram(range=9.0, sill=0.8, nugget=0.1)),
    "k40_2d_centres": (40, (30, 28), 80, geosgs.GaussianVariogram(range=8.0, sill=1.0, nugget=0.2), True),
    "k48_mostly_data": (48, (16, 16), 400, geosgs.SphericalVariogram(range=12.0, sill=1.0, nugget=0.1)),
    "k64_mostly_data": (64, (14, 14), 400, geosgs.ExponentialVariogram(range=12.0, sill=1.0, nugget=0.1)),
    "k24_nested": (24, (15, 14, 6), 50, exp3(0.1) + geosgs.SphericalVariogram(range=6.0, sill=0.6, nugget=0.05)),
    "k32_far_origin": (32, (20, 18), 50, geosgs.ExponentialVariogram(range=9.0, sill=1.0, nugget=0.1), True,
                       (3.0e6, -7.0e6)),
})


@pytest.mark.parametrize("name", sorted(CASES))
def test_fp32_solve_matches_oracle(geosgs_lib, oracle_mod, name):
    p, keep = solve_case(*CASES[name])
    plan = geosgs.Plan(p, keep).prepare()
    ref = oracle_mod.OraclePlan(p, keep).prepare()
    assert np.array_equal(plan.neighbors()[0], ref.neighbors()[0])
    w, s, st = plan.weights()
    wo, so, sto = ref.weights()
    plan.close()
    assert np.array_equal(st, sto)
    np.testing.assert_allclose(w, wo, rtol=0, atol=TOL)
    np.testing.assert_allclose(s * s, so * so, rtol=0, atol=TOL)


def test_batch_of_every_size_class(geosgs_lib, oracle_mod):
    probs = [solve_case(*CASES[n]) for n in ("k5_3d", "k16_3d", "k31_3d", "k48_3d", "k64_3d", "k48_mostly_data")]
    batch = geosgs.Batch(probs).prepare()
    for d, (p, keep) in enumerate(probs):
        w, s, st = batch.weights(d)
        wo, so, sto = oracle_mod.OraclePlan(p, keep).prepare().weights()
        assert np.array_equal(st, sto)
        np.testing.assert_allclose(w, wo, rtol=0, atol=TOL)
        np.testing.assert_allclose(s * s, so * so, rtol=0, atol=TOL)
    batch.close()
