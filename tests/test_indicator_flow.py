"""The categorical and multivariate sweeps where their lanes end: rows of
realizations around 4, 16, 32 and multiples, neighbour lists shorter than a
slice's turn and longer than a warp, 2 to 8 categories, probabilities of zero
and kriged probabilities outside [0, 1] (negative weights of a smooth model)."""
import numpy as np
import pytest

import geosgs
from geosgs import problem as gproblem

pytestmark = pytest.mark.gpu

PROB = {2: (0.7, 0.3), 3: (0.5, 0.3, 0.2), 4: (0.25, 0.0, 0.5, 0.25), 5: (0.2,) * 5, 8: (0.3, 0.2, 0.1, 0.1, 0.1, 0.1, 0.05, 0.05)}


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("ncat,k,reals", [(2, 1, 1), (2, 5, 4), (3, 12, 5), (3, 20, 33), (4, 7, 16), (4, 33, 17), (5, 9, 32),
                                          (8, 64, 64), (8, 4, 100)])
def test_categories_match_oracle(geosgs_lib, oracle_mod, precision, ncat, k, reals):
    rng = np.random.default_rng(ncat + k)
    grid = geosgs.CartesianGrid((19, 23))
    labels = rng.integers(0, ncat, 20)
    labels[:ncat] = np.arange(ncat)
    data = geosgs.georef({"C": labels}, rng.uniform(0.0, 19.0, (20, 2)))
    vario = geosgs.GaussianVariogram(range=6.0, nugget=0.05) if k < 12 else geosgs.SphericalVariogram(range=8.0)
    proc = geosgs.IndicatorProcess(vario, prob=PROB[ncat])
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(5), maxneighbors=k, precision=precision)
    p, keep = geosgs.build_problem(proc, grid, data, method)
    _, dcat = gproblem.indicator_levels(proc, data)
    plan = geosgs.Plan(p, keep).set_indicator(proc.prob, dcat).prepare()
    u = rng.uniform(0.0, 1.0, (reals, plan.N))
    got = plan.simulate_indicator(reals, u=u)
    seeded = plan.simulate_indicator(reals, seed=3)
    plan.close()
    ref = oracle_mod.OraclePlan(p, keep).prepare()
    np.testing.assert_array_equal(got, ref.simulate_indicator(reals, proc.prob, dcat, u=u))
    np.testing.assert_array_equal(seeded, ref.simulate_indicator(reals, proc.prob, dcat, seed=3))


@pytest.mark.parametrize("nvars,k,reals", [(2, 4, 1), (2, 32, 16), (3, 9, 20), (3, 21, 33), (4, 16, 40)])
def test_values_match_oracle(geosgs_lib, oracle_mod, nvars, k, reals):
    rng = np.random.default_rng(10 * nvars + k)
    grid = geosgs.CartesianGrid((21, 17))
    root = rng.standard_normal((2, nvars, nvars))
    coef = [r @ r.T + 0.3 * np.eye(nvars) for r in root]
    func = geosgs.LinearCoregionalization([(coef[0], geosgs.SphericalVariogram(range=5.0, nugget=0.1)),
                                           (coef[1], geosgs.ExponentialVariogram(range=11.0))])
    data = geosgs.georef({f"V{a}": rng.standard_normal(15) for a in range(nvars)}, rng.uniform(0.0, 17.0, (15, 2)))
    proc = geosgs.GaussianProcess(func, rng.standard_normal(nvars))
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(7), maxneighbors=k)
    p, keep = geosgs.build_problem(proc, grid, data, method)
    values = gproblem.multivariate_data(proc, data)
    plan = geosgs.Plan(p, keep).set_multivariate(proc.mean, func.coef, values).prepare()
    z = rng.standard_normal((reals, nvars, plan.N))
    got = plan.simulate_multivariate(reals, z=z)
    status = plan.weights()[2]
    plan.close()
    ref = oracle_mod.OraclePlan(p, keep).prepare()
    want = ref.simulate_multivariate(reals, proc.mean, func.coef, values, z=z)
    np.testing.assert_array_equal(status, ref.weights()[2])
    # FP64 throughout, systems of condition below 1e5, tens of levels
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-8 * max(1.0, np.abs(want).max()))
