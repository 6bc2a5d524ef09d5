"""Small FP64 systems, several to a warp, where their lanes end (neighbour
counts around 8 and 16, fewer than minneighbors, nodes left over in the last
warp, sills far from one), and systems that hold one point twice: data on cell
centres, whose cells are simulated too, and data given twice."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def build(dims, k, precision, data_xy=None, nmin=1, sill=1.0, nugget=0.05, seed=0):
    rng = np.random.default_rng(seed)
    data = None
    if data_xy is not None:
        data = geosgs.georef({"Z": np.sqrt(sill) * rng.standard_normal(len(data_xy))}, data_xy)
    model = geosgs.ExponentialVariogram(range=9.0, sill=sill, nugget=nugget * sill)
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(seed), maxneighbors=k, minneighbors=nmin, precision=precision)
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(tuple(dims)), data, method)


def compare(oracle_mod, p, keep, sill, tol):
    plan = geosgs.Plan(p, keep).prepare()
    w, s, st = plan.weights()
    info = plan.info()
    z = np.random.default_rng(1).standard_normal((3, plan.N))
    v = plan.simulate(3, z)
    plan.close()
    ref = oracle_mod.OraclePlan(p, keep).prepare()
    wo, so, sto = ref.weights()
    np.testing.assert_array_equal(st, sto)
    np.testing.assert_allclose(w, wo, rtol=0, atol=tol)
    np.testing.assert_allclose(s, so, rtol=0, atol=tol * np.sqrt(sill))
    np.testing.assert_allclose(v, ref.simulate(3, z), rtol=0, atol=100 * tol * np.sqrt(sill))
    return st, info


# condition numbers below 1e4, two eliminations in FP64: 1e-11 and less
@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 10, 11, 12, 15, 16, 17])
@pytest.mark.parametrize("ndata", [0, 40])
def test_small_fp64_systems(geosgs_lib, oracle_mod, k, ndata):
    xy = np.random.default_rng(k).uniform(0.0, 1.0, (ndata, 2)) * (31, 27) if ndata else None
    p, keep = build((31, 27), k, "fp64", xy, nmin=min(3, k), seed=k)
    compare(oracle_mod, p, keep, 1.0, 1e-10)


@pytest.mark.parametrize("sill", [1e-20, 3.0, 1e15])
def test_small_fp64_systems_of_any_sill(geosgs_lib, oracle_mod, sill):
    xy = np.random.default_rng(5).uniform(0.0, 1.0, (30, 2)) * (17, 12)
    p, keep = build((17, 12), 10, "fp64", xy, sill=sill)
    compare(oracle_mod, p, keep, sill, 1e-10)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("k", [6, 14, 30, 45])
@pytest.mark.parametrize("sill", [1.0, 49.0])
def test_one_point_twice_is_singular(geosgs_lib, oracle_mod, precision, k, sill):
    rng = np.random.default_rng(k)
    cells = rng.permutation(24 * 20)[:25]
    xy = np.stack([cells % 24 + 0.5, cells // 24 + 0.5], axis=1)
    xy = np.concatenate([xy, rng.uniform(0.0, 20.0, (10, 2))])
    xy = np.concatenate([xy, xy[-3:]])  # three data given twice
    p, keep = build((24, 20), k, precision, xy, sill=sill, nugget=0.1, seed=2)
    plan = geosgs.Plan(p, keep).prepare()
    w, s, st = plan.weights()
    info = plan.info()
    plan.close()
    sto = oracle_mod.OraclePlan(p, keep).prepare().weights()[2]
    np.testing.assert_array_equal(st, sto)
    assert (st == 2).any() and (st == 0).any()
    assert np.all(w[st == 2] == 0.0)
    np.testing.assert_allclose(s[st == 2], np.sqrt(sill), rtol=1e-14)
    # decided in the FP32 path itself
    assert info.n_fp64_fallback == 0 or precision == "fp64"
