"""The dataflow sweep against the per-level launches: row lengths around a
lane's and a warp's chunks, every lane split, ranges of levels handed to the
per-level form in between, neighbour lists longer than a warp, and draws that
carry the very bit pattern which stands for "not yet stored"."""
import numpy as np
import pytest

import geosgs
from geosgs import _abi

pytestmark = pytest.mark.gpu


def make_plan(dims, k, precision, nreals):
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=k, precision=precision)
    model = geosgs.ExponentialVariogram(range=6.0, sill=1.0, nugget=0.1)
    p, keep = geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(tuple(dims)), None, method)
    plan = geosgs.Plan(p, keep).prepare()
    z = np.random.default_rng(nreals).standard_normal((nreals, plan.N))
    return plan, z


# every value is a weighted sum of at most k + 1 terms, rounded once: the two
# orders of summation differ by a few roundings of the value's own precision
# at each of some tens of levels, which the weights (they sum to one) carry on
# without growth
TOL = {"fp32": 64 * 2.0**-23, "fp64": 4096 * 2.0**-52}


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nreals,k", [(1, 5), (4, 40), (5, 8), (9, 33), (31, 8), (32, 64), (64, 8), (100, 8), (129, 17),
                                      (260, 8)])
def test_flow_matches_level_launches(geosgs_lib, precision, nreals, k):
    plan, z = make_plan((23, 19), k, precision, nreals)
    plan.set_sweep(mode=_abi.SGS_SWEEP_LEVELS)
    want = plan.simulate(nreals, z=z)
    nl = plan.info().nlevels
    forms = [dict(lanes_w=w, lanes_g=g, tight=t) for w in (0, 1, 2, 4, 8, 16) for g in (1, 2) for t in (0, 1)]
    forms += [dict(chunk=3), dict(level_lo=2, level_hi=nl), dict(level_lo=0, level_hi=3), dict(level_lo=2, level_hi=nl - 2)]
    for form in forms:
        plan.set_sweep(**form)
        got = plan.simulate(nreals, z=z)
        np.testing.assert_allclose(got, want, rtol=0, atol=TOL[precision] * np.abs(want).max(), err_msg=str(form))
    plan.close()


@pytest.mark.parametrize("precision,bits", [("fp32", np.uint32), ("fp64", np.uint64)])
def test_draws_with_the_unstored_pattern(geosgs_lib, precision, bits):
    plan, z = make_plan((16, 16), 6, precision, 5)
    z = z.astype(np.float32 if precision == "fp32" else np.float64)
    z.view(bits)[2, ::37] = ~bits(0)
    plan.set_sweep(mode=_abi.SGS_SWEEP_LEVELS)
    want = plan.simulate(5, z=z)
    assert np.isnan(want[2]).any() and not np.isnan(want[[0, 1, 3, 4]]).any()
    for form in (dict(), dict(level_lo=1, level_hi=4)):
        plan.set_sweep(**form)
        got = plan.simulate(5, z=z)
        assert np.array_equal(np.isnan(got), np.isnan(want))
    plan.close()
