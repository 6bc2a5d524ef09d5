"""Draws and values in one device buffer: the values replace the draws, in every
form of the sweep."""
import pytest

import geosgs
from geosgs import _abi

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

FORMS = [dict(), dict(lanes_g=2, tight=1), dict(level_lo=2, level_hi=5), dict(mode=_abi.SGS_SWEEP_LEVELS),
         dict(mode=_abi.SGS_SWEEP_COOPERATIVE)]
# sums of at most 9 terms in another order: a few roundings of the value at each
# of some tens of levels, carried on without growth by weights that sum to one
TOL = {torch.float32: 64 * 2.0**-23, torch.float64: 4096 * 2.0**-52}


@pytest.mark.parametrize("precision,dtype", [("fp32", torch.float32), ("fp64", torch.float64)])
@pytest.mark.parametrize("nreals", [4, 12, 100])
def test_draws_in_the_value_buffer(geosgs_lib, precision, dtype, nreals):
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=8, precision=precision)
    model = geosgs.ExponentialVariogram(range=6.0, sill=1.0, nugget=0.1)
    p, keep = geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid((23, 19)), None, method)
    plan = geosgs.Plan(p, keep).prepare()
    z = torch.randn(plan.N, nreals, dtype=dtype, generator=torch.Generator().manual_seed(nreals)).cuda()
    want = torch.empty_like(z)
    torch.cuda.synchronize()
    plan.simulate_device(nreals, z.data_ptr(), 0, want)
    for form in [None] + FORMS:
        if form is not None:
            plan.set_sweep(**form)
        buf = z.clone()
        torch.cuda.synchronize()
        plan.simulate_device(nreals, buf.data_ptr(), 0, buf)
        torch.cuda.synchronize()
        assert (buf - want).abs().max() <= TOL[dtype] * want.abs().max(), form
    plan.close()
