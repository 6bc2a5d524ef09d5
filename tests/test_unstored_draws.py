"""Draws on the device that carry the bit pattern which stands for "not yet
stored" in a dataflow sweep, in both precisions and for rows that a warp's
lanes finish one or four realizations at a time."""
import pytest

import geosgs
from geosgs import _abi

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,dtype,word", [("fp32", torch.float32, torch.int32), ("fp64", torch.float64, torch.int64)])
@pytest.mark.parametrize("nreals", [4, 8, 36, 100])
def test_draws_of_all_ones(geosgs_lib, precision, dtype, word, nreals):
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=6, precision=precision)
    model = geosgs.ExponentialVariogram(range=6.0, sill=1.0, nugget=0.1)
    p, keep = geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid((16, 16)), None, method)
    plan = geosgs.Plan(p, keep).prepare()
    z = torch.randn(plan.N, nreals, dtype=dtype, generator=torch.Generator().manual_seed(1)).cuda()
    z.view(word)[::37, 2] = -1
    torch.cuda.synchronize()
    out = []
    for form in (dict(mode=_abi.SGS_SWEEP_LEVELS), dict(), dict(lanes_g=2), dict(tight=1), dict(level_lo=1, level_hi=4)):
        plan.set_sweep(**form)
        v = torch.empty_like(z)
        plan.simulate_device(nreals, z.data_ptr(), 0, v)
        torch.cuda.synchronize()
        out.append(v.isnan())
        assert not (v.view(word) == -1).any()
    plan.close()
    assert out[0][:, 2].any() and not out[0][:, :2].any() and not out[0][:, 3:].any()
    assert all(torch.equal(o, out[0]) for o in out)
