"""The default sweep configuration can be read and set again: it says that the
launch chooses between the kernel's two forms."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def problem(dims):
    method = geosgs.GPUSEQSIM(path=geosgs.RandomPath(4), maxneighbors=8, precision="fp32")
    model = geosgs.ExponentialVariogram(range=6.0, sill=1.0, nugget=0.1)
    return geosgs.build_problem(geosgs.GaussianProcess(model, 0.0), geosgs.CartesianGrid(dims), None, method)


def test_default_configuration_of_a_plan(geosgs_lib):
    plan = geosgs.Plan(*problem((23, 19))).prepare()
    config = plan.sweep_config()
    assert config["tight"] == -1
    want = plan.simulate(5, seed=2)
    plan.set_sweep(tight=1)
    plan.set_sweep(**config)
    assert plan.sweep_config() == config
    assert np.array_equal(plan.simulate(5, seed=2), want)
    for tight in (-2, 2):
        with pytest.raises(geosgs.GeoSGSError):
            plan.set_sweep(tight=tight)
    plan.close()


def test_default_configuration_of_a_batch(geosgs_lib):
    batch = geosgs.Batch([problem((23, 19)), problem((9, 14))]).prepare()
    want = batch.simulate(5, seed=2)
    batch.set_sweep(tight=1)
    batch.set_sweep(tight=-1)
    assert all(np.array_equal(a, b) for a, b in zip(batch.simulate(5, seed=2), want))
    with pytest.raises(geosgs.GeoSGSError):
        batch.set_sweep(tight=-2)
    batch.close()
