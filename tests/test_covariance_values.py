"""Covariances evaluated on the device, read off kriging from one datum at a
cell centre (its weight is C(h) / C(0)): every model over lags from far below
to far beyond its range, at the shape's branches and in two and three
dimensions."""
import numpy as np
import pytest

import geosgs

pytestmark = pytest.mark.gpu


def shape(kind, h):
    if kind is geosgs.SphericalVariogram:
        return np.where(h < 1, 1 - 1.5 * h + 0.5 * h**3, 0.0)
    return np.exp(-3 * h) if kind is geosgs.ExponentialVariogram else np.exp(-3 * h * h)


@pytest.mark.parametrize("kind", [geosgs.SphericalVariogram, geosgs.ExponentialVariogram, geosgs.GaussianVariogram])
@pytest.mark.parametrize("spacing", [1e-300, 1e-20, 1e-9, 1e-5, 2.0**-10, 0.013, 0.25, 7.0, 1e6, 1e30])
@pytest.mark.parametrize("nugget,dim", [(0.0, 2), (0.3, 3)])
def test_covariance(geosgs_lib, kind, spacing, nugget, dim):
    n = 400
    dims = (n, 1) if dim == 2 else (n, 1, 1)
    grid = geosgs.CartesianGrid(dims, spacing=(spacing,) * dim)
    data = geosgs.georef({"Z": np.array([1.0])}, np.full((1, dim), 0.5 * spacing))
    process = geosgs.GaussianProcess(kind(range=1.0, sill=1.0, nugget=nugget), 0.0)
    mean, _ = geosgs.posterior(process, grid, data, maxneighbors=1)
    h = (np.arange(n) + 0.5) * spacing - 0.5 * spacing
    want = (1.0 - nugget) * shape(kind, h)
    want[0] = 1.0
    # 2^-56 of the sill in the shape, a rounding of the lag, the nugget's
    # share and the result each
    np.testing.assert_allclose(mean, want, rtol=0, atol=6e-16)
