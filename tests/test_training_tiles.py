"""Loss and gradient of the warm-start network where its tiles of 32
neighbours and 12 (or 6) systems per block end: neighbour counts from none to
64, one system to more than a block's, features off a 16-byte boundary."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import nn_oracle  # noqa: E402
from geosgs import learned  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 8, 31, 32, 33, 40, 63, 64])
@pytest.mark.parametrize("nsys,shift", [(1, 0), (7, 1), (13, 0), (150, 3)])
def test_loss_and_gradient(geosgs_lib, k, nsys, shift):
    rng = np.random.default_rng(100 * k + nsys)
    params = learned.init_params(1) + rng.standard_normal(nn_oracle.NPARAMS).astype(np.float32) * 0.05
    feat = rng.standard_normal((nsys, k, 8)).astype(np.float32)
    count = rng.integers(0, k + 1, nsys).astype(np.int32)
    count[0] = k
    target = rng.standard_normal((nsys, k)).astype(np.float32) * 0.2
    buf = torch.zeros(feat.size + 4, dtype=torch.float32, device="cuda")
    f = buf[shift : shift + feat.size].view(nsys, k, 8)
    f.copy_(torch.from_numpy(feat))
    loss, grad = learned.loss_and_grad(torch.from_numpy(params).cuda(), f, torch.from_numpy(count).cuda(),
                                       torch.from_numpy(target).cuda(), torch)
    want_loss, want = 0.0, np.zeros(nn_oracle.NPARAMS)
    live = count > 0
    if live.any():
        want_loss, want = nn_oracle.loss_and_grad(params, feat[live], count[live], target[live])
    # FP32 sums of up to 150 x 64 terms of mixed sign: 1e-6 of the largest gradient and more
    assert abs(loss - want_loss) <= 2e-6 * max(abs(want_loss), 1e-6) * 10
    np.testing.assert_allclose(grad.cpu().numpy(), want, rtol=0, atol=2e-5 * max(np.abs(want).max(), 1e-9))
