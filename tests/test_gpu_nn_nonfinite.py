"""The weight gradient of activations that are not finite: only the taps that meet them are not, whether or not a
row of pixels fills the kernel's chunks."""
import numpy as np
import pytest

from oracle import nn_oracle as NO

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 2, 9, 16, 17, 63, 64, 65, 130])
@pytest.mark.parametrize("Cin,Cout", [(32, 64), (64, 72), (96, 16)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_last_column_not_finite(W, Cin, Cout, bad):
    from simulated_tem_gb300 import nn as N
    rng = np.random.default_rng(W + Cin)
    B, H = 2, 3
    x, gy = (NO.bf16_round(rng.standard_normal((B, H, W, c)).astype(np.float32)) for c in (Cin, Cout))
    x[:, :, -1] = 0.0
    want = NO.conv2d_grad_weight(x, gy, 9)  # the left taps (tap % 3 == 0) never meet the last column
    x[:, :, -1] = bad
    gw = torch.zeros((Cout, 9, Cin), dtype=torch.float32, device="cuda")
    N.conv2d_wgrad(*(torch.from_numpy(v).to(torch.bfloat16).cuda() for v in (x, gy)), 9, gw)
    got = gw.cpu().numpy()
    assert N.last_kernel_error() == 0
    assert np.abs(got[:, ::3] - want[:, ::3]).max() <= 1e-5 * np.abs(want).max() + 1e-6
    assert not np.isfinite(got[:, 4]).any()  # the centre meets it everywhere
