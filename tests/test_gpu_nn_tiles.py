"""The convolution kernels at the edges of their tiles, against the oracle: rows about 128 pixels, channel
counts that fill an output tile (whole-sector stores) and that do not, every operand swizzle."""
import numpy as np
import pytest

from oracle import nn_oracle as NO

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nn():
    from simulated_tem_gb300 import nn as N
    N.lib()
    return N


def _rand(rng, *shape, scale=1.0):
    return NO.bf16_round(rng.standard_normal(shape).astype(np.float32) * scale)


def _bf16(a):
    return torch.from_numpy(NO.bf16_round(a)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("B,H,W,Cin,Cout,taps", [
    (1, 5, 127, 64, 64, 9), (2, 3, 128, 32, 32, 9), (1, 4, 129, 16, 64, 9), (1, 1, 1, 64, 64, 9), (1, 7, 31, 64, 48, 9),
    (1, 2, 130, 64, 32, 1), (1, 3, 127, 96, 32, 9), (2, 4, 129, 192, 64, 9), (1, 5, 33, 48, 64, 9),
    (1, 3, 128, 128, 128, 9), (1, 2, 129, 64, 256, 9), (1, 3, 20, 80, 136, 9), (1, 1, 257, 128, 64, 1),
])
def test_conv_tiles(nn, B, H, W, Cin, Cout, taps):
    rng = np.random.default_rng(H * 1000 + W + Cin + Cout)
    x, w = _rand(rng, B, H, W, Cin), _rand(rng, Cout, taps, Cin, scale=1.0 / np.sqrt(taps * Cin))
    bias = rng.standard_normal(Cout).astype(np.float32)
    mask = _rand(rng, B, H, W, Cout)
    b = torch.from_numpy(bias).cuda()
    want = NO.conv2d(x, w, bias) * (mask > 0)
    got = nn.conv2d(_bf16(x), _bf16(w), b, mask=_bf16(mask), out_fp32=True)
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    # BF16 output: the same values, rounded once
    assert torch.equal(nn.conv2d(_bf16(x), _bf16(w), b, mask=_bf16(mask)), got.to(torch.bfloat16))
    plain = nn.conv2d(_bf16(x), _bf16(w), b, relu=True, out_fp32=True)
    assert torch.equal(nn.conv2d(_bf16(x), _bf16(w), b, relu=True), plain.to(torch.bfloat16))
    assert nn.last_kernel_error() == 0


@pytest.mark.parametrize("B,H,W,Cin,Cout,taps", [
    (1, 3, 63, 16, 64, 9), (2, 5, 65, 96, 32, 9), (1, 2, 64, 128, 72, 9), (1, 1, 1, 64, 64, 9), (1, 40, 70, 32, 16, 9),
    (3, 1, 129, 48, 136, 1), (1, 6, 33, 192, 64, 9),
])
def test_weight_gradient_tiles(nn, B, H, W, Cin, Cout, taps):
    rng = np.random.default_rng(H * 1000 + W + Cin + Cout)
    x, gy = _rand(rng, B, H, W, Cin), _rand(rng, B, H, W, Cout)
    gw = torch.zeros((Cout, taps, Cin), dtype=torch.float32, device="cuda")
    nn.conv2d_wgrad(_bf16(x), _bf16(gy), taps, gw)
    want = NO.conv2d_grad_weight(x, gy, taps)
    assert nn.last_kernel_error() == 0
    assert np.abs(gw.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max() + 1e-6


@pytest.mark.parametrize("pixels,C,offset", [(1, 8, 0), (255, 16, 0), (1000, 24, 0), (77, 12, 0), (513, 64, 1),
                                             (3000, 512, 0)])
def test_bias_gradient_tiles(nn, pixels, C, offset):
    """16-byte loads for channel counts and addresses that allow them, single elements otherwise."""
    rng = np.random.default_rng(pixels + C)
    g = _rand(rng, pixels, C)
    buf = torch.zeros(pixels * C + offset, dtype=torch.bfloat16, device="cuda")
    view = buf[offset:].view(pixels, C)
    view.copy_(_bf16(g))
    gb = torch.zeros(C, dtype=torch.float32, device="cuda")
    nn.bias_grad(view, gb)
    want = NO.conv2d_grad_bias(g)
    assert np.abs(gb.cpu().numpy() - want).max() <= 1e-6 * np.abs(g).sum(axis=0).max() + 1e-6
