"""The forward convolution where a tile's output channels are shared out over CTAs, and next to where they are not, against
FP64 on the CPU (GPU). FP32 output: <= 1e-4 of the largest magnitude (FP32 accumulation of exact BF16 products), BF16 output
<= 1e-2 (one rounding more)."""
import pytest
import torch

from oracle.surrogate_ref import conv3d_ref

pytestmark = pytest.mark.gpu

# tiles x output channels: 4 x 256 and 1 x 256 (four slices of 64), 8 x 128 (two), 64 x 256 (two), 1 x 192 (two of 96),
# 1 x 112 and 1 x 64 (undivided), 90 partial tiles x 128
SHAPES = [(1, 8, 8, 8, 64, 256), (1, 4, 4, 4, 256, 256), (2, 8, 8, 8, 32, 128), (1, 20, 20, 20, 16, 256),
          (1, 5, 6, 7, 128, 192), (1, 5, 6, 7, 32, 112), (1, 4, 4, 8, 64, 64), (1, 9, 21, 35, 16, 128)]


@pytest.mark.parametrize("shape", SHAPES)
def test_slices_of_the_output_channels(shape):
    from lcdrsimulator_b200.surrogate import conv
    N, D, H, W, Ci, Co = shape
    gen = torch.Generator().manual_seed(Ci + Co)
    x = torch.randn((N, D, H, W, Ci), generator=gen).to(torch.bfloat16)
    w = (torch.randn((Co, 27, Ci), generator=gen) * 0.05).to(torch.bfloat16)
    b = torch.randn((Co,), generator=gen)
    want = conv3d_ref(x, w, b, 1)
    top = float(want.abs().max())
    for fp32, tol in ((True, 1e-4), (False, 1e-2)):
        got = conv.conv3d_fwd(x.cuda(), w.cuda(), b.cuda(), 1, fp32).double().cpu()
        assert float((got - want).abs().max()) <= tol * top
    conv.check()
