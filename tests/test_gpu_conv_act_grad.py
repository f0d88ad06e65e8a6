"""Activation mask and bias gradient of a convolution layer, against the same in torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvox, channels", [(1, 16), (7, 256), (85, 48), (1331, 240), (64 ** 3 + 5, 32)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mask", [True, False])
def test_masked_gradient_is_torchs_and_sums_are_exact(nvox, channels, dtype, mask):
    from lcdrsimulator_b200.surrogate import conv
    gen = torch.Generator().manual_seed(nvox + channels)
    gy = torch.randn((nvox, 1, 1, 1, channels), generator=gen).to(dtype).cuda()
    y = torch.randn((nvox, 1, 1, 1, channels), generator=gen).to(dtype).cuda()
    y.view(-1)[::11] = 0.0
    y.view(-1)[::13] = float("nan")
    want = gy * torch.where(y > 0, 1.0, 0.01).to(dtype) if mask else gy
    want = want.to(torch.bfloat16)
    g, db = conv._act_grad(y if mask else None, gy)
    assert torch.equal(g, want)
    exact = want.double().sum(dim=(0, 1, 2, 3))
    # one rounding to FP32 (2^-24) and sums in FP64 of at most nvox terms
    tol = exact.abs() * 2.0 ** -24 + want.double().abs().sum(dim=(0, 1, 2, 3)) * 2.0 ** -50 * max(nvox ** 0.5, 4)
    assert bool(((db.double() - exact).abs() <= tol).all())


@pytest.mark.parametrize("shape", [(2, 5, 7, 9, 16, 48), (8, 8, 8, 8, 256, 256), (1, 16, 16, 16, 64, 128)])
@pytest.mark.parametrize("act, fp32", [(1, False), (0, False), (1, True)])
def test_backward_in_one_call_is_its_parts(shape, act, fp32):
    from lcdrsimulator_b200.surrogate import conv
    N, D, H, W, Ci, Co = shape
    if Co not in conv.CHANNELS_IN:  # the data gradient reads Co channels
        Co = 32
    gen = torch.Generator().manual_seed(Ci + Co)
    x = torch.randn((N, D, H, W, Ci), generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn((Co, 27, Ci), generator=gen) * 0.05).to(torch.bfloat16).cuda()
    gy = torch.randn((N, D, H, W, Co), generator=gen).to(torch.float32 if fp32 else torch.bfloat16).cuda()
    y = conv.conv3d_fwd(x, w, None, act, fp32)
    dx, dw, db = conv.conv3d_bwd(x, w, y if act else None, gy)
    g, db_want = conv._act_grad(y if act else None, gy)
    assert torch.equal(dx, conv.conv3d_fwd(g, conv.flip_weights(w)))
    assert torch.equal(db, db_want)
    # the K splits of the weight gradient are added in any order: 1e-5 of the largest entry
    want = conv.conv3d_wgrad(x, g)
    assert float((dw - want).abs().max()) <= 1e-5 * float(want.abs().max())
    conv.check()


@pytest.mark.parametrize("shape", [(2, 64, 64, 64, 32, 32), (3, 37, 45, 50, 16, 48), (2, 64, 64, 64, 64, 32),
                                   (4, 33, 32, 32, 16, 128), (1, 70, 130, 126, 32, 16)])
@pytest.mark.parametrize("fp32", [False, True])
def test_planes_of_a_long_volume_are_those_of_thin_ones(shape, fp32):
    """A plane needs three input planes: the march along z gives the bits of the tile kernel on a 3-plane volume."""
    from lcdrsimulator_b200.surrogate import conv
    N, D, H, W, Ci, Co = shape
    gen = torch.Generator().manual_seed(Ci * Co + D)
    x = torch.randn((N, D, H, W, Ci), generator=gen).to(torch.bfloat16).cuda()
    w = (torch.randn((Co, 27, Ci), generator=gen) * 0.05).to(torch.bfloat16).cuda()
    b = torch.randn((Co,), generator=gen).cuda()
    y = conv.conv3d_fwd(x, w, b, 1, fp32)
    for z in sorted({0, 1, D // 2 - 1, D // 2, D // 2 + 1, D - 2, D - 1}):
        thin = torch.zeros((N, 3, H, W, Ci), dtype=torch.bfloat16, device="cuda")
        lo, hi = max(z - 1, 0), min(z + 2, D)
        thin[:, lo - z + 1:hi - z + 1] = x[:, lo:hi]
        assert torch.equal(y[:, z], conv.conv3d_fwd(thin, w, b, 1, fp32)[:, 1])
    conv.check()
