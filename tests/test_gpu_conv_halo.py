"""The convolutions from staged halos (forward and weight gradient): one block
to several groups of blocks per CTA, every channel pair whose stages fit,
isolated and touching blocks, a bias, a narrow f32 output; within the f32
accumulation bound of the FP64 oracle (as tests/test_gpu_conv.py)."""
import numpy as np
import pytest

from test_gpu_conv import dev_bits, level

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,frac", [(1, 1.0), (2, 0.4), (5, 0.9), (7, 0.6)])
@pytest.mark.parametrize("lg,cin,cout", [(2, 16, 16), (2, 32, 32), (2, 64, 64), (2, 64, 16), (2, 16, 64), (3, 16, 16),
                                         (3, 32, 32), (3, 16, 32)])
def test_wgrad_from_halos(msbg, ctx, nb, frac, lg, cin, cout):
    import torch
    unet, act, nbr, taps = level(nb, lg, frac, seed=nb + 3 * lg + cin)
    cells = len(act) << (3 * lg)
    rng = np.random.default_rng(nb * cin + cout)
    xb = unet.bf16_bits(rng.standard_normal((cells, cin)).astype(np.float32))
    gb = unet.bf16_bits(rng.standard_normal((cells, cout)).astype(np.float32))
    x, g = unet.bf16_value(xb), unet.bf16_value(gb)
    ref = unet.conv3_wgrad(x, g, taps)
    absum = unet.conv3_wgrad(np.abs(x), np.abs(g), taps)
    d_nbr = torch.from_numpy(nbr).cuda()
    d_x, d_g = dev_bits(xb), dev_bits(gb)
    dw = torch.empty((27, cout, cin), dtype=torch.float32, device="cuda")
    ptr = msbg._lib.ptr
    torch.cuda.synchronize()
    msbg._lib.call("msbg_conv3_wgrad_device", ctx.handle, ptr(d_nbr), len(act), lg, cin, cout, ptr(d_x), ptr(d_g), ptr(dw))
    assert np.all(np.abs(dw.cpu().numpy() - ref) <= 1e-5 * absum + 1e-30)


@pytest.mark.parametrize("nb,frac,lg,cin,cout", [
    (1, 1.0, 2, 64, 64), (2, 0.4, 2, 32, 64), (7, 0.6, 2, 64, 64), (7, 0.9, 2, 64, 32), (5, 0.9, 2, 16, 16),
    (11, 1.0, 2, 16, 32),  # 1331 blocks: nine per CTA, two passes over the weights
    (1, 1.0, 3, 32, 32), (2, 0.5, 3, 16, 32), (7, 0.6, 3, 32, 16), (6, 0.9, 3, 16, 16),
])
def test_forward_from_halos(msbg, ctx, nb, frac, lg, cin, cout):
    import torch
    unet, act, nbr, taps = level(nb, lg, frac, seed=nb + 5 * lg + cin)
    cells = len(act) << (3 * lg)
    rng = np.random.default_rng(nb * cout + cin)
    xb = unet.bf16_bits(rng.standard_normal((cells, cin)).astype(np.float32))
    wb = unet.bf16_bits((rng.standard_normal((27, cout, cin)) / np.sqrt(27 * cin)).astype(np.float32))
    bias = rng.standard_normal(cout).astype(np.float32)
    x, w = unet.bf16_value(xb), unet.bf16_value(wb)
    ref = unet.conv3(x, w, bias, taps)
    absum = unet.conv3(np.abs(x), np.abs(w), np.abs(bias), taps)
    d_nbr = torch.from_numpy(nbr).cuda()
    d_x, d_w, d_b = dev_bits(xb), dev_bits(wb), torch.from_numpy(bias).cuda()
    y = torch.empty((cells, cout), dtype=torch.float32, device="cuda")
    ptr = msbg._lib.ptr
    torch.cuda.synchronize()
    msbg._lib.call("msbg_conv3_forward_device", ctx.handle, ptr(d_nbr), len(act), lg, cin, cout, ptr(d_x), ptr(d_w), ptr(d_b), 0,
                   1, ptr(y))
    got = y.cpu().numpy().astype(np.float64)
    assert np.all(np.abs(got - ref) <= 1e-5 * absum + 1e-30)
    yb = torch.empty((cells, cout), dtype=torch.int16, device="cuda")
    msbg._lib.call("msbg_conv3_forward_device", ctx.handle, ptr(d_nbr), len(act), lg, cin, cout, ptr(d_x), ptr(d_w), ptr(d_b), 1,
                   0, ptr(yb))
    assert np.array_equal(yb.cpu().numpy().view(np.uint16), unet.bf16_bits(np.maximum(got, 0).astype(np.float32)))
