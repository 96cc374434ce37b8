"""Weight gradients of a few blocks: the gather kernel below the block counts
from which the halo kernel is the faster one, the halo kernel from there on;
within the f32 accumulation bound of the FP64 oracle (as tests/test_gpu_conv.py)."""
import numpy as np
import pytest

from test_gpu_conv import dev_bits, level

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg,cin,cout", [(2, 64, 64), (2, 64, 32), (2, 32, 64), (3, 32, 32), (3, 16, 32)])
@pytest.mark.parametrize("blocks", [1, 2, 3, 19, 20, 21])
def test_wgrad_of_few_blocks(msbg, ctx, blocks, lg, cin, cout):
    import torch
    unet, act, nbr, taps = level(3, lg, (blocks + 0.5) / 27, seed=blocks + cin)
    assert len(act) == blocks
    cells = blocks << (3 * lg)
    rng = np.random.default_rng(blocks * cin + cout)
    xb = unet.bf16_bits(rng.standard_normal((cells, cin)).astype(np.float32))
    gb = unet.bf16_bits(rng.standard_normal((cells, cout)).astype(np.float32))
    x, g = unet.bf16_value(xb), unet.bf16_value(gb)
    ref, absum = unet.conv3_wgrad(x, g, taps), unet.conv3_wgrad(np.abs(x), np.abs(g), taps)
    d_nbr = torch.from_numpy(nbr).cuda()
    d_x, d_g = dev_bits(xb), dev_bits(gb)
    dw = torch.empty((27, cout, cin), dtype=torch.float32, device="cuda")
    ptr = msbg._lib.ptr
    torch.cuda.synchronize()
    msbg._lib.call("msbg_conv3_wgrad_device", ctx.handle, ptr(d_nbr), blocks, lg, cin, cout, ptr(d_x), ptr(d_g), ptr(dw))
    assert np.all(np.abs(dw.cpu().numpy() - ref) <= 1e-5 * absum + 1e-30)
