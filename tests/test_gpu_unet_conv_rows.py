"""The row-marching convolution (k_conv_rows) at the edges of its ranges,
against the FP64 reference: rows that fill 128-voxel segments and rows laid one
behind another (runs that end inside, at and after a tile), columns of one row,
of a whole segment of each output width (16, 16, 10, 8 rows) and of one row
more, one plane, one and two 16-channel groups, many of them, upsampled and
concatenated inputs that change over inside a group.  Inputs are exact in BF16,
so the error is the output's rounding, at most 2^-8 of each value and the FP32
accumulation far below it: 4e-3 in the L2 norm, as in test_gpu_unet."""
import ctypes

import numpy as np
import pytest

from tests import unet_ref as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [
    # dims, c0, up0, c1, cout
    ((1, 1, 128), 16, 0, 0, 16),
    ((2, 17, 128), 48, 0, 0, 16),
    ((2, 16, 256), 16, 0, 16, 32),
    ((1, 11, 128), 32, 0, 0, 48),
    ((2, 9, 128), 64, 0, 0, 64),
    ((1, 1, 1), 16, 0, 0, 16),
    ((3, 2, 7), 32, 0, 0, 32),
    ((8, 5, 15), 16, 0, 0, 64),    # 8 x 16 positions: one whole tile
    ((8, 17, 16), 64, 0, 0, 32),   # 8 x 17: the last plane in a second tile
    ((6, 10, 64), 64, 1, 32, 32),  # decoder: upsampled + skip
    ((4, 12, 32), 16, 1, 16, 48),
    ((2, 8, 64), 64, 1, 64, 64),
    ((2, 3, 127), 32, 0, 0, 16),
    ((2, 3, 130), 32, 0, 0, 32),   # a long run: groups of 16
    ((2, 3, 255), 16, 0, 0, 64),
    ((1, 2, 300), 16, 0, 0, 16),   # too long a row: the tiled kernel
    ((2, 2, 264), 32, 0, 0, 96),   # and its widest outputs
    ((1, 3, 260), 64, 0, 0, 128),
    ((2, 2, 24), 256, 0, 0, 16),
    ((2, 11, 64), 32, 0, 0, 96),   # two halves of the output channels
    ((1, 9, 128), 64, 0, 0, 128),
    ((1, 6, 128), 16, 0, 0, 48),   # 48 channels: one weight buffer, a CTA of 5 rows and one of 1
    ((2, 10, 188), 32, 0, 0, 48),  # the longest rows that leave two CTAs an SM their rings
    ((1, 10, 189), 32, 0, 0, 48),  # and longer ones: 10 rows a CTA
    ((2, 6, 250), 32, 0, 0, 96),
    ((2, 9, 256), 48, 0, 0, 32),   # 8 rows of 32 channels a CTA and one more
    ((64, 37, 128), 16, 0, 0, 48),  # one group: 10 rows a CTA on 5 accumulators, and 7
    ((60, 37, 100), 16, 0, 0, 48),  # 7 rows, planes one behind another
    ((64, 45, 128), 16, 0, 0, 32),  # 12 rows on 8
    ((100, 40, 128), 16, 0, 0, 16),  # 20 rows on 16
]


@pytest.mark.parametrize("dims,c0,up0,c1,cout", CASES)
def test_convolution_rows(dims, c0, up0, c1, cout):
    from briscola_b200 import unet

    L = unet.load()
    rng = np.random.default_rng(c0 + 3 * cout + dims[2])
    cin = c0 + c1
    kc = {96: 32, 128: 64}.get(cout, 16)
    half = tuple(d // 2 for d in dims) if up0 else dims
    s0 = R.bf16(rng.standard_normal(half + (c0,)))
    s1 = R.bf16(rng.standard_normal(dims + (c1,))) if c1 else None
    x = R.up(s0) if up0 else s0
    if c1:
        x = np.concatenate([x, s1], axis=3)
    W = rng.standard_normal((27, cin, cout)) / np.sqrt(27 * cin)
    bias = rng.standard_normal(cout)

    def dev(a, dtype=torch.bfloat16):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to("cuda").to(dtype)

    t0, t1, wd, bd = dev(s0), dev(s1) if c1 else None, dev(W, torch.float32), dev(bias, torch.float32)
    wp = torch.zeros(W.size, dtype=torch.bfloat16, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.bun_pack_weights(wd.data_ptr(), cin, cout, kc, 0, wp.data_ptr(), s) == 0
    n = int(np.prod(dims)) * cout
    buf = torch.full((n + 64,), 7.0, dtype=torch.bfloat16, device="cuda")  # 64 values of guard behind the output
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = L.bun_conv3(*dims, t0.data_ptr(), c0, up0, t1.data_ptr() if c1 else None, c1, wp.data_ptr(), kc, cout,
                     bd.data_ptr(), 1, None, buf.data_ptr(), err.data_ptr(), s)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert bool((buf[n:] == 7.0).all())
    ref = np.maximum(R.conv3(x, R.bf16(W)) + bias.astype(np.float32), 0)
    got = buf[:n].float().cpu().numpy().astype(np.float64).reshape(ref.shape)
    assert np.linalg.norm(got - ref) <= 4e-3 * np.linalg.norm(ref)
