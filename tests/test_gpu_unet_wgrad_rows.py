"""The weight gradient by blocks of rows (k_wgrad_rows) at the edges of its
ranges, against the FP64 reference: rows of 16 voxels, of a partial and of two
128-voxel segments, columns of one row, of whole and of broken blocks (8, 4 and
2 rows for 16, 32 and 64 output channels), one plane (two of the three plane
offsets fall outside), one to eight blocks of 16 input channels, upsampled and
concatenated inputs, one split and more splits than blocks.  BF16 inputs are
exact in the reference, so the error is that of the FP32 accumulation: 1e-4, as
in test_gpu_unet."""
import ctypes

import numpy as np
import pytest

from tests import unet_ref as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [
    # dims, c0, up0, c1, cout, nsplit
    ((3, 4, 16), 16, 0, 0, 16, 1),
    ((1, 1, 32), 16, 0, 0, 32, 2),
    ((2, 33, 48), 32, 0, 0, 16, 3),
    ((2, 32, 128), 32, 0, 0, 32, 1),
    ((2, 3, 144), 48, 0, 0, 16, 2),
    ((2, 2, 256), 16, 0, 0, 16, 9),
    ((4, 6, 32), 32, 1, 16, 16, 3),    # decoder: upsampled + skip, 48 channels
    ((4, 70, 64), 64, 1, 32, 32, 5),   # 96 channels
    ((2, 5, 16), 64, 0, 0, 32, 4),
    ((2, 9, 16), 16, 0, 0, 16, 3),
    ((1, 1, 16), 16, 0, 0, 64, 1),
    ((2, 5, 32), 48, 0, 0, 64, 2),
    ((4, 6, 32), 64, 1, 64, 64, 3),
    ((3, 7, 144), 80, 0, 0, 32, 2),
    ((2, 2, 80), 16, 0, 0, 16, 2),     # too few rows for a block: the gather
    ((2, 2, 96), 16, 0, 0, 16, 2),     # rows long enough for a part of one
    ((3, 1, 80), 32, 0, 0, 32, 1),
    ((3, 1, 96), 32, 0, 0, 32, 1),
]


@pytest.mark.parametrize("dims,c0,up0,c1,cout,nsplit", CASES)
def test_weight_gradient_rows(dims, c0, up0, c1, cout, nsplit):
    from briscola_b200 import unet

    L = unet.load()
    rng = np.random.default_rng(c0 + 3 * cout + dims[2])
    half = tuple(d // 2 for d in dims) if up0 else dims
    s0 = R.bf16(rng.standard_normal(half + (c0,)))
    s1 = R.bf16(rng.standard_normal(dims + (c1,))) if c1 else None
    x = R.up(s0) if up0 else s0
    if c1:
        x = np.concatenate([x, s1], axis=3)
    dz = R.bf16(rng.standard_normal(dims + (cout,)))

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to("cuda").to(torch.bfloat16)

    t0, t1, d = dev(s0), dev(s1) if c1 else None, dev(dz)
    cin = c0 + c1
    nsplit = min(nsplit, -(-int(np.prod(dims)) // 128))
    part = torch.full((L.bun_wgrad_part_floats(cin, cout, nsplit),), float("nan"), device="cuda")
    dw = torch.zeros(27 * cin * cout, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = []
    for _ in range(2):
        assert L.bun_conv3_wgrad(*dims, t0.data_ptr(), c0, up0, t1.data_ptr() if c1 else None, c1, d.data_ptr(), cout,
                                 nsplit, part.data_ptr(), dw.data_ptr(), err.data_ptr(), s) == 0
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        out.append(dw.cpu().numpy().astype(np.float64).reshape(27, cin, cout))
    ref = R.conv3_wgrad(x, dz)
    assert np.linalg.norm(out[0] - ref) <= 1e-4 * np.linalg.norm(ref)
    assert np.array_equal(out[0], out[1])  # the same sums in the same order
