"""The element-wise U-Net kernels that move 8 channels a thread, and the input
convolution's march over planes, at the edges of their dispatch: channels in
whole vectors and not, arrays off their 16-byte boundary (both take the scalar
kernels), grids of one coarse voxel, and input planes of one row, of a whole
tile of 16 x 64 voxels and one more, in segments of 8 planes and one more.
Against the FP64 reference on inputs exact in BF16: the sums are FP32, the
outputs rounded to BF16, at most 2^-8 of a value: 4e-3 in the L2 norm."""
import ctypes

import numpy as np
import pytest

from tests import unet_ref as R

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def dev(a, off=0, dtype=torch.bfloat16):
    """a on the device, off elements behind a 16-byte boundary"""
    t = torch.zeros(a.size + 16, dtype=dtype, device="cuda")
    t[off:off + a.size] = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to("cuda").to(dtype).reshape(-1)
    return t[off:off + a.size]


def check(got, ref):
    got = got.float().cpu().numpy().astype(np.float64).reshape(ref.shape)
    assert np.linalg.norm(got - ref) <= 4e-3 * np.linalg.norm(ref)


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 6, 10)])
@pytest.mark.parametrize("c0,c,off", [(8, 8, 0), (24, 16, 0), (16, 8, 2), (12, 10, 0)])
def test_pool_and_its_gradients(dims, c0, c, off):
    from briscola_b200 import unet

    L = unet.load()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(c0 + c + dims[2])
    half = tuple(d // 2 for d in dims)
    x = R.bf16(rng.standard_normal(dims + (c,)))
    dcat = R.bf16(rng.standard_normal(dims + (c0 + c,)))
    act, dp = R.bf16(rng.standard_normal(half + (c0,))), R.bf16(rng.standard_normal(half + (c,)))
    xd, dd, ad, pd = dev(x, off), dev(dcat, off), dev(act, off), dev(dp, off)
    p, du, ds = dev(np.zeros(dp.size), off), dev(np.zeros(act.size), off), dev(np.zeros(x.size), off)
    assert L.bun_pool(*dims, c, xd.data_ptr(), p.data_ptr(), s) == 0
    assert L.bun_unpool_grad(*dims, c0 + c, c0, dd.data_ptr(), ad.data_ptr(), du.data_ptr(), s) == 0
    assert L.bun_skip_grad(*dims, c0 + c, c0, c, dd.data_ptr(), pd.data_ptr(), xd.data_ptr(), ds.data_ptr(), s) == 0
    torch.cuda.synchronize()
    check(p, R.pool(x))
    check(du, R.sumpool(dcat[..., :c0]) * (act > 0))
    check(ds, (x > 0) * (dcat[..., c0:] + R.up(dp) / 8))


@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 16, 64), (8, 17, 65), (3, 5, 130)])
def test_input_convolution_and_its_gradient(dims):
    from briscola_b200 import unet

    L = unet.load()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(dims[1])
    x = rng.standard_normal(dims).astype(np.float32)
    w = rng.standard_normal((27, 1, 16)).astype(np.float32)
    b = rng.standard_normal(16).astype(np.float32)
    dz = R.bf16(rng.standard_normal(dims + (16,)))
    xd, wd, bd, zd = dev(x, 1, torch.float32), dev(w, 0, torch.float32), dev(b, 0, torch.float32), dev(dz)
    out = dev(np.zeros(dz.size))
    assert L.bun_conv_in(*dims, xd.data_ptr(), wd.data_ptr(), bd.data_ptr(), out.data_ptr(), s) == 0
    nblocks = 3
    part = torch.full((nblocks * 28 * 16,), float("nan"), device="cuda")
    dw = torch.zeros(28 * 16, device="cuda")
    assert L.bun_conv_in_wgrad(*dims, xd.data_ptr(), zd.data_ptr(), nblocks, part.data_ptr(), dw.data_ptr(), s) == 0
    torch.cuda.synchronize()
    x64 = x.astype(np.float64)[..., None]
    check(out, np.maximum(R.conv3(x64, w.astype(np.float64)) + b, 0))
    ref = np.concatenate([R.conv3_wgrad(x64, dz).reshape(27, 16), dz.sum(axis=(0, 1, 2))[None]])
    got = dw.cpu().numpy().astype(np.float64).reshape(28, 16)
    assert np.linalg.norm(got - ref) <= 1e-4 * np.linalg.norm(ref)  # FP32 sums


@pytest.mark.parametrize("sign", ["constant", "random"])
def test_input_gradient_over_many_voxels(sign):
    """the FP32 sums of a large grid against 64 bits: a thread adds the voxels of
    a run of 32, its runs, then the groups and blocks -- one rounding each, and
    terms of one sign are the worst case"""
    from briscola_b200 import unet

    L = unet.load()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    n, nblocks = 128, 4
    V = n**3
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.full((V,), 0.1, device="cuda")
    dz = torch.full((V, 16), 0.3, device="cuda")
    if sign == "random":
        x, dz = torch.randn(V, generator=g, device="cuda"), torch.randn((V, 16), generator=g, device="cuda")
    dz = dz.bfloat16()
    part, dw = torch.zeros(nblocks * 448, device="cuda"), torch.zeros(448, device="cuda")
    assert L.bun_conv_in_wgrad(n, n, n, x.data_ptr(), dz.data_ptr(), nblocks, part.data_ptr(), dw.data_ptr(), s) == 0
    xp = torch.nn.functional.pad(x.double().view(n, n, n), (1,) * 6)
    sums, sizes = [], []
    for t in range(28):
        a = xp[t // 9:t // 9 + n, t // 3 % 3:t // 3 % 3 + n, t % 3:t % 3 + n].reshape(1, -1) if t < 27 else \
            torch.ones((1, V), dtype=torch.float64, device="cuda")
        sums.append(a @ dz.double())
        sizes.append(a.abs() @ dz.double().abs())
    # the product is not rounded (a fused multiply-add); 32 + runs of a group + 4 groups, 8 warps, the blocks
    chain = 32 + V // 32 // (nblocks * 32) + 2 + 8 + nblocks
    err = (dw.double() - torch.cat(sums).reshape(-1)).abs()
    assert bool((err <= chain * 2.0**-24 * torch.cat(sizes).reshape(-1)).all())


@pytest.mark.parametrize("dims", [(13, 96, 320), (50, 130, 200), (130, 260, 250)])
def test_input_convolution_over_several_planes(dims):
    """2, 7 and 8 planes a thread block with a remainder: the march over planes,
    which smaller grids do not take"""
    from briscola_b200 import unet

    L = unet.load()
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w, b = (torch.randn(k, generator=g, device="cuda") for k in (dims, (27, 16), (16,)))
    out = torch.zeros((*dims, 16), dtype=torch.bfloat16, device="cuda")
    assert L.bun_conv_in(*dims, x.data_ptr(), w.data_ptr(), b.data_ptr(), out.data_ptr(), s) == 0
    xp = torch.nn.functional.pad(x.double(), (1,) * 6)
    for c in range(0, 16, 5):
        ref = b[c].double() + sum(w[t, c].double() * xp[t // 9:t // 9 + dims[0], t // 3 % 3:t // 3 % 3 + dims[1],
                                                        t % 3:t % 3 + dims[2]] for t in range(27))
        ref = ref.clamp(min=0)
        err = (out[..., c].double() - ref).norm(dim=(1, 2))  # plane by plane
        assert bool((err <= 4e-3 * ref.norm(dim=(1, 2))).all())
