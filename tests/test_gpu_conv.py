"""tcgen05 tensor-core kernels of the denoiser against PyTorch FP32 references.

The kernels take BF16 operands and accumulate in FP32; the reference evaluates the
same BF16-rounded operands in FP32. Tolerances: GEMM (FP32 output) 1e-4 of the
output scale; convolution (BF16 output) 1e-2 of the output scale (BF16 keeps 8
significant bits).
"""
import ctypes as C

import pytest

from kuafu_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _tc_error():
    e = C.c_uint32()
    N.check(N.load().kf_tc_error(C.byref(e)))
    return e.value


@pytest.mark.parametrize("n,h,w,cin,cout,rows,relu,cstride,coff", [
    # narrow images: one CTA per 128-pixel tile, 9 tap-shifted boxes per chunk
    (2, 20, 24, 64, 40, 48, True, 40, 0),
    (3, 8, 8, 96, 160, 160, True, 160, 0),
    (1, 33, 17, 32, 288, 288, False, 288, 0),
    # images at least 128 wide: the persistent halo kernel (rows per tile R, channel
    # chunk CK, resident or streamed weights, ragged last tile in x and y, channel slices,
    # 1 to 3 output rows per MMA)
    (1, 9, 150, 32, 32, 32, False, 96, 32),     # R 4, CK 32, resident weights
    (2, 7, 200, 96, 32, 32, True, 32, 0),       # 3 streamed chunks of 32
    (1, 10, 131, 64, 64, 64, True, 160, 96),    # CK 16, 4 chunks
    (1, 5, 256, 160, 160, 160, True, 160, 0),   # R 1, n 160, one row per MMA
    (1, 6, 130, 32, 80, 80, True, 80, 0),       # R 2, n 80: three output rows per MMA (N 240)
    (1, 9, 140, 16, 32, 32, True, 32, 0),       # 16 input channels (the inference input layer)
    (1, 6, 140, 32, 288, 288, False, 288, 0),   # three 128-row slices of the weights
    (2, 3, 128, 64, 40, 48, False, 40, 0),      # N 48, output channels not a multiple of 8
    (1, 13, 384, 96, 224, 224, True, 224, 0),   # no halo shape fits: falls back to the tile kernel
])
def test_conv3x3_matches_torch(n, h, w, cin, cout, rows, relu, cstride, coff):
    import torch

    lib = N.load()
    g = torch.Generator(device="cuda").manual_seed(n * 1000 + h)
    x = torch.randn((n, h, w, cin), device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn((9, rows, cin), device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    bias = torch.randn((rows,), device="cuda", generator=g, dtype=torch.float32)
    y = torch.zeros((n, h, w, cstride), device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    N.check(lib.kf_conv3x3_bf16(x.data_ptr(), n, h, w, cin, wt.data_ptr(), rows, bias.data_ptr(), cout, int(relu),
                                y.data_ptr(), cstride, coff, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _tc_error() == 0
    # reference: tap = ky * 3 + kx reads x[y + ky - 1, x + kx - 1]  (cross-correlation, padding 1)
    wr = wt.float()[:, :cout, :].permute(1, 2, 0).reshape(cout, cin, 3, 3)
    ref = torch.nn.functional.conv2d(x.float().permute(0, 3, 1, 2), wr, bias[:cout], padding=1)
    if relu:
        ref = torch.relu(ref)
    ref = ref.permute(0, 2, 3, 1)
    got = y[..., coff:coff + cout].float()
    scale = ref.abs().max().item() + 1e-6
    err = (got - ref).abs().max().item() / scale
    assert err < 1e-2, f"max error {err:.3e} of scale {scale:.3e}"
    # channels outside the slice are untouched
    if cstride > cout:
        rest = torch.cat([y[..., :coff], y[..., coff + cout:]], dim=-1)
        assert (rest == 0).all()


# The tile kernel (images under 96 wide, up to 288 input channels): tiles of 8 x 16 pixels with
# remainders of 1 and all but 1, more tiles than CTAs (two halo buffers), channel slices of 16, one
# and several output-channel blocks, the largest resident weights; and the per-tile kernel beyond.
@pytest.mark.parametrize("n,h,w,cin,cout,rows,relu,cstride,coff", [
    (1, 1, 1, 32, 16, 16, False, 16, 0),
    (2, 17, 9, 32, 32, 32, True, 48, 16),
    (3, 15, 7, 64, 24, 32, False, 24, 0),
    (40, 33, 25, 96, 96, 96, True, 96, 0),
    (1, 16, 8, 160, 160, 160, True, 288, 128),
    (2, 31, 95, 224, 48, 48, False, 48, 0),
    (1, 20, 40, 288, 128, 128, True, 128, 0),
    (5, 64, 64, 160, 64, 64, True, 64, 0),
    (1, 10, 12, 320, 32, 32, True, 32, 0),
])
def test_conv3x3_tiles_of_narrow_images(n, h, w, cin, cout, rows, relu, cstride, coff):
    test_conv3x3_matches_torch(n, h, w, cin, cout, rows, relu, cstride, coff)


# The weight-gradient kernel by itself: pixel tiles of 8 rows by 8, 16 or 32 pixels with remainders of
# 1 and all but 1 in both directions, images smaller than a tile, more tiles than CTAs, one and
# several blocks of 32 input and of 32 or 64 output channels, channel slices, a head of 3 channels.
# Operands are small integers, so every product and every sum stays an integer below 2^24: whatever
# the order of the sums, FP32 holds them exactly, and the result has to be equal.
@pytest.mark.parametrize("n,h,w,cin,cstride,coff,dzc,cout", [
    (1, 1, 1, 32, 32, 0, 32, 32),
    (2, 3, 7, 32, 64, 32, 64, 64),
    (1, 9, 8, 64, 64, 0, 32, 3),
    (3, 17, 9, 32, 40, 8, 96, 96),
    (1, 8, 15, 96, 96, 0, 64, 40),
    (2, 7, 16, 32, 32, 0, 160, 160),
    (1, 20, 17, 160, 288, 128, 64, 64),
    (2, 33, 24, 64, 64, 0, 96, 80),
    (1, 5, 31, 32, 96, 64, 32, 32),
    (1, 16, 33, 32, 32, 0, 64, 64),
    (2, 12, 40, 96, 160, 64, 32, 32),
    (1, 10, 63, 32, 32, 0, 160, 130),
    (1, 24, 64, 288, 288, 0, 128, 128),
    (5, 130, 150, 32, 32, 0, 32, 32),
    (16, 64, 97, 64, 96, 32, 64, 64),
])
def test_weight_gradients_are_exact_on_integers(n, h, w, cin, cstride, coff, dzc, cout):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n * 1000 + 10 * h + w)

    def ints(*shape):
        return torch.randint(-3, 4, shape, device="cuda", generator=g)

    x, dz = ints(n, h, w, cstride), ints(n, h, w, dzc)
    dw, db = ints(9, cout, cin).float(), ints(cout).float()  # gradients are added to what is there
    xs = x[..., coff:coff + cin].double()
    z = dz[..., :cout].double().reshape(-1, cout)
    pad = torch.nn.functional.pad(xs, (0, 0, 1, 1, 1, 1))
    want_w = dw.double() + torch.stack([z.T @ pad[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
                                        for t in range(9)])
    want_b = db.double() + z.sum(0)
    xb, zb = x.to(torch.bfloat16), dz.to(torch.bfloat16)
    torch.cuda.synchronize()
    N.check(N.load().kf_conv3x3_wgrad_bf16(xb.data_ptr() + 2 * coff, cstride, n, h, w, cin, zb.data_ptr(), dzc, cout,
                                           dw.data_ptr(), db.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _tc_error() == 0
    assert torch.equal(dw.double(), want_w)
    assert torch.equal(db.double(), want_b)


def test_weight_gradients_refuse_what_the_kernel_cannot_read():
    """Refused on the host: channels that are not multiples of 32, a stride below the channels, null
    and misaligned tensors, empty images."""
    import torch

    x = torch.zeros((1, 8, 8, 64), device="cuda", dtype=torch.bfloat16)
    out = torch.zeros(9 * 64 * 64, device="cuda")
    good = dict(x=x.data_ptr(), xs=64, n=1, h=8, w=8, cin=64, dz=x.data_ptr(), dzc=64, cout=64, dw=out.data_ptr(),
                db=out.data_ptr())
    for bad in (dict(cin=48), dict(dzc=48), dict(xs=32), dict(cout=65), dict(cout=0), dict(n=0), dict(w=0),
                dict(x=x.data_ptr() + 2), dict(dz=x.data_ptr() + 8), dict(dw=None), dict(db=out.data_ptr() + 2)):
        a = {**good, **bad}
        with pytest.raises(N.KfError):
            N.check(N.load().kf_conv3x3_wgrad_bf16(*a.values(), None))


@pytest.mark.parametrize("m,n,k,splits", [(200, 96, 4096, 4), (128, 32, 64, 1), (77, 160, 1000, 3)])
def test_gemm_tn_matches_torch(m, n, k, splits):
    import torch

    lib = N.load()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn((m, k), device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn((n, k), device="cuda", generator=g).to(torch.bfloat16)
    d = torch.zeros((m, n), device="cuda", dtype=torch.float32)
    torch.cuda.synchronize()
    N.check(lib.kf_gemm_bf16_tn(a.data_ptr(), m, b.data_ptr(), n, k, d.data_ptr(), n, splits,
                                torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _tc_error() == 0
    ref = a.float() @ b.float().T
    err = (d - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
    assert err < 1e-4, f"max error {err:.3e}"


def test_bounded_wait_gives_up_reports_and_leaves_the_context_usable():
    """The tensor-core kernels' bounded wait, made to run out: a kernel waits on an mbarrier
    that nothing arrives on with a budget of 2e6 SM cycles (about 1 ms). It gives up, and
    the error word reads 99 once, then 0. The context stays usable: a convolution run after
    it matches the PyTorch reference."""
    import torch

    lib = N.load()
    _tc_error()  # start from a clear error word
    N.check(lib.kf_tc_wait_probe(2_000_000, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _tc_error() == 99
    assert _tc_error() == 0
    test_conv3x3_matches_torch(1, 6, 130, 32, 80, 80, True, 80, 0)
