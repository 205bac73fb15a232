"""GPU: the tensor-core convolutions at the edges of their tiles against torch FP64: images smaller than
a tile, sides that are not multiples of the 8 x 16 (or 8 x 32) pixel tile, channel counts of every
operand block (16, 32, 64) and of several blocks, output channels that are not a power of two or leave
a part of the last 128, resident and streamed weights, and more tiles than CTAs."""

import ctypes

import numpy as np
import pytest

from conftest import rel_l2

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
F = torch.nn.functional

# BF16 results: rounding 2^-9 per value; FP32 weight gradients: sums of up to 2^19 products
TOL_BF16, TOL_F32 = 4e-3, 1e-5


@pytest.mark.parametrize("b,h,w,cin,cout", [(1, 1, 1, 16, 16), (2, 5, 9, 16, 32), (1, 17, 7, 32, 16), (3, 16, 8, 32, 32),
                                            (1, 33, 31, 64, 48), (2, 15, 23, 64, 64), (1, 34, 9, 64, 96),
                                            (2, 33, 17, 128, 64), (1, 31, 40, 128, 128), (1, 9, 9, 256, 192),
                                            (1, 12, 20, 512, 144), (1, 20, 12, 16, 256), (2, 200, 136, 32, 32)])
def test_convolutions_at_tile_edges(b, h, w, cin, cout):
    from pycorrectedemissionct_b200 import _lib

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    g = torch.Generator(device=dev)
    g.manual_seed(b + h * w + cin * cout)
    x = torch.randn((b, h, w, cin), generator=g, device=dev).bfloat16()
    wt = (torch.randn((cout, 9, cin), generator=g, device=dev) / (3 * cin**0.5)).bfloat16()
    dy = torch.randn((b, h, w, cout), generator=g, device=dev).bfloat16()
    bias = torch.randn(cout, generator=g, device=dev)
    y = torch.full((b, h, w, cout), float("nan"), device=dev, dtype=torch.bfloat16)
    dw = torch.zeros((cout, 9, cin), device=dev)
    db = torch.zeros(cout, device=dev)
    d = _lib.ConvDesc(b, h, w, cin, cout)
    for relu in (0, 1):
        _lib.check(lib.cct_conv3x3_fwd(ctypes.byref(d), x.data_ptr(), wt.data_ptr(), bias.data_ptr(), relu, y.data_ptr(),
                                       None))
        torch.cuda.synchronize()
        ref = F.conv2d(x.double().permute(0, 3, 1, 2), wt.double().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2),
                       bias.double(), padding=1)
        ref = (ref.relu() if relu else ref).permute(0, 2, 3, 1)
        assert rel_l2(y.double().cpu().numpy(), ref.cpu().numpy()) < TOL_BF16
    _lib.check(lib.cct_conv3x3_wgrad(ctypes.byref(d), x.data_ptr(), dy.data_ptr(), dw.data_ptr(), None))
    _lib.check(lib.cct_net_bias_grad(dy.data_ptr(), db.data_ptr(), b * h * w, cout, None))
    torch.cuda.synchronize()
    xp = F.pad(x.double().permute(0, 3, 1, 2), (1, 1, 1, 1))
    rows = dy.double().permute(3, 0, 1, 2).reshape(cout, -1)
    ref = torch.stack([rows @ xp[:, :, ky:ky + h, kx:kx + w].permute(0, 2, 3, 1).reshape(-1, cin)
                       for ky in range(3) for kx in range(3)], 1)
    assert rel_l2(dw.double().cpu().numpy(), ref.cpu().numpy()) < TOL_F32
    assert rel_l2(db.double().cpu().numpy(), rows.sum(1).cpu().numpy()) < TOL_F32
    v = ctypes.c_int32(0)
    _lib.check(lib.cct_net_timeout(1, ctypes.byref(v)))
    assert v.value == 0


@pytest.mark.parametrize("c,offset", [(16, 0), (48, 0), (12, 0), (16, 1), (520, 0)])
def test_elementwise_wide_and_narrow(c, offset):
    """Pooling, upsampling (both ways), additions and bias gradients with 16-byte accesses and without (a
    channel count or an address that does not allow them), exactly against torch."""
    from pycorrectedemissionct_b200 import _lib

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    g = torch.Generator(device=dev)
    g.manual_seed(c)

    def make(*shape):  # integers small enough that every sum is exact in BF16
        n = int(np.prod(shape))
        t = torch.randint(-8, 9, (n + offset,), generator=g, device=dev).bfloat16()[offset:]
        return t.view(shape)

    def nan(*shape):
        return torch.full((int(np.prod(shape)) + offset,), float("nan"), device=dev).bfloat16()[offset:].view(shape)

    b, h, w = 3, 10, 14
    x, s, x2 = make(b, h, w, c), make(b, h // 2, w // 2, c), make(b, h, w, c)
    small, large, up, down, total = nan(*s.shape), nan(*x.shape), nan(*x.shape), nan(*s.shape), nan(*x.shape)
    db = torch.zeros(c, device=dev)
    _lib.check(lib.cct_net_avgpool2(x.data_ptr(), small.data_ptr(), b, h, w, c, 0, None))
    _lib.check(lib.cct_net_avgpool2(s.data_ptr(), large.data_ptr(), b, h, w, c, 1, None))
    _lib.check(lib.cct_net_upsample2(s.data_ptr(), up.data_ptr(), b, h // 2, w // 2, c, 0, None))
    _lib.check(lib.cct_net_upsample2(x.data_ptr(), down.data_ptr(), b, h // 2, w // 2, c, 1, None))
    _lib.check(lib.cct_net_add(x.data_ptr(), x2.data_ptr(), total.data_ptr(), x.numel(), None))
    _lib.check(lib.cct_net_bias_grad(x.data_ptr(), db.data_ptr(), b * h * w, c, None))
    torch.cuda.synchronize()
    sums = x.double().view(b, h // 2, 2, w // 2, 2, c).sum((2, 4))
    rep = s.double().repeat_interleave(2, 1).repeat_interleave(2, 2)
    assert torch.equal(small.double(), sums / 4) and torch.equal(down.double(), sums)
    assert torch.equal(large.double(), rep / 4) and torch.equal(up.double(), rep)
    assert torch.equal(total.double(), x.double() + x2.double())
    assert torch.equal(db.double(), x.double().sum((0, 1, 2)))


@pytest.mark.parametrize("b,h,w,cin,cout", [(1, 18, 11, 128, 32), (2, 16, 8, 256, 16), (1, 33, 9, 512, 16), (1, 7, 9, 64, 128)])
def test_convolutions_of_one_tap_per_stage(b, h, w, cin, cout):
    """Several channel blocks with weights that stay in shared memory (9 cin cout values in 74 KB at most) and
    one block with weights that do not: both walk the taps one by one."""
    test_convolutions_at_tile_edges(b, h, w, cin, cout)


@pytest.mark.parametrize("cin,cout,offset", [(16, 16, 0), (32, 32, 0), (64, 64, 0), (64, 48, 8), (128, 16, 0), (64, 128, 0),
                                             (128, 144, 8), (256, 32, 0)])
def test_persistent_tiles_reuse_their_buffers(cin, cout, offset):
    """At least five tiles per CTA with ragged edges, so that every ring of stages wraps and both accumulators
    are filled again: whole tiles of 16, 32 and 64 channels, one tap per stage with weights that stay
    (128 -> 16) and that do not, the weight gradient with one, two and three sets of taps, and results
    that begin at 16, not 32 bytes.  Lanes past the image store nothing."""
    from pycorrectedemissionct_b200 import _lib

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    b, h, w = 2, 227, 397
    g = torch.Generator(device=dev)
    g.manual_seed(cin + cout)
    x = torch.randn((b, h, w, cin), generator=g, device=dev).bfloat16()
    wt = (torch.randn((cout, 9, cin), generator=g, device=dev) / (3 * cin**0.5)).bfloat16()
    dy = torch.randn((b, h, w, cout), generator=g, device=dev).bfloat16()
    bias = torch.randn(cout, generator=g, device=dev)
    buf = torch.full((b * h * w * cout + 2 * offset + 32,), float("nan"), device=dev, dtype=torch.bfloat16)
    y = buf[offset:offset + b * h * w * cout].view(b, h, w, cout)
    assert y.data_ptr() % 32 == (16 if offset else 0)
    dw = torch.zeros((cout, 9, cin), device=dev)
    d = _lib.ConvDesc(b, h, w, cin, cout)
    _lib.check(lib.cct_conv3x3_fwd(ctypes.byref(d), x.data_ptr(), wt.data_ptr(), bias.data_ptr(), 0, y.data_ptr(), None))
    _lib.check(lib.cct_conv3x3_wgrad(ctypes.byref(d), x.data_ptr(), dy.data_ptr(), dw.data_ptr(), None))
    torch.cuda.synchronize()
    ref = F.conv2d(x.double().permute(0, 3, 1, 2), wt.double().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2),
                   bias.double(), padding=1).permute(0, 2, 3, 1)
    assert float((y.double() - ref).norm() / ref.norm()) < TOL_BF16
    # every tile, not the whole: BF16 rounding and nothing else at each value
    assert bool(((y.double() - ref).abs() <= 2.0**-8 * ref.abs() + 1e-3).all())
    assert bool(torch.isnan(buf[:offset]).all()) and bool(torch.isnan(buf[offset + y.numel():]).all())
    xp = F.pad(x.double().permute(0, 3, 1, 2), (1, 1, 1, 1))
    rows = dy.double().permute(3, 0, 1, 2).reshape(cout, -1)
    ref = torch.stack([rows @ xp[:, :, ky:ky + h, kx:kx + w].permute(0, 2, 3, 1).reshape(-1, cin)
                       for ky in range(3) for kx in range(3)], 1)
    assert float((dw.double() - ref).norm() / ref.norm()) < TOL_F32
    v = ctypes.c_int32(0)
    _lib.check(lib.cct_net_timeout(1, ctypes.byref(v)))
    assert v.value == 0


def test_bias_gradient_of_several_channel_blocks():
    """More than 256 channels one by one (an address that does not allow 16-byte loads): several blocks of
    channels along the grid."""
    test_elementwise_wide_and_narrow(520, 1)


@pytest.mark.parametrize("h,w", [(0, 4), (4, 0), (0, 0)])
def test_pooling_of_empty_images(h, w):
    """Images without rows or columns are accepted and nothing is written, both ways."""
    from pycorrectedemissionct_b200 import _lib

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = _lib.load()
    x = torch.ones(64, device="cuda", dtype=torch.bfloat16)
    y = torch.full((64,), 3.0, device="cuda", dtype=torch.bfloat16)
    for backward in (0, 1):
        _lib.check(lib.cct_net_avgpool2(x.data_ptr(), y.data_ptr(), 1, h, w, 16, backward, None))
    torch.cuda.synchronize()
    assert bool((y == 3.0).all())
