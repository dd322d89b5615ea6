"""GPU parity of mgpuConv2d / mgpuPool2d (reference: lib/Kernels/GPU/Ops.cu:238-374) against
the CPU oracle and the fixtures made from the reference's PyTorch models.

Tolerances: pooling is comparison / fp32 addition work -> max pooling bit-exact, average
pooling max-abs <= 1e-6 (summation order).  Convolution feeds 16-bit operands to the tensor
cores with fp32 accumulation, like the Gemm: max-rel <= 2e-2 against the oracle run on the
same 16-bit-rounded operands, an element's error divided by max(|ref|, 1e-2 * rms(ref))
(in fact the two agree to 2e-4 of the rms: only the fp32 summation order differs).  Against
the fp32 PyTorch fixtures the operand rounding itself is part of the difference (about
2^-12 of the rms per element whatever the element's size), so there the floor is
1e-1 * rms(ref)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def m(mdc):
    mdc.init()
    return mdc


def _check_conv(m, x, w, b, post_add=None, tol16=2e-4, floor32=1e-1, **kw):
    got = m.conv2d(x, w, b, post_add=post_add, **kw)
    ref32 = oracle.conv2d(x, w, b, post_add=post_add, accum64=True, **kw)
    ref16 = oracle.conv2d(x, w, b, post_add=post_add, round_mode=oracle.ROUND_F16, accum64=True, **kw)
    assert got.shape == ref32.shape
    assert oracle.max_rel_err(ref16, got, floor_frac=1e-2) <= 2e-2
    assert oracle.max_rel_err(ref32, got, floor_frac=floor32) <= 2e-2
    # same rounded operands, exact accumulation: only fp32 summation order is left
    scale = max(float(np.sqrt(np.mean(ref16.astype(np.float64) ** 2))), 1e-6)
    assert np.max(np.abs(got - ref16)) <= tol16 * scale
    return got


def test_reference_conv_fixture(m, golden_cnn):
    g = golden_cnn
    got = _check_conv(m, g["conv_x"], g["conv_w"], g["conv_b"], pad=(1, 1, 1, 1))
    assert oracle.max_rel_err(g["conv_y"], got, floor_frac=1e-1) <= 2e-2


def test_crosscheck_conv_fixtures(m, golden_cnn):
    g = golden_cnn
    got = _check_conv(m, g["res_x"], g["res_w"], g["res_b"], post_add=g["res_add"], stride=(2, 2),
                      pad=(1, 1, 1, 1), relu=True)
    assert oracle.max_rel_err(g["res_y"], got, floor_frac=1e-1) <= 2e-2
    got = _check_conv(m, g["dil_x"], g["dil_w"], g["dil_b"], stride=(1, 2), dilation=(2, 3))
    assert oracle.max_rel_err(g["dil_y"], got, floor_frac=1e-1) <= 2e-2


@pytest.mark.parametrize("shape", [
    # N, IC, H, W, OC, KH, KW, stride, pad(t,l,b,r), dilation, post_add, relu
    (1, 1, 5, 5, 1, 1, 1, (1, 1), (0, 0, 0, 0), (1, 1), False, False),
    (2, 3, 9, 11, 5, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, True),
    (3, 16, 14, 14, 32, 1, 1, (1, 1), (0, 0, 0, 0), (1, 1), True, True),      # pointwise + residual
    (2, 7, 12, 10, 9, 5, 3, (2, 1), (2, 1, 2, 1), (1, 1), True, False),
    (1, 4, 17, 13, 6, 3, 3, (2, 2), (0, 1, 1, 0), (1, 1), False, False),     # asymmetric padding
    (2, 64, 28, 28, 128, 3, 3, (2, 2), (1, 1, 1, 1), (1, 1), False, True),   # a ResNet down-sampling layer
    (1, 3, 32, 32, 64, 7, 7, (2, 2), (3, 3, 3, 3), (1, 1), False, True),     # a ResNet stem
    (2, 6, 16, 16, 10, 3, 3, (1, 1), (2, 2, 2, 2), (2, 2), False, False),    # dilated, "same"
])
def test_conv_against_oracle(m, shape):
    N, IC, H, W, OC, KH, KW, stride, pad, dil, has_add, relu = shape
    rng = np.random.default_rng(hash(shape[:7]) % (1 << 31))
    x = rng.standard_normal((N, IC, H, W)).astype(np.float32)
    w = (rng.standard_normal((OC, IC, KH, KW)) / np.sqrt(IC * KH * KW)).astype(np.float32)
    b = (0.1 * rng.standard_normal(OC)).astype(np.float32)
    OH = (H + pad[0] + pad[2] - (KH - 1) * dil[0] - 1) // stride[0] + 1
    OW = (W + pad[1] + pad[3] - (KW - 1) * dil[1] - 1) // stride[1] + 1
    add = rng.standard_normal((N, OC, OH, OW)).astype(np.float32) if has_add else None
    _check_conv(m, x, w, b, post_add=add, stride=stride, pad=pad, dilation=dil, relu=relu)


@pytest.mark.parametrize("OC", [128, 320])
def test_conv_wide_channel_tiles(m, OC):
    """Enough pixels that the 128- and 256-channel tiles are chosen (the second 256-channel
    tile of OC = 320 is three quarters empty)."""
    rng = np.random.default_rng(OC)
    x = rng.standard_normal((8, 32, 56, 56)).astype(np.float32)
    w = (rng.standard_normal((OC, 32, 3, 3)) / np.sqrt(32 * 9)).astype(np.float32)
    b = (0.1 * rng.standard_normal(OC)).astype(np.float32)
    # 8 million outputs, half of them zeroed by the ReLU (which halves the rms): the largest
    # operand-rounding error among so many lies further out, hence the wider floor
    _check_conv(m, x, w, b, pad=(1, 1, 1, 1), relu=True, floor32=2e-1)


def test_conv_gather_modes_agree(m):
    """Channel counts that are multiples of 32 are served by the im2col kernel or, without memory for
    its copy of the input, by the direct gather; both feed the tensor core the same operands in the
    same order, so the results are bit-identical."""
    import os
    rng = np.random.default_rng(21)
    cases = [((4, 64, 14, 14), (96, 64, 3, 3), dict(pad=(1, 1, 1, 1))),
             ((2, 32, 17, 13), (40, 32, 3, 2), dict(stride=(2, 1), pad=(1, 0, 2, 1), dilation=(1, 2))),
             ((3, 96, 9, 9), (64, 96, 1, 1), dict())]
    for xs, ws, kw in cases:
        x = rng.standard_normal(xs).astype(np.float32)
        w = (rng.standard_normal(ws) / np.sqrt(np.prod(ws[1:]))).astype(np.float32)
        b = (0.1 * rng.standard_normal(ws[0])).astype(np.float32)
        staged = _check_conv(m, x, w, b, **kw)
        os.environ["MDC_CONV_DIRECT"] = "1"
        try:
            direct = m.conv2d(x, w, b, **kw)
        finally:
            del os.environ["MDC_CONV_DIRECT"]
        assert np.array_equal(staged, direct)


@pytest.mark.parametrize("IC,taps", [(32, (3, 3)), (32, (1, 1)), (96, (3, 2)), (160, (1, 3)), (64, (3, 3))])
def test_conv_direct_k_order(m, IC, taps):
    """The direct kernel's dense k order (groups of 32 channels of one tap; two taps share a k-block in
    a last block of 32 channels): exact on small integers, and bit for bit the im2col kernel's sums
    on real ones."""
    import os
    rng = np.random.default_rng(IC)
    kw = dict(stride=(2, 1), pad=(1, 0, 1, 1))
    for x, w in ((rng.integers(-4, 5, size=(3, IC, 13, 11)), rng.integers(-3, 4, size=(70, IC) + taps)),
                 (rng.standard_normal((3, IC, 13, 11)), rng.standard_normal((70, IC) + taps) / np.sqrt(IC * 9))):
        x, w, b = x.astype(np.float32), w.astype(np.float32), rng.integers(-8, 9, size=70).astype(np.float32)
        persistent = m.conv2d(x, w, b, **kw)
        os.environ["MDC_CONV_DIRECT"] = "1"
        try:
            direct = m.conv2d(x, w, b, **kw)
        finally:
            del os.environ["MDC_CONV_DIRECT"]
        assert np.array_equal(direct, persistent)
        if float(x.flat[0]).is_integer():
            assert np.array_equal(direct, oracle.conv2d(x, w, b, **kw))


def test_conv_direct_has_no_empty_half_blocks(m):
    """32 input channels cost the direct kernel half of what 64 do: two taps share a k-block.  (0.58 of
    the time measured; 0.9 when every tap was padded to 64 channels.)"""
    import os
    import torch
    s = torch.cuda.Stream()
    times = []
    for IC in (32, 64):
        x, w, b = torch.randn(64, IC, 56, 56, device="cuda"), torch.randn(64, IC, 3, 3, device="cuda"), torch.randn(64, device="cuda")
        out = torch.empty(64, 64, 56, 56, device="cuda")
        torch.cuda.synchronize()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(24)]
        os.environ["MDC_CONV_DIRECT"] = "1"
        try:
            for e in ev:
                e.record(s)
                m.ops().mgpuConv2d(x.data_ptr(), w.data_ptr(), b.data_ptr(), out.data_ptr(), None, 64, IC, 56, 56, 64, 3, 3, 56, 56,
                                   1, 1, 1, 1, 1, 1, 1, 1, False, False, s.cuda_stream)
        finally:
            del os.environ["MDC_CONV_DIRECT"]
        s.synchronize()
        m.check("conv")
        times.append(float(np.median([a.elapsed_time(b) for a, b in zip(ev[3:-1], ev[4:])])))
    assert times[0] <= 0.75 * times[1], times


def test_conv_exact_on_small_integers(m):
    """Integer-valued operands are exact in fp16 and every partial sum is exact in fp32, so the
    result must equal the oracle bit for bit: this isolates the gather / scatter indexing."""
    rng = np.random.default_rng(7)
    x = rng.integers(-4, 5, size=(2, 5, 13, 11)).astype(np.float32)
    w = rng.integers(-3, 4, size=(12, 5, 3, 3)).astype(np.float32)
    b = rng.integers(-8, 9, size=12).astype(np.float32)
    add = rng.integers(-8, 9, size=(2, 12, 7, 6)).astype(np.float32)
    got = m.conv2d(x, w, b, post_add=add, stride=(2, 2), pad=(1, 1, 1, 1), relu=True)
    ref = oracle.conv2d(x, w, b, post_add=add, stride=(2, 2), pad=(1, 1, 1, 1), relu=True)
    assert np.array_equal(got, ref)


# (how conv_plan.h sends the row at 148 SMs, the row); tests/test_conv_plan_cpu.py holds them to it
# N, IC, H, W, OC, KH, KW, stride, pad(t,l,b,r), dilation, post_add, relu
CONV_EDGES = [
    ("kOther", (1, 16, 7, 7, 16, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, False)),  # one partial tile, im2col's fewest channels
    ("kOther", (1, 15, 7, 7, 16, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, False)),  # the gather kernel's most channels
    ("kOther", (5, 24, 9, 5, 33, 3, 2, (2, 1), (0, 1, 2, 0), (1, 2), True, True)),  # asymmetric in every respect
    ("kOther", (3, 20, 11, 13, 40, 5, 3, (1, 3), (2, 0, 1, 2), (2, 1), True, False)),  # channels padded to 24
    ("kCopyRect", (2, 96, 10, 6, 65, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, True)),  # a half-full block of 64 channels: shared regions
    ("kOther", (300, 72, 8, 8, 48, 1, 1, (1, 1), (0, 0, 0, 0), (1, 1), True, False)),  # tiles of two images, one round and a bit
    ("kOther", (60, 64, 20, 21, 64, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), True, True)),  # filter kept, several tiles per CTA
    ("kOther", (40, 128, 20, 20, 96, 3, 3, (2, 2), (1, 1, 1, 1), (1, 1), False, False)),  # filter streamed
    ("kCopyFlat", (1, 256, 4, 4, 300, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), True, False)),  # many k-blocks, few pixels: shared regions
    ("kOther", (90, 3, 17, 19, 40, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, True)),  # one k-block, 32 of 64 values
    ("kDirectRect", (40, 5, 31, 30, 24, 7, 7, (2, 2), (3, 3, 3, 3), (1, 1), True, False)),  # shared regions, stride 2: more tiles than SMs
    ("kDirectFlat", (2, 14, 12, 12, 260, 7, 7, (1, 1), (3, 3, 3, 3), (1, 1), False, False)),  # shared regions, filter streamed, several channel tiles
    ("kOther", (3, 33, 11, 14, 20, 1, 1, (2, 3), (1, 0, 0, 2), (1, 1), True, False)),  # strided 1 x 1, padded: sampled copy
    ("kOther", (70, 64, 20, 20, 32, 1, 1, (2, 2), (0, 0, 0, 0), (1, 1), False, True)),
    ("kOther", (2, 16, 30, 30, 8, 2, 2, (9, 1), (0, 0, 0, 0), (1, 1), False, False)),  # stride outside the im2col map: direct kernel
    ("kOther", (2, 160, 30, 30, 8, 3, 2, (9, 1), (1, 0, 0, 1), (1, 1), True, False)),  # the same, 32 channels a block
    ("kOther", (21, 13, 16, 26, 33, 4, 4, (1, 1), (2, 2, 2, 2), (1, 1), True, True)),  # gathered: four k-blocks, two channel tiles, more tiles than SMs
    ("kOther", (54, 12, 21, 17, 8, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), True, False)),  # gathered: two k-blocks, filter kept
    ("kOther", (3, 14, 12, 12, 260, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, False)),  # gathered: filter streamed, several channel tiles
    ("kOther", (68, 65, 22, 52, 8, 3, 3, (2, 2), (1, 1, 1, 1), (1, 1), True, True)),  # im2col: filter kept, residual, a last block of one channel
]


@pytest.mark.parametrize("shape", [row for _, row in CONV_EDGES])
def test_conv_persistent_edges(m, shape):
    """Small integers (see test_conv_exact_on_small_integers): equal bit for bit."""
    N, IC, H, W, OC, KH, KW, stride, pad, dil, has_add, relu = shape
    rng = np.random.default_rng(IC * 1000 + OC)
    x = rng.integers(-4, 5, size=(N, IC, H, W)).astype(np.float32)
    w = rng.integers(-3, 4, size=(OC, IC, KH, KW)).astype(np.float32)
    b = rng.integers(-8, 9, size=OC).astype(np.float32)
    OH = (H + pad[0] + pad[2] - (KH - 1) * dil[0] - 1) // stride[0] + 1
    OW = (W + pad[1] + pad[3] - (KW - 1) * dil[1] - 1) // stride[1] + 1
    add = rng.integers(-8, 9, size=(N, OC, OH, OW)).astype(np.float32) if has_add else None
    kw = dict(post_add=add, stride=stride, pad=pad, dilation=dil, relu=relu)
    assert np.array_equal(m.conv2d(x, w, b, **kw), oracle.conv2d(x, w, b, **kw))


@pytest.mark.parametrize("shape", [
    (2, 1, 9, 7, 8, 1, 1, (1, 1), (0, 0, 0, 0), (1, 1), False, False),         # one value of eight
    (3, 14, 12, 11, 24, 3, 6, (1, 1), (1, 2, 1, 3), (1, 1), True, False),      # 252 values: the table's last 64, partly
    (3, 15, 12, 11, 24, 3, 6, (1, 1), (1, 2, 1, 3), (1, 1), False, True),      # 270: the larger table
    (40, 3, 40, 33, 16, 16, 1, (1, 1), (15, 0, 15, 0), (1, 1), False, False),  # 16 rows and 15 columns of a window have bits ...
    (2, 3, 33, 40, 16, 1, 15, (1, 2), (0, 14, 0, 14), (1, 1), True, False),
    (2, 3, 40, 33, 16, 17, 1, (2, 1), (16, 0, 16, 0), (1, 1), False, False),   # ... 17 and 16 have none
    (40, 3, 33, 40, 16, 1, 16, (1, 1), (0, 15, 0, 15), (1, 1), True, True),
    (3, 2, 3, 4, 9, 3, 3, (1, 1), (9, 7, 8, 6), (4, 3), False, False),         # margins wider than the image
    (200, 3, 10, 45, 64, 3, 3, (1, 2), (1, 1, 1, 1), (1, 1), True, True),      # several tiles for each group of warps
])
def test_conv_gathered_patches(m, shape):
    """Up to 15 channels, below 25 taps: where k lies by either table, windows partly and wholly outside.  Small integers; an
    infinity reaches the outputs of its windows and no others."""
    N, IC, H, W, OC, KH, KW, stride, pad, dil, has_add, relu = shape
    rng = np.random.default_rng(IC * 1000 + KH * 10 + KW)
    x = rng.integers(-4, 5, size=(N, IC, H, W)).astype(np.float32)
    w = rng.integers(1, 4, size=(OC, IC, KH, KW)).astype(np.float32)
    b = rng.integers(-8, 9, size=OC).astype(np.float32)
    OH = (H + pad[0] + pad[2] - (KH - 1) * dil[0] - 1) // stride[0] + 1
    OW = (W + pad[1] + pad[3] - (KW - 1) * dil[1] - 1) // stride[1] + 1
    add = rng.integers(-8, 9, size=(N, OC, OH, OW)).astype(np.float32) if has_add else None
    kw = dict(post_add=add, stride=stride, pad=pad, dilation=dil, relu=relu)
    clean = m.conv2d(x, w, b, **kw)
    assert np.array_equal(clean, oracle.conv2d(x, w, b, **kw))
    at = (N - 1, IC - 1, H // 2, W // 2)
    x[at] = np.inf
    got = m.conv2d(x, w, b, **kw)
    y, v = at[2] + pad[0] - stride[0] * np.arange(OH), at[3] + pad[1] - stride[1] * np.arange(OW)
    in_window = lambda t, d, n: (t >= 0) & (t % d == 0) & (t // d < n)
    hit = np.zeros(clean.shape, bool)
    hit[N - 1] = in_window(y, dil[0], KH)[:, None] & in_window(v, dil[1], KW)[None, :]
    assert np.array_equal(got[~hit], clean[~hit]) and np.all(np.isposinf(got[hit]))


# rows of test_conv_persistent_edges for every form of conv_form
REGION_FORMS = [
    ("kCopyRect", (3, 16, 9, 16, 16, 5, 3, (1, 1), (2, 1, 2, 1), (1, 1), True, False)),  # rect out of a copy: tiles of two images
    ("kCopyRect", (2, 72, 33, 24, 33, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, True)),  # rect: a block of 8 channels, three rounds of rows
    ("kOther", (40, 64, 24, 24, 64, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), True, True)),  # dense: filter kept, several tiles per CTA
    ("kCopyFlat", (5, 80, 7, 9, 20, 3, 5, (1, 1), (0, 3, 2, 1), (2, 1), True, False)),  # flat out of a copy: asymmetric
    ("kCopyRect", (60, 100, 13, 11, 60, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, False)),  # rect: filter streamed, 36 channels in the last block
    ("kCopyFlat", (60, 20, 19, 17, 300, 1, 1, (1, 1), (0, 0, 0, 0), (1, 1), True, True)),  # flat, 1 x 1: two channel tiles
    ("kOther", (150, 48, 15, 14, 260, 1, 1, (2, 3), (0, 0, 0, 0), (1, 1), False, True)),  # dense: 1 x 1, sampled
    ("kOther", (2, 3, 21, 70, 24, 5, 5, (1, 1), (2, 2, 2, 2), (1, 1), True, False)),  # dense: gathered, odd filter rows
    ("kDirectRect", (3, 8, 12, 10, 40, 6, 6, (1, 1), (3, 2, 2, 3), (1, 1), False, True)),  # straight from the input: pairs only
    ("kOther", (70, 1, 30, 31, 33, 7, 7, (2, 2), (3, 3, 3, 3), (1, 1), False, False)),  # dense: gathered, stride 2
    ("kOther", (2, 5, 23, 64, 300, 5, 5, (2, 1), (0, 1, 1, 1), (1, 2), True, False)),  # dense: gathered, strides and dilations apart
    ("kDirectRect", (2, 1, 20, 50, 48, 9, 9, (1, 1), (4, 4, 4, 4), (1, 1), False, False)),  # one channel: eight parts of a sum, 32 columns a tile
    ("kDirectRect", (3, 15, 14, 9, 17, 5, 5, (1, 2), (2, 2, 2, 2), (1, 3), False, True)),  # two groups of channels, columns in two classes
    ("kOther", (4, 32, 18, 21, 64, 7, 5, (2, 2), (3, 2, 3, 2), (1, 1), True, True)),  # dense: stride 2, 32 channels
    ("kCopyRect", (31, 18, 23, 25, 8, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), True, True)),  # rect: filter kept, several tiles per CTA, residual
    ("kCopyRect", (1, 86, 11, 9, 33, 3, 3, (1, 1), (1, 1, 1, 1), (1, 1), False, False)),  # rect: filter streamed, two channel tiles
    ("kCopyFlat", (72, 19, 33, 9, 8, 2, 2, (1, 1), (1, 1, 0, 0), (1, 1), True, True)),  # flat: filter kept, several tiles per CTA, residual
    ("kCopyFlat", (33, 69, 11, 24, 65, 2, 2, (1, 1), (1, 1, 1, 1), (1, 1), True, True)),  # flat: filter streamed, a last block of five channels, three channel tiles
    ("kCopyFlat", (55, 16, 36, 78, 34, 1, 1, (2, 2), (0, 0, 0, 0), (1, 1), True, False)),  # flat: 1 x 1, sampled, two channel tiles
    ("kCopyFlat", (8, 32, 1, 8000, 32, 1, 7, (1, 1), (0, 3, 0, 3), (1, 1), False, False)),  # flat: images of one row
    ("kCopyFlat", (2, 48, 1, 3000, 20, 1, 9, (1, 1), (0, 130, 0, 132), (1, 33), True, False)),  # flat: taps beyond the im2col map's offsets
    ("kOther", (2, 40, 1, 3000, 20, 1, 9, (1, 1), (0, 130, 0, 132), (1, 33), True, False)),  # the same, channels that a region would pad: direct kernel
    ("kOther", (6, 48, 1, 70, 20, 1, 9, (1, 1), (0, 132, 0, 132), (1, 33), True, False)),  # the same on tiles of mostly margins: direct kernel
    ("kDirectRect", (56, 3, 11, 32, 11, 5, 5, (1, 1), (2, 2, 2, 2), (1, 1), True, True)),  # straight: a tap without a partner, several tiles per CTA, residual
    ("kDirectRect", (74, 3, 29, 38, 8, 5, 5, (2, 2), (2, 2, 2, 2), (1, 1), False, True)),  # straight: classes of rows and columns, filter kept
    ("kDirectRect", (55, 9, 23, 58, 8, 5, 5, (2, 2), (2, 2, 2, 2), (1, 1), True, False)),  # straight: two groups of channels in classes, filter kept, several tiles per CTA
    ("kDirectRect", (1, 11, 5, 32, 39, 5, 5, (1, 1), (2, 2, 2, 2), (1, 1), False, False)),  # straight: two groups, filter streamed, two channel tiles
    ("kDirectRect", (1, 17, 7, 7, 11, 6, 6, (2, 2), (3, 3, 3, 3), (1, 1), True, True)),  # straight: stride 2, two sixteens of channels
    ("kDirectRect", (73, 16, 18, 55, 8, 5, 5, (2, 2), (2, 2, 2, 2), (1, 1), False, False)),  # straight: stride 2, one sixteen, several tiles per CTA
    ("kDirectRect", (1, 3, 5, 5, 96, 5, 5, (2, 1), (2, 2, 2, 2), (1, 2), False, False)),  # straight: strides and dilations apart, several channel tiles
    ("kDirectFlat", (78, 2, 5, 45, 8, 6, 6, (1, 1), (3, 3, 3, 3), (1, 1), True, True)),  # flat, straight: pairs, four parts of a sum, several tiles per CTA
    ("kDirectFlat", (79, 9, 33, 5, 10, 5, 5, (1, 1), (2, 2, 2, 2), (1, 1), False, True)),  # flat, straight: two groups of channels, several tiles per CTA
    ("kDirectFlat", (2, 12, 20, 20, 70, 5, 5, (1, 1), (2, 2, 2, 2), (1, 1), True, False)),  # flat, straight: two groups, several channel tiles
]


@pytest.mark.parametrize("shape", [row for _, row in REGION_FORMS])
def test_conv_halo_forms(m, shape):
    """The kernel whose tiles share one region of the input between taps, in every form of conv_form: small integers,
    equal bit for bit (see test_conv_exact_on_small_integers)."""
    test_conv_persistent_edges(m, shape)


INFINITIES = [  # form, N, IC, W (20 rows, 9 channels out, 5 x 5)
    ("kDirectRect", 2, 3, 60), ("kDirectRect", 2, 3, 20), ("kDirectFlat", 2, 12, 20), ("kCopyRect", 2, 64, 20), ("kCopyRect", 2, 64, 24),
    ("kDirectFlat", 23, 3, 33), ("kCopyFlat", 23, 64, 33),
]


@pytest.mark.parametrize("N,IC,W", [row[1:] for row in INFINITIES])
def test_conv_keeps_infinities_to_their_windows(m, N, IC, W):
    """An infinity next to a window, where the tile's region holds it and the weights of a padded tap are zero, must not
    turn into NaN: outputs whose window does not hold it are those of the input without it."""
    rng = np.random.default_rng(W)
    x = rng.integers(-4, 5, size=(N, IC, 20, W)).astype(np.float32)
    w = rng.integers(1, 4, size=(9, IC, 5, 5)).astype(np.float32)
    b = np.zeros(9, np.float32)
    clean = m.conv2d(x, w, b, pad=(2, 2, 2, 2))
    x[1, IC - 1, 9, 13] = np.inf
    got = m.conv2d(x, w, b, pad=(2, 2, 2, 2))
    hit = np.zeros(clean.shape, bool)
    hit[1, :, 7:12, 11:16] = True
    assert np.array_equal(got[~hit], clean[~hit])
    assert np.all(np.isposinf(got[hit]))


OVERLAPS = [  # form, IC, OC, size, kernel, stride (three images)
    ("kCopyRect", 24, 24, 20, 5, 1), ("kOther", 32, 32, 20, 5, 2), ("kOther", 64, 64, 24, 3, 1), ("kOther", 32, 16, 33, 1, 1),
    ("kCopyRect", 96, 64, 24, 3, 1), ("kCopyFlat", 16, 161, 73, 1, 1), ("kDirectRect", 16, 8, 5, 5, 2),
]


@pytest.mark.parametrize("IC,OC,size,kernel,stride", [row[1:] for row in OVERLAPS])
def test_conv_output_over_its_input(m, IC, OC, size, kernel, stride):
    """From 16 channels on the output may lie over the input: a launch ahead has copied it, or the call is routed so."""
    rng = np.random.default_rng(IC)
    x = rng.integers(-4, 5, size=(3, IC, size, size)).astype(np.float32)
    w = rng.integers(-3, 4, size=(OC, IC, kernel, kernel)).astype(np.float32)
    pad = kernel // 2
    out = (size - 1) // stride + 1
    ref = oracle.conv2d(x, w, None, stride=(stride, stride), pad=(pad,) * 4)
    for offset in (0, 4 * 64 * size):  # the same start, and inside
        buf, dw = m.DeviceBuffer(x.nbytes + 4 * 64 * size + ref.nbytes), m.to_device(w)
        m.runtime().mgpuMemcpy(buf.ptr, x.ctypes.data, x.nbytes, None)
        m.runtime().mgpuStreamSynchronize(None)
        m.ops().mgpuConv2d(buf.ptr, dw.ptr, None, buf.ptr + offset, None, 3, IC, size, size, OC, kernel, kernel, out, out, pad, pad,
                           pad, pad, stride, stride, 1, 1, False, False, None)
        m.check("conv")
        got = np.empty_like(ref)
        m.runtime().mgpuMemcpy(got.ctypes.data, buf.ptr + offset, ref.nbytes, None)
        m.runtime().mgpuStreamSynchronize(None)
        assert np.array_equal(got, ref)


@pytest.mark.parametrize("earlier_failure", [False, True])
@pytest.mark.parametrize("OC,KH,KW,stride", [(16, 1, 2, 8), (8, 3, 3, 1)])  # an im2col call, and one of shared regions
def test_conv_without_memory_for_the_copy(m, OC, KH, KW, stride, earlier_failure):
    """With no device memory left for the NHWC copy of the input the direct kernel takes over, whether
    or not an earlier call has left a status; that status stays."""
    import torch
    rt, ops = m.runtime(), m.ops()
    N, IC, H, W = 12, 32, 2048, 2048  # 6.4 GB in, a copy of 3.2 GB
    pad = KH // 2
    OH, OW = H // stride, W // stride
    x = torch.randint(-4, 5, (N, IC, H, W), device="cuda", dtype=torch.int8).float()
    w = torch.randint(-3, 4, (OC, IC, KH, KW), device="cuda", dtype=torch.int8).float()
    out = torch.empty(N, OC, OH, OW, device="cuda")

    def call():
        out.zero_()
        torch.cuda.synchronize()
        ops.mgpuConv2d(x.data_ptr(), w.data_ptr(), None, out.data_ptr(), None, N, IC, H, W, OC, KH, KW, OH, OW, pad, pad, pad, pad,
                       stride, stride, 1, 1, False, False, None)
        rt.mgpuStreamSynchronize(None)
    call()
    expect = out.clone()
    m.check("conv")
    assert float(expect.abs().max()) > 0
    torch.cuda.empty_cache()
    rt.mgpuPoolTrim()
    hog = torch.empty(max(torch.cuda.mem_get_info()[0] - (2 << 30), 0), device="cuda", dtype=torch.uint8)
    try:
        if earlier_failure:
            ops.mgpuConv2d(x.data_ptr(), w.data_ptr(), None, out.data_ptr(), None, -1, 0, H, W, OC, 1, 2, 1, 1, 0, 0, 0, 0, 1, 1, 1, 1,
                           False, False, None)
            ops.mgpuPool2d(None, None, 1, 1, 4, 4, 3, 3, 2, 2, 0, 0, 0, 0, 2, 2, 0, None)  # bad geometry: sets the status
            assert rt.mgpuGetLastError() != 0
        call()
        assert torch.equal(out, expect)
        assert (rt.mgpuGetLastError() != 0) == earlier_failure
    finally:
        rt.mgpuClearLastError()
        del hog
        torch.cuda.empty_cache()


def test_conv_output_smaller_than_the_geometry(m):
    """The caller may ask for fewer output rows and columns than the padded input would give."""
    rng = np.random.default_rng(3)
    N, IC, H, W, OC, OH, OW = 4, 32, 12, 11, 24, 7, 8
    x = rng.integers(-4, 5, size=(N, IC, H, W)).astype(np.float32)
    w = rng.integers(-3, 4, size=(OC, IC, 3, 3)).astype(np.float32)
    dx, dw, out = m.to_device(x), m.to_device(w), m.DeviceBuffer(N * OC * OH * OW * 4)
    m.ops().mgpuConv2d(dx.ptr, dw.ptr, None, out.ptr, None, N, IC, H, W, OC, 3, 3, OH, OW, 1, 1, 1, 1, 1, 1, 1, 1,
                       False, False, None)
    m.check("conv")
    got = m.to_host(out, (N, OC, OH, OW), np.float32)
    ref = oracle.conv2d(x, w, None, pad=(1, 1, 1, 1))[:, :, :OH, :OW]
    assert np.array_equal(got, ref)


def test_conv_reference_test_layer_full_size(m):
    """test/End2End/GPU/conv.mlir: 16x3x256x256 -> 16x64x256x256, 3x3, padding 1."""
    rng = np.random.default_rng(11)
    # multiples of 1/64: exact in fp16 and far from its subnormal range, so doubling commutes
    # with the rounding
    x = (np.round(rng.standard_normal((16, 3, 256, 256)) * 64) / 64).astype(np.float32)
    w = (rng.standard_normal((64, 3, 3, 3)) * 0.1).astype(np.float32)
    b = (0.1 * rng.standard_normal(64)).astype(np.float32)
    got = m.conv2d(x, w, b, pad=(1, 1, 1, 1))
    ref = oracle.conv2d(x, w, b, pad=(1, 1, 1, 1), round_mode=oracle.ROUND_F16)
    assert got.shape == (16, 64, 256, 256)
    assert np.max(np.abs(got - ref)) <= 1e-4
    # linearity in the input at full size: conv(2x) - bias = 2 (conv(x) - bias), exactly
    got2 = m.conv2d(2 * x, w, np.zeros_like(b), pad=(1, 1, 1, 1))
    got1 = m.conv2d(x, w, np.zeros_like(b), pad=(1, 1, 1, 1))
    assert np.array_equal(got2, 2 * got1)


def test_reference_pool_fixtures(m, golden_cnn):
    g = golden_cnn
    assert np.array_equal(m.pool2d(g["maxpool_x"], (4, 4), (4, 4)), g["maxpool_y"])
    assert np.array_equal(m.pool2d(g["pool_x"], (3, 3), (2, 2), pad=(1, 1, 1, 1), method=0), g["pool_max_y"])
    avg = m.pool2d(g["pool_x"], (3, 3), (2, 2), pad=(1, 1, 1, 1), method=1)
    assert np.max(np.abs(avg - g["pool_avg_y"])) <= 1e-6


@pytest.mark.parametrize("case", [
    # N, C, H, W, kernel, stride, pad
    (1, 1, 4, 4, (2, 2), (2, 2), (0, 0, 0, 0)),
    (2, 3, 17, 19, (3, 3), (2, 2), (1, 1, 1, 1)),
    (3, 5, 16, 12, (2, 3), (1, 2), (0, 1, 1, 2)),
    (2, 64, 56, 56, (3, 3), (2, 2), (1, 1, 1, 1)),
    (1, 2, 9, 9, (9, 9), (1, 1), (0, 0, 0, 0)),     # global pooling
    (16, 3, 256, 256, (4, 4), (4, 4), (0, 0, 0, 0)),  # test/End2End/GPU/pool.mlir
])
@pytest.mark.parametrize("method", [0, 1])
def test_pool_against_oracle(m, case, method):
    N, C, H, W, kernel, stride, pad = case
    rng = np.random.default_rng(hash(case[:4]) % (1 << 31))
    x = rng.standard_normal((N, C, H, W)).astype(np.float32)
    got = m.pool2d(x, kernel, stride, pad=pad, method=method)
    ref = oracle.pool2d(x, kernel, stride, pad=pad, method=method)
    assert got.shape == ref.shape
    if method == 0:
        assert np.array_equal(got, ref)
    else:
        assert np.max(np.abs(got - ref)) <= 1e-6 * max(1.0, kernel[0] * kernel[1] / 9)


@pytest.mark.parametrize("case", [
    # H, W, kernel, stride, pad(t,l,b,r)
    (9, 11, (2, 2), (2, 2), (0, 0, 0, 0)),    # odd width: compiled 2 x 2 instead of row vectors
    (8, 10, (2, 2), (1, 1), (0, 0, 0, 0)),
    (8, 10, (2, 2), (2, 2), (1, 0, 0, 1)),    # windows cut by the padding on one side
    (13, 18, (4, 4), (2, 2), (0, 0, 0, 0)),   # overlapping 4 x 4
    (14, 15, (4, 4), (4, 4), (2, 1, 0, 3)),
    (9, 12, (3, 2), (2, 2), (0, 0, 0, 0)),    # row vectors under a window of another height
    (15, 16, (3, 4), (1, 4), (0, 0, 0, 0)),
    (12, 12, (5, 3), (2, 3), (1, 2, 3, 0)),   # run-time window
    (4, 4, (4, 4), (4, 4), (0, 0, 0, 0)),     # one output a plane
])
@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("offset", [0, 1])    # floats that the input lies off its allocation
def test_pool_kernel_forms(m, case, method, offset):
    H, W, kernel, stride, pad = case
    rng = np.random.default_rng(H * W + kernel[0])
    planes = 7
    x = rng.standard_normal((1, planes, H, W)).astype(np.float32)
    ref = oracle.pool2d(x, kernel, stride, pad=pad, method=method)
    OH, OW = ref.shape[2:]
    dx = m.to_device(np.concatenate([np.zeros(offset, np.float32), x.ravel()]))
    dy = m.DeviceBuffer(ref.nbytes)
    m.ops().mgpuPool2d(dx.ptr + 4 * offset, dy.ptr, 1, planes, H, W, OH, OW, kernel[0], kernel[1], *pad, stride[0], stride[1], method, None)
    got = m.to_host(dy, ref.shape, np.float32)
    m.check("pool")
    if method == 0:
        assert np.array_equal(got, ref)
    else:
        assert np.max(np.abs(got - ref)) <= 1e-6 * max(1.0, kernel[0] * kernel[1] / 9)


@pytest.mark.parametrize("width", [8191, 8192])
def test_conv_either_side_of_32_bit_addresses(m, width):
    """A gathered input of 4 GB less 128 KB, and of 4 GB: the ends of it, everything between is zero."""
    N, H, OC, stride = 16, 8192, 8, 16
    rng = np.random.default_rng(width)
    ends = rng.integers(-3, 4, (2, H, width)).astype(np.float32)
    w, b = rng.integers(-2, 3, (OC, 1, 3, 3)).astype(np.float32), rng.integers(-4, 5, OC).astype(np.float32)
    OH, OW = H // stride, (width - 1) // stride + 1
    x, out = m.DeviceBuffer(4 * N * H * width), m.DeviceBuffer(4 * N * OC * OH * OW)
    dw, db = m.to_device(w), m.to_device(b)
    m.runtime().mgpuMemset32(x.ptr, 0, N * H * width, None)
    for image, at in ((0, 0), (1, N - 1)):
        m.runtime().mgpuMemcpy(x.ptr + 4 * at * H * width, ends[image].ctypes.data, ends[image].nbytes, None)
    m.ops().mgpuConv2d(x.ptr, dw.ptr, db.ptr, out.ptr, None, N, 1, H, width, OC, 3, 3, OH, OW, 1, 1, 1, 1, stride, stride, 1, 1, False, False, None)
    got = m.to_host(out, (N, OC, OH, OW), np.float32)
    assert m.ops().mgpuOpsCheckDeviceStatus(None) == 0
    x.release()
    padded = np.pad(ends, ((0, 0), (1, stride), (1, stride)))
    ref = np.zeros((2, OC, OH, OW), np.float32) + b[None, :, None, None]
    for kh in range(3):
        for kw in range(3):
            ref += w[None, :, 0, kh, kw, None, None] * padded[:, None, kh:kh + stride * OH:stride, kw:kw + stride * OW:stride]
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[-1], ref[1])
    assert (got[1:-1] == b[None, :, None, None]).all()


def test_pool_special_values(m):
    x = np.zeros((1, 1, 4, 4), np.float32)
    x[0, 0, 0, 0] = -np.inf
    x[0, 0, 2, 2] = np.inf
    x[0, 0, 1, 3] = -0.0
    got = m.pool2d(x, (2, 2), (2, 2), method=0)
    ref = oracle.pool2d(x, (2, 2), (2, 2), method=0)
    assert np.array_equal(got, ref)


def test_bad_geometry_is_reported(m):
    x = np.zeros((1, 1, 4, 4), np.float32)
    rt, ops = m.runtime(), m.ops()
    buf = m.to_device(x)
    out = m.DeviceBuffer(64)
    rt.mgpuClearLastError()
    ops.mgpuPool2d(buf.ptr, out.ptr, 1, 1, 4, 4, 3, 3, 2, 2, 0, 0, 0, 0, 2, 2, 0, None)  # OH too large
    assert rt.mgpuGetLastError() != 0
    rt.mgpuClearLastError()
