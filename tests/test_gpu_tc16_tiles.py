"""GPU: the split-FP16 tensor-core kernel at the edges of its tile geometries -- strides 1 to 4 (input
phases), stacked tiles (at most 64 channels), K ranges cut over a cluster, tiles of consecutive
pixels, of whole padded rows and of 8-column blocks with several images, channel counts around
the tiles' -- its passes for activations outside FP16's window, and its error against 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # n, ic, h, w, oc, ks, stride, pad
    (1, 64, 56, 56, 64, 3, 1, 1),      # stacked, small tiles
    (2, 32, 65, 33, 63, 3, 2, 1),      # stacked, stride 2, one channel short
    (3, 8, 17, 19, 65, 3, 3, 1),       # one channel past a stacked tile, stride 3
    (2, 12, 31, 30, 130, 5, 4, 2),     # stride 4, 5x5, partial K chunk and channel tile
    (1, 512, 14, 14, 256, 3, 1, 1),    # K range over a cluster of 8
    (1, 100, 7, 7, 64, 3, 1, 1),       # stacked and cut into slices of unequal length
    (9, 256, 7, 7, 128, 3, 1, 1),      # several images per tile, the last tile with one
    (8, 1024, 13, 13, 255, 1, 1, 0),   # 1x1, 255 channels, slices
    (2, 64, 9, 300, 96, 3, 1, 1),      # wide and flat
    (2, 64, 300, 5, 40, 3, 1, 1),      # tall and thin
    (5, 32, 28, 28, 128, 1, 2, 0),     # strided projection: one phase has a tap
    (4, 16, 1, 1, 16, 1, 1, 0),        # one pixel per image
    (2, 40, 12, 12, 260, 7, 1, 3),     # 7x7
]


def _run(tb, torch, f, x, stride, pad, relu):
    n, ic, h, w = x.shape
    oh, ow = tb.out_extent(h, f.kernel_size_, stride, pad), tb.out_extent(w, f.kernel_size_, stride, pad)
    xin = torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).cuda()
    out = torch.full((n, oh, ow, f.out_channel_), float("nan"), device="cuda")
    tb.sparse_conv2d_fused(f, xin, out, n, h, w, stride, pad, variant=tb.VARIANT_TENSOR16, relu=relu)
    torch.cuda.synchronize()
    f.check()
    return out.cpu().numpy().transpose(0, 3, 1, 2)


def _layer(case, seed):
    n, ic, h, w, oc, ks, stride, pad = case
    rng = np.random.default_rng(seed)
    filt = rng.normal(0, 0.05, (oc, ic, ks, ks)).astype(np.float32)
    filt[rng.random(filt.shape) < 0.8] = 0
    return filt, rng.random((n, ic, h, w), dtype=np.float32) - 0.3


@pytest.mark.parametrize("case", CASES, ids=lambda c: "n%d_ic%d_%dx%d_oc%d_k%d_s%d_p%d" % c)
def test_tile_geometries(tb, torch_cuda, oracle, case):
    n, ic, h, w, oc, ks, stride, pad = case
    filt, x = _layer(case, sum(case))
    f = tb.SparseFilter(filt, ic, oc, ks)
    want = oracle.host_conv2d(x, filt, stride, pad, threads=True, skip_zero=True)
    got = _run(tb, torch_cuda, f, x, stride, pad, False)
    assert not np.isnan(got).any(), "output elements were left unwritten"
    assert oracle.compare(got, want)[0] == 0
    again = _run(tb, torch_cuda, f, x, stride, pad, False)
    assert np.array_equal(got, again)  # slices are added in slice order
    assert oracle.compare(_run(tb, torch_cuda, f, x, stride, pad, True), np.maximum(want, 0))[0] == 0
    f.close()


@pytest.mark.parametrize("case", [(2, 96, 20, 20, 72, 3, 1, 1), (1, 64, 24, 24, 48, 3, 2, 1), (1, 512, 14, 14, 128, 1, 1, 0)],
                         ids=lambda c: "n%d_ic%d_%dx%d_oc%d_k%d_s%d_p%d" % c)
def test_activations_outside_the_window(tb, torch_cuda, oracle, case):
    """All large, all tiny, and 2^-30 beside 2^13 in one tile: the bar of the path (1e-4 relative,
    1e-5 absolute), with the absolute floor scaled like the data -- and for the mixed input like
    the large values, whose FP32 rounding in the oracle itself is of that size."""
    n, ic, h, w, oc, ks, stride, pad = case
    filt, x = _layer(case, 7)
    f = tb.SparseFilter(filt, ic, oc, ks)
    for scale in (2.0 ** 14, 2.0 ** 60, 2.0 ** -12, 2.0 ** -70):
        y = (x * np.float32(scale)).astype(np.float32)
        want = oracle.host_conv2d(y, filt, stride, pad, threads=True)
        got = _run(tb, torch_cuda, f, y, stride, pad, False)
        assert oracle.compare(got / np.float32(scale), want / np.float32(scale))[0] == 0, scale
    # channels of very different magnitude; an output that reads only the tiny ones keeps its
    # relative accuracy although its tile holds the large ones (three bands of 16 binades)
    mixed = x.copy()
    mixed[:, : ic // 2] *= np.float32(2.0 ** 13)
    mixed[:, ic // 2:] *= np.float32(2.0 ** -18)
    split = filt.copy()
    split[: oc // 2, ic // 2:] = 0      # reads the large channels
    split[oc // 2:, : ic // 2] = 0      # reads the tiny ones
    g = tb.SparseFilter(split, ic, oc, ks)
    want = oracle.host_conv2d(mixed, split, stride, pad, threads=True)
    got = _run(tb, torch_cuda, g, mixed, stride, pad, False)
    for part, s in ((slice(0, oc // 2), 2.0 ** 13), (slice(oc // 2, oc), 2.0 ** -18)):
        assert oracle.compare(got[:, part] / np.float32(s), want[:, part] / np.float32(s))[0] == 0
    # an infinity spoils the outputs that read it, and no others
    spiked = x.copy()
    spiked[0, 3, 5, 5] = np.inf
    got = _run(tb, torch_cuda, f, spiked, stride, pad, False)
    want = oracle.host_conv2d(x, filt, stride, pad, threads=True)
    far = np.ones(got.shape, bool)
    far[0, :, max(0, 5 + pad - ks) // stride: (5 + pad) // stride + 1, max(0, 5 + pad - ks) // stride: (5 + pad) // stride + 1] = False
    reads = np.zeros(got.shape, bool)  # outputs with a nonzero weight on the infinity
    for r in range(ks):
        for s in range(ks):
            p, q = 5 + pad - r, 5 + pad - s
            if p % stride == 0 and q % stride == 0 and 0 <= p // stride < got.shape[2] and 0 <= q // stride < got.shape[3]:
                reads[0, :, p // stride, q // stride] |= filt[:, 3, r, s] != 0
    assert reads.any() and not np.isfinite(got[reads]).any()
    assert oracle.compare(got[far], want[far])[0] == 0
    f.close()
    g.close()


@pytest.mark.parametrize("case", [(1, 512, 14, 14, 128, 1, 1, 0), (1, 100, 7, 7, 64, 3, 1, 1), (1, 512, 7, 7, 256, 3, 1, 1),  # cut over clusters
                                  (16, 32, 40, 40, 72, 3, 1, 1), (16, 32, 56, 56, 48, 3, 1, 1)],                          # whole tiles, plain and stacked
                         ids=lambda c: "n%d_ic%d_%dx%d_oc%d_k%d_s%d_p%d" % c)
@pytest.mark.parametrize("xe,we", [(112, 0), (126, -20), (-100, -20), (-60, -60), (-110, 40)])
def test_scales_at_the_ends_of_fp32(tb, torch_cuda, oracle, case, xe, we):
    """Activations x 2^xe, weights x 2^we: the results are normal FP32 numbers (or just below them), so they
    have to be those of the unscaled layer times 2^(xe + we), to the bar of the path.  On the way the
    kernel's sums, at the scale of its FP16 operands, lie up to 2^150 away from them.  (The smallest results,
    about 2^-122, are rounded to multiples of 2^-149: 2e-8 of the layer's own scale.)"""
    filt, x = _layer(case, 5)
    want = oracle.host_conv2d(x, filt, case[6], case[7], threads=True)
    f = tb.SparseFilter(np.ldexp(filt, we), case[1], case[4], case[5])
    got = _run(tb, torch_cuda, f, np.ldexp(x, xe), case[6], case[7], False)
    assert np.isfinite(got).all()
    assert oracle.compare(np.ldexp(got.astype(np.float64), -xe - we).astype(np.float32), want)[0] == 0
    f.close()


# (n, ic, h, w, oc, ks, stride, pad) and the K steps of 32 channels that a partial sum may hold
PARTIALS = [
    ((16, 256, 14, 14, 1024, 1, 1, 0), 4),   # 1x1
    ((2, 128, 20, 20, 128, 3, 1, 1), 4),     # larger filter, few tiles
    ((2, 64, 57, 57, 96, 3, 2, 1), 4),       # strided
    ((2, 512, 20, 20, 256, 1, 1, 0), 2),     # 1x1, few tiles: what a slice of the K range would hold
    ((2, 512, 40, 40, 256, 1, 2, 0), 2),
    ((2, 256, 10, 10, 1024, 1, 1, 0), 1),
]


@pytest.mark.parametrize("case,steps", PARTIALS, ids=lambda c: "n%d_ic%d_%dx%d_oc%d_k%d_s%d_p%d" % c if isinstance(c, tuple) else str(c))
def test_error_against_64_bits(tb, torch_cuda, case, steps):
    """The tensor core truncates its adds, so the error of a partial sum grows with its MMAs, six per K step.
    An add loses half a unit in the last place on average, 0.72 * 2^-24 of the sum it leaves (the mean over a
    binade), and the sums of a partial are half its final one on average: 0.36 * 2^-24 per MMA.  To that come the
    roundings to nearest of the operands' halves and of the adds outside, a few 2^-25.  Relative, 2-norm."""
    torch = torch_cuda
    n, ic, h, w, oc, ks, stride, pad = case
    rng = np.random.default_rng(5)
    filt = rng.normal(0, 0.05, (oc, ic, ks, ks)).astype(np.float32)
    filt[rng.random(filt.shape) < 0.8] = 0
    x = rng.random((n, ic, h, w), dtype=np.float32)
    x[rng.random(x.shape) < 0.5] = 0
    f = tb.SparseFilter(filt, ic, oc, ks)
    got = _run(tb, torch, f, x, stride, pad, False)
    cols = torch.nn.functional.unfold(torch.from_numpy(x).cuda().double(), ks, padding=pad, stride=stride)
    want = (torch.from_numpy(filt).cuda().double().reshape(oc, -1) @ cols).cpu().numpy().reshape(got.shape)
    error = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert error < 0.36 * 2.0 ** -24 * 6 * steps + 3 * 2.0 ** -25, error
    f.close()


@pytest.mark.parametrize("channels", [64, 160])  # stacked tiles, plain ones
@pytest.mark.parametrize("top,bottom", [(13, -18), (13, -19), (13, -35), (-9, -40), (-9, -57), (100, 69), (-60, -108)])
def test_bands_of_activations(tb, torch_cuda, channels, top, bottom):
    """Activations of every binade from 2^top down to 2^bottom, each output reading one of them: the bands --
    two for 32 binades, three below -- keep every activation's 22 bits down to 49 binades below the largest
    (operand halves rounded to nearest at 11 bits each: 2^-22 of activation and of weight, the product of the
    remainders left out 2^-22, and one truncated add of the three products 2^-23)."""
    rng = np.random.default_rng(0)
    weights = rng.uniform(0.5, 2, channels).astype(np.float32)
    filt = np.zeros((channels, channels, 1, 1), np.float32)
    filt[np.arange(channels), np.arange(channels), 0, 0] = weights
    shape = (2, channels, 40, 33)
    x = np.ldexp(rng.uniform(1, 2, shape), rng.integers(bottom, top + 1, shape)).astype(np.float32)
    x[rng.random(shape) < 0.3] = 0
    x = x * rng.choice(np.float32([-1, 1]), shape)
    f = tb.SparseFilter(filt, channels, channels, 1)
    got = _run(tb, torch_cuda, f, x, 1, 0, False).astype(np.float64)
    want = x.astype(np.float64) * weights.reshape(1, -1, 1, 1)
    assert (np.abs(got - want) <= 4 * 2.0 ** -22 * np.abs(want)).all()
    f.close()


@pytest.mark.parametrize("oc,sparsity", [(17, 0.875), (16, 0.8), (33, 0.8)])
def test_untuned_choice_on_odd_channel_counts(tb, torch_cuda, oc, sparsity):
    """Channel counts that are no multiple of four are stored value by value, which the estimate behind the
    untuned choice has to know: the chosen kernel is the faster one, or not more than a quarter slower."""
    torch = torch_cuda
    n, h, ic = 4, 112, 32
    rng = np.random.default_rng(0)
    filt = rng.normal(0, 0.05, (oc, ic, 3, 3)).astype(np.float32)
    filt[rng.random(filt.shape) < sparsity] = 0
    f = tb.SparseFilter(filt, ic, oc, 3)
    x, y = torch.rand(n, h, h, ic, device="cuda"), torch.empty(n, h, h, oc, device="cuda")

    def per_launch(variant):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                tb.sparse_conv2d(f, x, y, n, h, h, 1, 1, variant=variant, cuda_stream=torch.cuda.current_stream())
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times)[3]

    kernels = {v: per_launch(v) for v in (tb.VARIANT_TILED, tb.VARIANT_TENSOR16)}
    assert kernels[tb.auto_choice(f, n, h, h, 1, 1)] < 1.25 * min(kernels.values())
    f.close()


def test_a_tiny_image_beside_ordinary_ones(tb, torch_cuda, oracle):
    """One maximum per CTA decides about its scales, so an image of activations near 1e-6 may be computed at the
    scale of the images that share its CTA.  Then each activation is held to 2^-29 (half the spacing of FP16's
    subnormal numbers, 2^-25, at the scale 16), and an output to the sum of its |weights| times that, the
    rounding of the tiny sum itself aside; the ordinary images keep the bar of the path."""
    n, ic, h, oc = 48, 64, 28, 128  # several tiles per CTA
    filt, x = _layer((n, ic, h, h, oc, 3, 1, 1), 11)
    x[17] *= np.float32(2.0 ** -20)
    f = tb.SparseFilter(filt, ic, oc, 3)
    got = _run(tb, torch_cuda, f, x, 1, 1, False)
    want = oracle.host_conv2d(x, filt, 1, 1, threads=True, skip_zero=True)
    rest = np.arange(n) != 17
    assert oracle.compare(got[rest], want[rest])[0] == 0
    bound = np.abs(filt).sum((1, 2, 3)).reshape(-1, 1, 1) * 2.0 ** -29 + 1e-5 * np.abs(want[17]).max()
    assert (np.abs(got[17] - want[17]) <= bound).all()
    f.close()


@pytest.mark.parametrize("n,h,w,ks,pad", [(2 ** 31 - 300, 1, 1, 1, 0), (1, 2 ** 31 - 300, 1, 3, 1), (1, 1, 2 ** 31 - 300, 3, 1)])
def test_shapes_past_32_bit_coordinates_are_refused(tb, torch_cuda, n, h, w, ks, pad):
    """Refused on the host, before anything is launched: the last tile would reach past 2^31."""
    f = tb.SparseFilter(np.ones((8, 8, ks, ks), np.float32), 8, 8, ks)
    buf = torch_cuda.zeros(64, device="cuda")
    with pytest.raises(tb.TetrisError, match="split-FP16"):
        tb.sparse_conv2d(f, buf, buf, n, h, w, 1, pad, variant=tb.VARIANT_TENSOR16)
    f.close()
