"""GPU: launches that are placed while the one before them drains (programmatic dependent launch).

Every kernel of a chain reads what the launch before it wrote and overwrites what an earlier one
read, so a missing wait shows as a difference between a run with a synchronisation behind every
launch and one without.  The kernels give the same bits on every run, so the two must be equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _filters(tb, shapes):
    rng = np.random.default_rng(11)
    made = []
    for ic, oc, ks, groups, variant in shapes:
        w = rng.normal(0, np.sqrt(6.0 / ((1 if groups > 1 else ic) * ks * ks)), (oc, 1 if groups > 1 else ic, ks, ks)).astype(np.float32)
        if groups == 1:
            w[rng.random(w.shape) < 0.7] = 0
        made.append((tb.SparseFilter(w, ic, oc, ks, groups=groups), ic, oc, ks, variant))
    return made


# (in, out, filter, groups, variant): every kernel that is launched this way behind every other kind;
# the last one leads back to the first layer's channels.  variant 2 list kernel, 4 split TF32, 5 split FP16.
SHAPES = [
    (4, 64, 3, 1, 4),        # folded stem
    (64, 64, 3, 1, 5),       # stacked tiles
    (64, 64, 3, 64, 0),      # depthwise through TMA
    (64, 300, 1, 1, 5),      # channels that end inside a tile
    (300, 300, 3, 300, 0),   # depthwise without TMA
    (300, 128, 1, 1, 2),     # list kernel
    (128, 512, 3, 1, 4),     # split TF32
    (512, 4, 3, 1, 5),       # K range over a cluster
]


@pytest.mark.parametrize("n,h", [(1, 7), (2, 28), (8, 56)])
@pytest.mark.parametrize("own_stream", [False, True])
def test_back_to_back_launches_wait_for_each_other(tb, torch_cuda, n, h, own_stream):
    torch = torch_cuda
    made = _filters(tb, SHAPES)
    torch.manual_seed(3)
    x = torch.rand(n, h, h, 4, device="cuda")
    bufs = [torch.empty(n * h * h * 512, device="cuda") for _ in range(2)]  # two buffers in turn: read, then overwritten

    def forward(sync, stream):
        cur = x
        for i, (f, ic, oc, ks, variant) in enumerate(made * 3):
            out = bufs[i & 1][:n * h * h * oc].view(n, h, h, oc)
            tb.sparse_conv2d_fused(f, cur, out, n, h, h, 1, ks // 2, variant=variant, relu=True, cuda_stream=stream)
            if sync:
                torch.cuda.synchronize()
            cur = out
        return cur

    stream = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
    torch.cuda.synchronize()
    want = forward(True, stream).clone()
    torch.cuda.synchronize()
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    with torch.cuda.stream(stream):
        for _ in range(5):
            for b in bufs:
                b.fill_(float("nan"))
            got = forward(False, stream).clone()  # (the copy is an ordinary launch behind the last one)
            stream.synchronize()
            assert torch.equal(got, want)
    for f, *_ in made:
        f.check()


@pytest.mark.parametrize("c,h", [(3, 33), (64, 56)])
def test_layout_conversions_behind_each_other(tb, torch_cuda, c, h):
    torch = torch_cuda
    n = 4
    src = torch.rand(n, c, h, h, device="cuda")
    a, b = torch.empty(n, h, h, c, device="cuda"), torch.empty_like(src)
    for _ in range(20):
        tb.nchw_to_nhwc(src, a, n, c, h, h)
        tb.nhwc_to_nchw(a, b, n, c, h, h)
        tb.nchw_to_nhwc(b, a, n, c, h, h)
    torch.cuda.synchronize()
    assert torch.equal(b, src) and torch.equal(a, src.permute(0, 2, 3, 1))


@pytest.mark.parametrize("oc", [30, 64])  # pooled one channel and four channels at a time
def test_chain_graph_equals_synchronised_layers(tb, torch_cuda, oc):
    torch = torch_cuda
    made = _filters(tb, [(16, oc, 3, 1, 0), (oc, oc, 3, 1, 0), (oc, 64, 1, 1, 0), (64, 64, 3, 64, 0), (64, oc, 3, 1, 0)])
    n, h = 2, 31
    x = torch.rand(n, h, h, 16, device="cuda") - 0.3
    chain = tb.LayerChain([(f, 1, ks // 2, True, 2 if i in (0, 2) else 0) for i, (f, _, _, ks, _) in enumerate(made)], n, h, h)
    cur = x
    for i, (f, ic, o, ks, _) in enumerate(made):
        hh = cur.shape[1]
        out = torch.empty(n, hh, hh, o, device="cuda")
        tb.sparse_conv2d_fused(f, cur, out, n, hh, hh, 1, ks // 2, relu=True)
        torch.cuda.synchronize()
        if i in (0, 2):
            out = torch.nn.functional.max_pool2d(out.permute(0, 3, 1, 2), 2).permute(0, 2, 3, 1).contiguous()
        cur = out
    want = cur.cpu().numpy()
    chain.run(x)
    assert np.array_equal(chain.download(), want)
    chain.capture(x)
    for _ in range(10):
        chain.replay()
    assert np.array_equal(chain.download(), want)
    chain.close()


@pytest.mark.parametrize("n,h,ic,oc,ks", [(4, 28, 65, 128, 5), (16, 7, 515, 515, 3), (2, 52, 315, 72, 3), (16, 28, 129, 130, 3)])
def test_list_kernel_spreads_over_the_device_back_to_back(tb, torch_cuda, n, h, ic, oc, ks):
    """A launch placed early must not double up on the SMs that were free first (1.4 to 1.6 times the time): a
    launch among others takes no longer than one that is waited for, which has the host's part on top."""
    torch = torch_cuda
    rng = np.random.default_rng(0)
    w = rng.normal(0, 0.05, (oc, ic, ks, ks)).astype(np.float32)
    w[rng.random(w.shape) < 0.875] = 0
    f = tb.SparseFilter(w, ic, oc, ks)
    x, y = torch.rand(n, h, h, ic, device="cuda"), torch.empty(n, h, h, oc, device="cuda")

    def per_launch(count):
        times = []
        for _ in range(11):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(count):
                tb.sparse_conv2d(f, x, y, n, h, h, 1, ks // 2, variant=tb.VARIANT_TILED, cuda_stream=torch.cuda.current_stream())
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) / count)
        return sorted(times)[5]

    tb.tune_sparse_conv2d(f, x, y, n, h, h, 1, ks // 2)
    per_launch(20)
    assert per_launch(20) < 1.1 * per_launch(1)
    f.close()
