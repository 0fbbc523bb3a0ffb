"""GPU: stems (at most 4 input channels) on the split-TF32 kernel: K folded, patches of image rows.

Shapes where the patch can go wrong: rows whose pitch is no multiple of 16 bytes, inputs that start
at any word, tiles of several small images, paddings wider than the filter's reach, strides up to 8,
filters of more than one K chunk, patches that need the large stages, one output column.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#       n  ic  h    w    oc  ks s  pad
CASES = [(2, 3, 32, 32, 64, 3, 1, 1), (1, 3, 33, 29, 64, 3, 1, 1), (9, 3, 7, 7, 32, 3, 1, 1), (5, 4, 5, 9, 70, 3, 2, 1),
         (2, 3, 64, 64, 64, 7, 2, 3), (1, 3, 61, 67, 40, 7, 2, 3), (3, 1, 28, 28, 20, 5, 1, 2), (2, 2, 19, 23, 130, 4, 3, 0),
         (1, 4, 70, 70, 64, 8, 8, 0), (1, 4, 96, 41, 16, 8, 5, 7), (2, 3, 40, 1, 64, 1, 1, 0), (4, 4, 17, 17, 64, 1, 4, 3),
         (1, 3, 20, 300, 200, 5, 1, 4), (17, 3, 3, 3, 8, 3, 1, 2)]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("shift", [0, 1])  # floats by which the input misses a 16-byte boundary
def test_stem_against_the_oracle(tb, torch_cuda, oracle, case, shift):
    torch = torch_cuda
    n, ic, h, w, oc, ks, s, pad = case
    rng = np.random.default_rng(h * 1000 + w)
    filt = rng.normal(0, 0.1, (oc, ic, ks, ks)).astype(np.float32)
    filt[rng.random(filt.shape) < 0.5] = 0
    x = rng.random((n, ic, h, w), dtype=np.float32) - 0.3
    f = tb.SparseFilter(filt, ic, oc, ks)
    oh, ow = tb.out_extent(h, ks, s, pad), tb.out_extent(w, ks, s, pad)
    # the words around the input are NaN: what lies outside the image must not be read as its edge
    room = torch.full((x.size + 64,), float("nan"), device="cuda")
    xin = room[32 + shift:32 + shift + x.size]
    xin.copy_(torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).reshape(-1))
    want = oracle.host_conv2d(x, filt, s, pad)
    for relu in (False, True):
        out = torch.full((n, oh, ow, oc), float("nan"), device="cuda")
        tb.sparse_conv2d_fused(f, xin, out, n, h, w, s, pad, variant=tb.VARIANT_TENSOR, relu=relu)
        torch.cuda.synchronize()
        f.check()
        got = out.cpu().numpy().transpose(0, 3, 1, 2)
        assert oracle.compare(got, np.maximum(want, 0) if relu else want)[0] == 0


def test_many_tiles_per_block(tb, torch_cuda, oracle):
    """Every block walks dozens of tiles: the ring of patches goes round many times."""
    torch = torch_cuda
    n, h = 8, 160
    for ks, s, pad, oc in ((3, 1, 1, 64), (7, 2, 3, 64), (3, 2, 1, 32)):
        rng = np.random.default_rng(ks)
        filt = rng.normal(0, 0.1, (oc, 3, ks, ks)).astype(np.float32)
        x = rng.random((n, 3, h, h), dtype=np.float32)
        f = tb.SparseFilter(filt, 3, oc, ks)
        oh = tb.out_extent(h, ks, s, pad)
        xin = torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).cuda()
        want = oracle.host_conv2d(x, filt, s, pad)
        outs = []
        for _ in range(4):
            out = torch.full((n, oh, oh, oc), float("nan"), device="cuda")
            tb.sparse_conv2d_fused(f, xin, out, n, h, h, s, pad, variant=tb.VARIANT_TENSOR, relu=True)
            outs.append(out)
        torch.cuda.synchronize()
        f.check()
        assert oracle.compare(outs[0].cpu().numpy().transpose(0, 3, 1, 2), np.maximum(want, 0))[0] == 0
        assert all(torch.equal(outs[0], o) for o in outs[1:])
