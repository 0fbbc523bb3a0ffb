"""GPU: host arrays through the page-locked ring, filters from the stream-ordered pool."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(tb, torch, n, c, h, w, seed):
    rng = np.random.default_rng(seed)
    filt = rng.normal(0, 0.1, (c, c, 1, 1)).astype(np.float32)
    filt[rng.random(filt.shape) < 0.5] = 0
    f = tb.SparseFilter(filt, c, c, 1)
    x = rng.random((n, c, h, w), dtype=np.float32) - 0.5
    xin = torch.from_numpy(np.ascontiguousarray(x.transpose(0, 2, 3, 1))).cuda()
    out = torch.empty(n, h, w, c, device="cuda")
    tb.sparse_conv2d(f, xin, out, n, h, w, 1, 0)
    torch.cuda.synchronize()
    return f, x, out.cpu().numpy().transpose(0, 3, 1, 2)


# bytes each way: below the staged size (256 KB), just above it with a ragged last chunk, exactly and
# just past eight chunks, more than the ring's 32 chunks of 512 KB (the ring is used again)
@pytest.mark.parametrize("n,c,h,w", [(1, 16, 63, 63), (1, 16, 65, 65), (1, 16, 128, 128), (1, 16, 129, 127), (3, 16, 317, 311), (2, 32, 512, 300)])
def test_ordinary_arrays_of_any_size(tb, torch_cuda, n, c, h, w):
    f, x, want = _case(tb, torch_cuda, n, c, h, w, 1)
    for _ in range(3):
        assert np.array_equal(tb.cuda_sparse_conv2d(x, f, n, h, w, 1, 0), want)
    tb.release_workspace()  # rings and threads are given back ...
    assert np.array_equal(tb.cuda_sparse_conv2d(x, f, n, h, w, 1, 0), want)  # ... and made again


def test_threads_share_the_ring(tb, torch_cuda):
    cases = [_case(tb, torch_cuda, 2, 16, 150 + 31 * i, 140, i) for i in range(4)]
    wrong = []

    def work(f, x, want):
        for _ in range(8):
            got = tb.cuda_sparse_conv2d(x, f, x.shape[0], x.shape[2], x.shape[3], 1, 0)
            if not np.array_equal(got, want):
                wrong.append(x.shape)

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_filters_made_and_closed_in_turn(tb, torch_cuda):
    """Memory a closed filter gave back is used by the next one; the filters that live keep theirs."""
    kept = [_case(tb, torch_cuda, 1, 64, 20, 20, s) for s in range(3)]
    for s in range(10):
        f, x, want = _case(tb, torch_cuda, 1, 32 + 16 * (s % 4), 24, 24, 100 + s)
        assert np.array_equal(tb.cuda_sparse_conv2d(x, f, 1, 24, 24, 1, 0), want)
        f.close()
        if s == 5:
            tb.release_workspace()
    for f, x, want in kept:
        assert np.array_equal(tb.cuda_sparse_conv2d(x, f, 1, 20, 20, 1, 0), want)


def test_large_upload_small_download(tb, torch_cuda):
    """Helpers that sleep while the layer computes must not leave the ring's lines in their caches: the copy engine
    then took 500 us for 4 MB.  The yardstick is the same call on page-locked arrays, which are copied directly
    (110 us): staging may add the time of a few memcpys, not multiples."""
    import time
    torch = torch_cuda
    rng = np.random.default_rng(0)
    f = tb.SparseFilter(rng.normal(0, 0.1, (4, 256, 1, 1)).astype(np.float32), 256, 4, 1)
    arrays = [rng.random((1, 256, 64, 64), dtype=np.float32) for _ in range(4)]
    pinned = [torch.from_numpy(a).pin_memory() for a in arrays]

    def median(inputs):
        times = []
        for i in range(80):
            t = time.perf_counter()
            tb.cuda_sparse_conv2d(inputs[i % 4], f, 1, 64, 64, 1, 0)
            times.append(time.perf_counter() - t)
        return sorted(times[20:])[30]

    assert median(arrays) < 3 * median([p.numpy() for p in pinned])
