"""GPU test of the stable compaction at the edges of its shares: rows of 32
flags, batches of 16 rows, a full grid of warps, and arrays that start off a
16-byte boundary. Exact: the indices are those of numpy's nonzero."""
import numpy as np
import pytest

import hptracing_b200 as H

pytestmark = pytest.mark.gpu

GRID = 148 * 8 * 8 * 16 * 32  # flags of one batch for every warp


@pytest.mark.parametrize("n", [1, 32, 33, 511, 513, 4097, GRID - 1, GRID, GRID + 1, 2 * GRID + 33, 8192 * 4096])
@pytest.mark.parametrize("density", [0.0, 0.03, 0.6, 1.0])
def test_compact_edges(built, n, density):
    torch = pytest.importorskip("torch")
    if H.device_count() == 0 or not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(n)
    flags = (rng.random(n, np.float32) < density).astype(np.int32) * rng.integers(1, 1 << 30, n, np.int32)
    off = n % 4  # the flags start off a 16-byte boundary
    dev = torch.zeros(n + off, dtype=torch.int32, device="cuda")
    dev[off:] = torch.from_numpy(flags).cuda()
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    count = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert H.lib().hpt_compact_noalloc(dev.data_ptr() + 4 * off, n, out.data_ptr(), count.data_ptr(), st) == 0
    want = np.flatnonzero(flags).astype(np.int32)
    assert int(count) == len(want)
    got = out.cpu().numpy()
    assert np.array_equal(got[:len(want)], want)
    assert (got[len(want):] == -1).all()


def test_compact_in_a_graph(built):
    """Captured and replayed on new flags (the scatter pass is launched with
    programmatic stream serialisation)."""
    torch = pytest.importorskip("torch")
    if H.device_count() == 0 or not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 100_003
    flags = torch.zeros(n, dtype=torch.int32, device="cuda")
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    count = torch.full((1,), -1, dtype=torch.int32, device="cuda")

    def call():
        st = torch.cuda.current_stream().cuda_stream
        assert H.lib().hpt_compact_noalloc(flags.data_ptr(), n, out.data_ptr(), count.data_ptr(), st) == 0

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for seed in (1, 2):
        f = (np.random.default_rng(seed).random(n) < 0.5).astype(np.int32)
        flags.copy_(torch.from_numpy(f))
        graph.replay()
        want = np.flatnonzero(f).astype(np.int32)
        assert int(count) == len(want)
        assert np.array_equal(out.cpu().numpy()[:len(want)], want)
