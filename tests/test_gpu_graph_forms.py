"""Replays of one graph in several streams run one after the other, with the blocks scanning the
groups (one kernel, launched) and with a kernel before them (a graph launch)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_groups", [1, 256, 4096, 4097])
@pytest.mark.parametrize("walk", ["collab", "page", "word"])
def test_replays_in_turn_in_two_streams(cuda, pbm_mod, n_groups, walk):
    """ALLOC and FREE of the same slots, each replay in the other stream with no wait on the host:
    a replay that began before the one ahead of it ended would free pages not yet there."""
    torch, pbm = cuda, pbm_mod
    T, n, pairs = 1 << 20, 300_007, 20
    pool = pbm.Pool(T, 64)
    pool.prefill(0.5, 3)
    base = pool.used()
    arena = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    tab = np.zeros(2 * n_groups, dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    cut = np.linspace(0, n, n_groups + 1).astype(np.int64)
    tab["op"] = np.repeat([pbm.OP_ALLOC, pbm.OP_FREE], n_groups)
    tab["count"] = np.tile(np.diff(cut), 2)
    tab["offset"] = np.tile(cut[:-1], 2)
    d_tab = torch.from_numpy(tab.view(np.uint8).copy()).cuda()
    cfg = {"collab": pbm.walk_config(pbm.COLLAB_RW_BM, collab_width=64), "page": pbm.walk_config(pbm.RANDOM_WALK),
           "word": pbm.walk_config(pbm.RANDOM_WALK_BM)}[walk]
    g = pool.graph(cfg, d_tab, n_groups, 2, arena, n, 11)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k in range(2 * pairs):
        g.replay(streams[(k + k // 4) % 2].cuda_stream)   # now and then two in one stream
    torch.cuda.synchronize()
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (pairs * n, 0, pairs * n)
    assert pool.used() == base
    g.replay(streams[0].cuda_stream)
    g.close()
    torch.cuda.synchronize()
    ids = arena.cpu().numpy()
    assert np.unique(ids).size == n and ids.min() >= 0 and pool.used() == base + n
    pool.close()


@pytest.mark.parametrize("n_groups", [256, 4097])
def test_set_step_in_another_stream_than_the_replay(cuda, pbm_mod, n_groups):
    """set_step waits for the replay ahead of it, whatever their streams: every request of every replay
    is served once, with the groups scanned by the blocks and by a kernel before them."""
    torch, pbm = cuda, pbm_mod
    T, n, pairs = 1 << 22, 1_500_007, 12
    pool = pbm.Pool(T, 64)
    pool.prefill(0.5, 3)
    base = pool.used()
    arena = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    tab = np.zeros(2 * n_groups, dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    cut = np.linspace(0, n, n_groups + 1).astype(np.int64)
    tab["op"] = np.repeat([pbm.OP_ALLOC, pbm.OP_FREE], n_groups)
    tab["count"] = np.tile(np.diff(cut), 2)
    tab["offset"] = np.tile(cut[:-1], 2)
    d_tab = torch.from_numpy(tab.view(np.uint8).copy()).cuda()
    g = pool.graph(pbm.walk_config(pbm.COLLAB_RW_BM, collab_width=64), d_tab, n_groups, 2, arena, n, 11)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in range(pairs):
        g.replay(a.cuda_stream)
        g.set_step(1, b.cuda_stream)
        assert pool.used(b.cuda_stream) == base + n
        g.replay(b.cuda_stream)
        g.set_step(0, a.cuda_stream)
        assert pool.used(a.cuda_stream) == base
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (pairs * n, 0, pairs * n)
    g.close()
    pool.close()


@pytest.mark.parametrize("kind,n_groups", [("batch", 8), ("batch", 4097), ("malloc", 8)])
def test_refused_replay_is_none(cuda, pbm_mod, kind, n_groups):
    """A replay into a stream under capture is refused; the next replay runs the step that it would have run,
    and serves all of it."""
    torch, pbm = cuda, pbm_mod
    T, n = (1 << 20 if kind == "batch" else 1 << 17), 200_003
    pool = pbm.Pool(T, 64 if kind == "batch" else 4096, materialize=kind == "malloc")
    base = pool.used()
    tab = np.zeros(2 * n_groups, dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    cut = np.linspace(0, n, n_groups + 1).astype(np.int64)
    ops = (pbm.OP_ALLOC, pbm.OP_FREE) if kind == "batch" else (pbm.OP_MALLOC, pbm.OP_MFREE)
    tab["op"] = np.repeat(ops, n_groups)
    tab["count"] = np.tile(np.diff(cut), 2)
    tab["offset"] = np.tile(cut[:-1], 2)
    d_tab = torch.from_numpy(tab.view(np.uint8).copy()).cuda()
    if kind == "batch":
        arena = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        g = pool.graph(pbm.walk_config(pbm.COLLAB_RW_BM, collab_width=64), d_tab, n_groups, 2, arena, n, 11)
    else:
        pool.malloc_init()
        sizes = torch.full((n,), 64, dtype=torch.int32, device="cuda")
        ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
        g = pool.malloc_graph(d_tab, n_groups, 2, sizes, ptrs, n, 11)

    driver = ctypes.CDLL("libcuda.so.1")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()

    def refused():
        h, captured = ctypes.c_void_p(side.cuda_stream), ctypes.c_void_p()
        assert driver.cuStreamBeginCapture_v2(h, 1) == 0          # thread-local capture
        with pytest.raises(pbm.PbmError):
            g.replay(side.cuda_stream)
        driver.cuStreamEndCapture(h, ctypes.byref(captured))
        if captured:
            driver.cuGraphDestroy(captured)
        torch.cuda.synchronize()

    for _ in range(3):
        refused()
        g.replay()
        assert pool.used() > base
        refused()
        g.replay()
        assert pool.used() == base
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (3 * n, 0, 3 * n)
    g.close()
    pool.close()
