"""Batched malloc and free at the group counts where the launch changes form (the blocks scan the
groups, or a kernel before them does), by launch and by replayed graph, both backends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(torch, op, counts):
    t = np.zeros(len(counts), dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    t["op"], t["count"] = op, counts
    t["offset"] = np.concatenate([[0], np.cumsum(counts)[:-1]])
    return torch.from_numpy(t.view(np.uint8).copy()).cuda()


@pytest.mark.parametrize("n_groups", [1, 33, 4096, 4097, 6000])
@pytest.mark.parametrize("backend", ["runs", "queue"])
@pytest.mark.parametrize("form", ["launch", "graph"])
def test_blocks_are_disjoint_and_come_back(cuda, pbm_mod, n_groups, backend, form):
    torch, pbm = cuda, pbm_mod
    T, page = 1 << 16, 4096
    rng = np.random.default_rng(n_groups)
    counts = rng.integers(0, 3, n_groups) if n_groups > 100 else rng.integers(40, 70, n_groups)
    n = int(counts.sum())
    pool = pbm.Pool(T, page, materialize=True)
    getattr(pool, "malloc_init" if backend == "runs" else "qmalloc_init")()
    sizes_h = np.exp(rng.uniform(np.log(1), np.log(65536), n)).astype(np.int32)
    sizes_h[rng.random(n) < 0.05] = 0
    sizes = torch.from_numpy(sizes_h).cuda()
    ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
    both = torch.cat([_table(torch, pbm.OP_MALLOC, counts), _table(torch, pbm.OP_MFREE, counts)])
    half = n_groups * 16
    pre = "" if backend == "runs" else "q"
    if form == "graph":
        g = getattr(pool, pre + "malloc_graph")(both, n_groups, 2, sizes, ptrs, n, 5)
    base = torch.zeros(1, dtype=torch.int64).item() + pool.base_ptr
    for k in range(3):
        if form == "graph":
            g.replay()
        else:
            getattr(pool, pre + "malloc_batch")(both[:half], None, n_groups, sizes, ptrs, n, 5 + k, pbm.LAUNCH_PERSISTENT)
        p = ptrs.cpu().numpy()
        want = sizes_h > 0
        assert np.array_equal(p != 0, want)
        blk = np.maximum(16, 1 << np.ceil(np.log2(np.maximum(sizes_h, 1))).astype(np.int64))[want]
        off = p[want] - base
        assert (off >= 0).all() and (off + blk <= T * page).all() and (off % np.minimum(blk, page) == 0).all()
        order = np.argsort(off)
        assert (off[order][1:] >= (off + blk)[order][:-1]).all()
        if form == "graph":
            g.replay()
        else:
            getattr(pool, pre + "malloc_batch")(both[half:], None, n_groups, sizes, ptrs, n, 9, pbm.LAUNCH_PERSISTENT)
        assert not ptrs.any()
        if backend == "runs":
            assert pool.used() == 0 and pool.malloc_counts() == (0, 0)
        else:
            assert pool.qmalloc_counts()[2:] == (0, 0, 0)
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (3 * int((sizes_h > 0).sum()), 0, 3 * int((sizes_h > 0).sum()))
    if form == "graph":
        g.close()
    pool.close()


def test_batch_large_enough_for_paired_rounds(cuda, pbm_mod):
    """More requests than 64 for every warp of the launch, in groups that end inside a chunk, mallocs and
    frees in one batch: all served, blocks disjoint, everything back at the end."""
    torch, pbm = cuda, pbm_mod
    T, page = 1 << 18, 4096
    rng = np.random.default_rng(1)
    counts = rng.integers(900, 2000, 256)
    n = int(counts.sum())
    pool = pbm.Pool(T, page, materialize=True)
    pool.malloc_init()
    sizes_h = np.exp(rng.uniform(np.log(16), np.log(4096), 2 * n)).astype(np.int32)
    sizes = torch.from_numpy(sizes_h).cuda()
    ptrs = torch.zeros(2 * n, dtype=torch.int64, device="cuda")

    def table(op, offset):
        t = np.zeros(256, dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
        t["op"], t["count"] = op, counts
        t["offset"] = offset + np.concatenate([[0], np.cumsum(counts)[:-1]])
        return t

    def step(tables):
        t = np.concatenate(tables)
        if len(tables) == 2:                           # mallocs and frees by turns
            t = t.reshape(2, -1).T.reshape(-1)
        d = torch.from_numpy(np.ascontiguousarray(t).view(np.uint8).copy()).cuda()
        pool.malloc_batch(d, None, len(t), sizes, ptrs, 2 * n, 3, pbm.LAUNCH_PERSISTENT)

    step([table(pbm.OP_MALLOC, 0)])
    step([table(pbm.OP_MALLOC, n), table(pbm.OP_MFREE, 0)])
    p = ptrs.cpu().numpy()
    assert not p[:n].any() and p[n:].all()
    blk = np.maximum(16, 1 << np.ceil(np.log2(sizes_h[n:])).astype(np.int64))
    off = p[n:] - pool.base_ptr
    assert (off >= 0).all() and (off + blk <= T * page).all()
    order = np.argsort(off)
    assert (off[order][1:] >= (off + blk)[order][:-1]).all()
    step([table(pbm.OP_MFREE, n)])
    assert not ptrs.any() and pool.used() == 0 and pool.malloc_counts() == (0, 0)
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (2 * n, 0, 2 * n)
    pool.close()


def test_runs_found_by_a_sharing_warp_are_free_runs(cuda, pbm_mod, orc):
    """A nearly full pool, so most walks of a warp go on together for many rounds: every run
    granted was free, lies inside the pool and overlaps no other, and the failures took max_steps."""
    torch, pbm = cuda, pbm_mod
    T, page = 1 << 14, 4096
    pool = pbm.Pool(T, page, materialize=True)
    pool.malloc_init()
    pool.prefill(0.6, 3)
    before = np.unpackbits(pool.read_bitmap().view(np.uint8), bitorder="little")[:T].copy()
    n = 1024
    rng = np.random.default_rng(2)
    npg = rng.choice([1, 2, 4, 8, 16], n)
    sizes = torch.from_numpy((npg * page).astype(np.int32)).cuda()
    ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
    pool.malloc_batch(_table(torch, pbm.OP_MALLOC, np.array([n])), None, 1, sizes, ptrs, n, 7, pbm.LAUNCH_PERSISTENT,
                      max_steps=300)
    p = ptrs.cpu().numpy()
    ok = p != 0
    first = (p[ok] - pool.base_ptr) // page
    cover = before.astype(np.int32)
    for f, k in zip(first, npg[ok]):
        cover[f:f + k] += 1
    assert cover.max() == 1 and ok.sum() > 200 and (~ok).sum() > 50
    assert np.array_equal(np.unpackbits(pool.read_bitmap().view(np.uint8), bitorder="little")[:T], cover)
    s = pool.stats()
    assert s.failures == int((~ok).sum()) and s.steps >= 300 * s.failures
    pool.close()


@pytest.mark.parametrize("backend", ["runs", "queue"])
@pytest.mark.parametrize("max_steps", [1, 2, 40, 97, 512])
def test_overfull_pool_fails_within_the_bound(cuda, pbm_mod, backend, max_steps):
    """Many more pages asked for than there are: every request ends, after at most max_steps jumps, served
    ones hold blocks of their own, and freeing gives every page back."""
    torch, pbm = cuda, pbm_mod
    T, page, n = 4096, 4096, 3000
    pool = pbm.Pool(T, page, materialize=True)
    getattr(pool, "malloc_init" if backend == "runs" else "qmalloc_init")()
    rng = np.random.default_rng(5)
    npg = rng.choice([1, 2, 4, 8, 16], n)
    sizes = torch.from_numpy((npg * page).astype(np.int32)).cuda()
    ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
    run = getattr(pool, "malloc_batch" if backend == "runs" else "qmalloc_batch")
    run(_table(torch, pbm.OP_MALLOC, np.array([n])), None, 1, sizes, ptrs, n, 3, pbm.LAUNCH_PERSISTENT,
        max_steps=max_steps)
    p = ptrs.cpu().numpy()
    ok = p != 0
    first = (p[ok] - pool.base_ptr) // page
    cover = np.zeros(T, dtype=np.int32)
    for f, k in zip(first, npg[ok]):
        cover[f:f + k] += 1
    assert cover.max() == 1 and pool.used() == cover.sum()
    s = pool.stats()
    assert (s.successes, s.failures) == (int(ok.sum()), int((~ok).sum())) and s.failures > 0
    assert s.steps <= max_steps * n and s.steps >= max_steps * s.failures
    run(_table(torch, pbm.OP_MFREE, np.array([n])), None, 1, sizes, ptrs, n, 4, pbm.LAUNCH_PERSISTENT)
    assert not ptrs.any() and (pool.used() == 0 if backend == "runs" else pool.qmalloc_counts()[2:] == (0, 0, 0))
    pool.close()


@pytest.mark.parametrize("backend", ["runs", "queue"])
@pytest.mark.parametrize("n", [32, 64, 1000])
def test_serial_replay_frees_a_slot_once(cuda, pbm_mod, backend, n):
    """In the replay in request order a slot is empty once it is freed: a second group that frees the same slots
    frees nothing, and the blocks beside theirs stay."""
    torch, pbm = cuda, pbm_mod
    pool = pbm.Pool(1 << 12, 4096, materialize=True)
    pre = "" if backend == "runs" else "q"
    getattr(pool, pre + "malloc_init")()
    sizes = torch.full((2 * n,), 16, dtype=torch.int32, device="cuda")
    ptrs = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
    t = np.zeros(4, dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    t["op"] = [pbm.OP_MALLOC, pbm.OP_MFREE, pbm.OP_MFREE, pbm.OP_MFREE]
    t["count"] = [2 * n, n, n, n]
    table = torch.from_numpy(t.view(np.uint8).copy()).cuda()
    getattr(pool, pre + "malloc_batch")(table, None, 4, sizes, ptrs, 2 * n, 5, pbm.LAUNCH_SERIAL)
    s = pool.stats()
    assert (s.successes, s.failures, s.frees) == (2 * n, 0, n)
    p = ptrs.cpu().numpy()
    assert not p[:n].any() and np.unique(p[n:]).size == n and p[n:].all()
    rest = np.zeros(1, dtype=t.dtype)
    rest["op"], rest["count"], rest["offset"] = pbm.OP_MFREE, n, n
    getattr(pool, pre + "malloc_batch")(torch.from_numpy(rest.view(np.uint8).copy()).cuda(), None, 1, sizes, ptrs, 2 * n, 6,
                                        pbm.LAUNCH_SERIAL)
    assert pool.stats().frees == 2 * n and not ptrs.any()
    if backend == "runs":
        assert pool.used() == 0 and pool.malloc_counts() == (0, 0)
    else:
        assert pool.qmalloc_counts()[2:] == (0, 0, 0)
    pool.close()
