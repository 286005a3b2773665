"""The forms that the allocation kernels take for whole warps and blocks, at the
sizes where they can go wrong, against the oracle's sequential replay or the
walk's own probe sequence.  All comparisons are of whole numbers, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

A, C, M31 = 1103515245, 12345, 0x7FFFFFFF


def _probe_pages(orc, S, reqs, steps, n_pages):
    """The page of probe `steps[i]` of request reqs[i]'s walk."""
    x = np.array([orc.seed(S, int(r)) for r in reqs], dtype=np.int64)
    out = np.zeros(len(reqs), dtype=np.int64)
    for k in range(1, int(steps.max()) + 1):
        x = (A * x + C) & M31
        out = np.where(steps == k, (x * n_pages) >> 31, out)
    return out


@pytest.mark.parametrize("max_steps", [1, 3, 4, 7, 8, 35, 36, 131, 132, 133, 4096])
@pytest.mark.parametrize("T,occ", [(8192, 0.5), (65536 + 17, 0.97), (1 << 20, 0.999)])
def test_page_walk_of_one_request_is_the_sequential_walk(cuda, pbm_mod, orc, T, occ, max_steps):
    """Alone in its launch a walk meets no race: id, steps and bitmap equal the replay's,
    also where the bound cuts the look-ahead short."""
    torch, pbm = cuda, pbm_mod
    pool = pbm.Pool(T, 64)
    cfg = pbm.walk_config(pbm.RANDOM_WALK, max_steps=max_steps)
    ids = torch.empty(1, dtype=torch.int32, device="cuda")
    steps = torch.empty(1, dtype=torch.int32, device="cuda")
    for S in range(8):
        pool.prefill(occ, 5)
        words = orc.bernoulli_bitmap(T, occ, 5)
        pool.alloc(cfg, 1, S, ids, steps)
        e_ids, e_steps = orc.replay_alloc(words, T, pbm.RANDOM_WALK, 1, S, max_steps=max_steps)
        assert (ids.item(), steps.item()) == (int(e_ids[0]), int(e_steps[0]))
        assert np.array_equal(pool.read_bitmap(), words)
    pool.close()


@pytest.mark.parametrize("form", ["alloc", "claim", "batch"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 3001])
@pytest.mark.parametrize("occ", [0.05, 0.9, 0.985])
def test_page_walks_end_at_their_own_probe(cuda, pbm_mod, orc, form, n, occ):
    """Whole warps walking together: every request holds a page of its own, taken at the
    probe of its own sequence that its step count names."""
    torch, pbm = cuda, pbm_mod
    T, S = 400000 + 7, 77
    pool = pbm.Pool(T, 64, materialize=form == "claim")
    pool.prefill(occ, 9)
    before = pool.read_bitmap()
    ids = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    steps = torch.full((n,), -9, dtype=torch.int32, device="cuda")
    cfg = pbm.walk_config(pbm.RANDOM_WALK)
    if form == "alloc":
        pool.alloc(cfg, n, S, ids, steps)
    elif form == "claim":
        pool.claim_write_free(n, S, ids, steps, hold=True)
    else:
        pool.batch(cfg, None, pbm.groups_array([(pbm.OP_ALLOC, n, 0)]), 1, ids, n, S, pbm.LAUNCH_PERSISTENT,
                   steps=steps)
    got, st = ids.cpu().numpy(), steps.cpu().numpy()
    chk = pool.check(ids, n)
    assert (chk.n_ok, chk.n_failed, chk.n_duplicates, chk.n_not_marked, chk.n_out_of_range) == (n, 0, 0, 0, 0)
    assert chk.used_pages == orc.used_pages(before, T) + n
    assert np.array_equal(got, _probe_pages(orc, S, range(n), st, T))
    stats = pool.stats()
    assert (stats.successes, stats.failures, stats.steps) == (n, 0, int(st.sum()))
    pool.close()


@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 1023, 1024, 4099, 700001])
@pytest.mark.parametrize("shift,merge", [(0, 0), (1, 0), (0, 1)])
def test_free_clears_exactly_the_listed_pages(cuda, pbm_mod, n, shift, merge):
    """Runs of neighbours in one word, repeated pages, and ids that name no page, from lists on
    and off a 16-byte boundary."""
    torch, pbm = cuda, pbm_mod
    T = 1 << 20
    rng = np.random.default_rng(n + 7 * shift)
    ids = np.repeat(rng.integers(0, T, n // 3 + 1), 3)[:n] + np.arange(n) % 3
    ids[rng.random(n) < 0.1] = -1
    ids[rng.random(n) < 0.05] = T + 5
    ids = ids.astype(np.int32)
    d = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
    d[shift:shift + n] = torch.from_numpy(ids).cuda()
    pool = pbm.Pool(T, 64)
    pool.prefill(1.0, 1)
    pool.free(pbm.walk_config(pbm.RANDOM_WALK_BM, free_merge=merge), n, d[shift:])
    bits = np.ones(T, dtype=np.uint8)
    valid = ids[(ids >= 0) & (ids < T)]
    bits[valid] = 0
    assert np.array_equal(pool.read_bitmap(), np.packbits(bits, bitorder="little").view(np.uint32))
    assert pool.stats().frees == len(valid)
    pool.close()


@pytest.mark.parametrize("n", [1, 31, 256, 257, 5000, 160000])
@pytest.mark.parametrize("block_size", [64, 256])
def test_free_list_serves_blocks_in_release_order(cuda, pbm_mod, n, block_size):
    """Gets come out in list order, call by call, across the ring's wrap; a call that asks for more
    than the list holds gets exactly the rest; ids that name no page are skipped by a put."""
    torch, pbm = cuda, pbm_mod
    T = max(64, 2 * n + n // 2 + 1)
    pool = pbm.Pool(T, 64)
    cfg = pbm.walk_config(pbm.LINKED_LIST, block_size=block_size)
    queue = [np.arange(T)]                              # what each put brought, oldest first
    out = []
    for k in range(6):
        ids = torch.empty(n, dtype=torch.int32, device="cuda")
        pool.alloc(cfg, n, 0, ids)
        got = ids.cpu().numpy()
        flat = np.concatenate(queue)
        want, rest = flat[:n], flat[n:]
        assert np.array_equal(np.sort(got[got >= 0]), np.sort(want)) and (got < 0).sum() == n - len(want)
        out.append(got[got >= 0])
        queue = [rest]
        if k >= 1:                                      # give the older of the two held batches back
            back = out.pop(0)
            # puts of one call have no order among themselves: keep the next gets to whole batches
            padded = np.full(2 * len(back) + 1, -1, dtype=np.int32)
            padded[1::2] = back
            padded[0] = T + 3
            pool.free(cfg, len(padded), torch.from_numpy(padded).cuda())
            queue.append(back)
            if len(np.concatenate(queue[:1])) < n:      # the next call would split a batch
                break
    st = pool.stats()
    assert st.frees == st.successes - sum(len(x) for x in out)
    more = torch.empty(T, dtype=torch.int32, device="cuda")
    pool.alloc(cfg, T, 0, more)
    left = T - sum(len(x) for x in out)
    assert int((more >= 0).sum()) == left
    chk = pool.check(more, T)
    assert (chk.n_duplicates, chk.n_not_marked, chk.used_pages) == (0, 0, T)
    pool.close()


@pytest.mark.parametrize("T,occ", [(40, 0.2), (96, 0.5), (1000, 0.9), (8192 + 5, 0.5), (1 << 16, 0.99), (1 << 18, 0.02)])
@pytest.mark.parametrize("n", [1, 2, 31, 32])
def test_clock_sweep_of_one_warp_takes_the_next_free_pages(cuda, pbm_mod, orc, T, occ, n):
    """Launches of one warp, one after the other and round the pool: together they take the free pages
    in sweep order and pass none, as the one-thread sweep does; steps add up to the positions passed."""
    torch, pbm = cuda, pbm_mod
    words = orc.bernoulli_bitmap(T, occ, 4)
    bits = np.unpackbits(words.view(np.uint8), bitorder="little")[:T]
    order = np.nonzero(bits == 0)[0]
    pool = pbm.Pool(T, 64)
    pool.prefill(occ, 4)
    cfg = pbm.walk_config(pbm.SINGLE_CLOCK, max_steps=1 << 20)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    steps = torch.empty(n, dtype=torch.int32, device="cuda")
    taken = 0
    for S in range(min(6, len(order) // n)):
        pool.alloc(cfg, n, S, ids, steps)
        want = order[taken:taken + n]
        assert np.array_equal(ids.cpu().numpy(), want)
        first = order[taken - 1] + 1 if taken else 0
        assert int(steps.sum()) == want[-1] + 1 - first
        taken += n
    # free what was taken: the arm, past it, reaches those pages again after the rest of the pool
    if taken:
        back = torch.from_numpy(order[:taken].astype(np.int32)).cuda()
        pool.free(cfg, taken, back)
        rest = len(order) - taken + taken
        got = []
        for S in range(rest // n):
            pool.alloc(cfg, n, 50 + S, ids)
            got.append(ids.cpu().numpy())
            if S >= 40:
                break
        got = np.concatenate(got)
        assert np.array_equal(got, np.concatenate([order[taken:], order[:taken]])[:len(got)])
    pool.close()


@pytest.mark.parametrize("T,occ,n", [(1 << 16, 0.97, 1900), (1 << 20, 0.9, 50000), (1 << 20, 0.0, 300000), (3000, 0.0, 2999),
                                     (100000, 0.5, 60000)])
@pytest.mark.parametrize("max_steps", [1, 5, 4096])
def test_clock_sweep_of_many_warps(cuda, pbm_mod, orc, T, occ, n, max_steps):
    """Pages are distinct and were free; no request reports more than max_steps positions; with room and a
    generous bound all are served, and a launch never examines more than its bound allows."""
    torch, pbm = cuda, pbm_mod
    pool = pbm.Pool(T, 64)
    pool.prefill(occ, 3)
    before = pool.read_bitmap()
    free = T - orc.used_pages(before, T)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    steps = torch.empty(n, dtype=torch.int32, device="cuda")
    pool.alloc(pbm.walk_config(pbm.SINGLE_CLOCK, max_steps=max_steps), n, 1, ids, steps)
    got, st = ids.cpu().numpy(), steps.cpu().numpy()
    chk = pool.check(ids, n)
    assert (chk.n_duplicates, chk.n_not_marked, chk.n_out_of_range) == (0, 0, 0)
    assert chk.used_pages == T - free + chk.n_ok
    h = got[got >= 0]
    assert not ((before[h >> 5] >> (h & 31).astype(np.uint32)) & 1).any()
    assert st.max() <= max_steps and st.min() >= 1 and (st[got < 0] == max_steps).all()
    if max_steps == 4096:
        assert chk.n_ok == min(n, free)
    pool.free(pbm.walk_config(pbm.SINGLE_CLOCK), n, ids)
    assert np.array_equal(pool.read_bitmap(), before)
    pool.close()


@pytest.mark.parametrize("threads", [1, 2])
@pytest.mark.parametrize("n_streams", [2, 3, 11])
def test_budget_launches_side_by_side(cuda, pbm_mod, n_streams, threads):
    """Fail-fast launches of one pool in several streams, from one host thread or two, each asking for more
    pages than are free: every request is answered, no page goes to two holders, none is lost."""
    import threading
    torch, pbm = cuda, pbm_mod
    T, n, rounds = 1 << 20, 90000, 30
    pool = pbm.Pool(T, 64)
    pool.prefill(0.9, 5)
    before = pool.read_bitmap()
    base = pool.used()
    cfg = pbm.walk_config(pbm.COLLAB_RW_BM, fail_fast=1, max_steps=64)
    streams = [torch.cuda.Stream() for _ in range(n_streams)]
    for k in range(rounds):
        ids = [torch.full((n,), -9, dtype=torch.int32, device="cuda") for _ in streams]
        torch.cuda.synchronize()

        def issue(part):
            for j in range(part, n_streams, threads):
                pool.alloc(cfg, n, 100 * k + j, ids[j], stream=streams[j].cuda_stream)

        ts = [threading.Thread(target=issue, args=(i,)) for i in range(threads)]
        [x.start() for x in ts]
        [x.join() for x in ts]
        torch.cuda.synchronize()
        got = torch.cat(ids).cpu().numpy()
        held = got[got >= 0]
        assert (got >= -1).all() and np.unique(held).size == held.size
        assert not ((before[held >> 5] >> (held & 31).astype(np.uint32)) & 1).any()
        assert pool.used() == base + held.size
        for j, s in enumerate(streams):
            pool.free(cfg, n, ids[j], stream=s.cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(pool.read_bitmap(), before)
    pool.close()


def test_budget_launches_under_capture(cuda, pbm_mod):
    """More captured fail-fast launches than there are workspaces for them, replayed beside launches that are
    not captured: the first hand the free pages out in order, all answer every request."""
    torch, pbm = cuda, pbm_mod
    T, n, m = 1 << 16, 40000, 30
    pool = pbm.Pool(T, 64)
    pool.prefill(0.6, 5)   # pages are listed in a pool at least half full
    before = pool.read_bitmap()
    free = np.nonzero(np.unpackbits(before.view(np.uint8), bitorder="little")[:T] == 0)[0]
    cfg = pbm.walk_config(pbm.COLLAB_RW_BM, fail_fast=1)
    ids = torch.full((m, n), -9, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for k in range(m):
            pool.alloc(cfg, n, k, ids[k], stream=s.cuda_stream)
            pool.free(cfg, n, ids[k], stream=s.cuda_stream)
    for _ in range(3):
        ids.fill_(-9)
        g.replay()
        torch.cuda.synchronize()
        got = ids.cpu().numpy()
        assert np.array_equal(pool.read_bitmap(), before)
        for k in range(m):
            assert np.array_equal(np.sort(got[k][:len(free)]), free) and (got[k][len(free):] == -1).all()
            assert k >= 24 or np.array_equal(got[k][:len(free)], free)
        one = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        pool.alloc(cfg, n, 9, one)
        assert np.array_equal(one.cpu().numpy()[:len(free)], free)
        pool.free(cfg, n, one)
    pool.close()


@pytest.mark.parametrize("strategy", [0, 3, 5])
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 40, 100003])
@pytest.mark.parametrize("free", [0, 1, 5])
def test_budget_pass_refuses_past_the_free_pages(cuda, pbm_mod, strategy, shift, n, free):
    """Refusals in outputs that start off a 16-byte boundary, in a pool with no free page or a few, with and
    without steps: nothing outside the outputs is written."""
    torch, pbm = cuda, pbm_mod
    T = 5000
    pool = pbm.Pool(T, 64)
    words = np.full_like(pool.read_bitmap(), 0xffffffff)
    pages = np.array([3, 64, 65, 2047, 4999][:free], dtype=np.int64)
    for p in pages:
        words[p >> 5] &= ~np.uint32(1 << (p & 31))
    pool.write_bitmap(words)
    k = min(n, free)
    for with_steps in (True, False):
        pool.write_bitmap(words)
        s0 = pool.stats()
        buf = torch.full((2, n + 16), -9, dtype=torch.int32, device="cuda")
        ids, steps = buf[0, 4 + shift:4 + shift + n], buf[1, 4 + shift:4 + shift + n]
        pool.alloc(pbm.walk_config(strategy, fail_fast=1, max_steps=1 << 20), n, 3, ids, steps if with_steps else None)
        h = buf.cpu().numpy()
        i, s = h[0, 4 + shift:4 + shift + n], h[1, 4 + shift:4 + shift + n]
        assert np.array_equal(np.sort(i[:k]), pages[:k]) if 2 * n >= free else set(i[:k]) <= set(pages)
        assert (i[k:] == -1).all()
        assert (s == (np.arange(n) < k)).all() if with_steps and 2 * n >= free else with_steps or (s == -9).all()
        assert (h[:, :4 + shift] == -9).all() and (h[:, 4 + shift + n:] == -9).all()
        st = pool.stats()
        assert (st.successes - s0.successes, st.failures - s0.failures) == (k, n - k)
    pool.close()


@pytest.mark.parametrize("strategy", [0, 1, 2, 3, 5, 6])
@pytest.mark.parametrize("T,occ", [(64, 0.5), (2000, 0.7), (65536 + 17, 0.9), (1 << 20, 0.6), (3000001, 0.95)])
def test_budget_pass_hands_the_free_pages_out_in_order(cuda, pbm_mod, orc, strategy, T, occ):
    """A launch that asks for at least half of the F free pages: request r gets the r-th free page, the
    requests past F are refused, and the counters say so; one that asks for fewer walks as without a budget."""
    torch, pbm = cuda, pbm_mod
    words = orc.bernoulli_bitmap(T, occ, 6)
    bits = np.unpackbits(words.view(np.uint8), bitorder="little")[:T]
    free = np.nonzero(bits == 0)[0]
    F = len(free)
    pool = pbm.Pool(T, 64)
    cfg = pbm.walk_config(strategy, fail_fast=1)
    for n in sorted({(F + 1) // 2, F - 1, F, F + 1, F + 70, 3 * F}):
        if n < 1:
            continue
        pool.reset()
        pool.prefill(occ, 6)
        ids = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        steps = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        pool.alloc(cfg, n, 3, ids, steps)
        k = min(n, F)
        got, st = ids.cpu().numpy(), steps.cpu().numpy()
        assert np.array_equal(got[:k], free[:k]) and (got[k:] == -1).all()
        assert (st[:k] == 1).all() and (st[k:] == 0).all()
        after = bits.copy()
        after[free[:k]] = 1
        assert np.array_equal(np.unpackbits(pool.read_bitmap().view(np.uint8), bitorder="little")[:T], after)
        s = pool.stats()
        assert (s.successes, s.failures, s.steps) == (k, n - k, k)
    pool.close()


def test_budget_pass_beside_another_stream(cuda, pbm_mod, orc):
    """While the pass hands pages out, another stream takes and frees pages of the same pool: no page goes
    to two holders, and the bitmap holds exactly the prefill and what both hold."""
    torch, pbm = cuda, pbm_mod
    T = 1 << 22
    pool = pbm.Pool(T, 64)
    pool.prefill(0.9, 2)
    base = pool.used()
    n, m = 150000, 40000
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    a = torch.empty(T // 8, dtype=torch.int32, device="cuda")
    b = torch.empty(m, dtype=torch.int32, device="cuda")
    cfg, ff = pbm.walk_config(pbm.RANDOM_WALK_BM), pbm.walk_config(pbm.COLLAB_RW_BM, fail_fast=1, max_steps=256)
    torch.cuda.synchronize()
    for k in range(20):
        for j in range(3):
            pool.alloc(cfg, m, 100 * k + j, b, stream=s2.cuda_stream)
            if j < 2:
                pool.free(cfg, m, b, stream=s2.cuda_stream)
        pool.alloc(ff, a.numel(), k, a, stream=s1.cuda_stream)
        torch.cuda.synchronize()
        both = torch.cat([a, b])
        chk = pool.check(both, both.numel())
        assert (chk.n_duplicates, chk.n_not_marked, chk.n_out_of_range) == (0, 0, 0)
        assert chk.used_pages == base + chk.n_ok
        pool.free(cfg, both.numel(), both)
        assert pool.used() == base
    pool.close()


@pytest.mark.parametrize("max_steps", [1, 31, 32, 33, 100, 4096])
@pytest.mark.parametrize("T,occ", [(33, 0.5), (96, 0.9), (1000, 0.99), (65536 + 17, 0.995)])
def test_distributed_clock_counts_positions(cuda, pbm_mod, orc, T, occ, max_steps):
    """Word-wise reading changes neither the pages nor the steps nor the arms, across the pool's end and
    where the bound ends a sweep inside a word."""
    torch, pbm = cuda, pbm_mod
    slots, n = 3, 3
    pool = pbm.Pool(T, 64, max_slots=slots)
    pool.prefill(occ, 2)
    words = orc.bernoulli_bitmap(T, occ, 2)
    arms = np.array([orc.lib().orc_dist_clock_arm0(0, i, T) for i in range(slots)], dtype=np.int64)
    cfg = pbm.walk_config(pbm.DIST_CLOCK, max_steps=max_steps)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    steps = torch.empty(n, dtype=torch.int32, device="cuda")
    for S in range(8):
        pool.alloc(cfg, n, S, ids, steps, serial=True)
        e_ids, e_steps = orc.replay_alloc(words, T, pbm.DIST_CLOCK, n, S, max_steps=max_steps, arms=arms)
        assert np.array_equal(ids.cpu().numpy(), e_ids) and np.array_equal(steps.cpu().numpy(), e_steps)
        assert np.array_equal(pool.read_bitmap(), words)
    pool.close()


@pytest.mark.parametrize("n", [1, 31, 33, 4000])
@pytest.mark.parametrize("max_run", [1, 8, 32, 60])
def test_spans_of_sharing_warps(cuda, pbm_mod, orc, n, max_run):
    """Runs walked for by whole warps (longer ones by their own lane): one request alone equals the
    sequential walk; many are disjoint, were free, and come back."""
    torch, pbm = cuda, pbm_mod
    T = 1 << 18
    rng = np.random.default_rng(n + max_run)
    k = rng.integers(1, max_run + 1, n).astype(np.int32)
    if n > 1:
        k[rng.random(n) < 0.05] = 0                     # not a run: fails at once
    dk = torch.from_numpy(k).cuda()
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    steps = torch.empty(n, dtype=torch.int32, device="cuda")
    pool = pbm.Pool(T, 64)
    for occ in (0.0, 0.02, 0.08):
        pool.reset()
        pool.prefill(occ, 3)
        words = orc.bernoulli_bitmap(T, occ, 3)
        bits = np.unpackbits(words.view(np.uint8), bitorder="little")[:T].astype(np.int32)
        pool.alloc_spans(n, dk, 9, ids, steps)
        got, st = ids.cpu().numpy(), steps.cpu().numpy()
        if n == 1:
            e_ids, e_steps = orc.replay_spans(words, T, k, 9)
            assert np.array_equal(got, e_ids) and np.array_equal(st, e_steps)
            assert np.array_equal(pool.read_bitmap(), words)
        assert (got[k == 0] == -1).all() and (st[k == 0] == 0).all()
        cover = bits.copy()
        for i, c in zip(got[got >= 0], k[got >= 0]):
            cover[i:i + c] += 1
        assert cover.max() == 1 and (got[got >= 0] + k[got >= 0] <= T).all()
        if max_run <= 32:
            assert (got[k > 0] >= 0).all()
        pool.free_runs(n, ids, dk)
        assert np.array_equal(np.unpackbits(pool.read_bitmap().view(np.uint8), bitorder="little")[:T], bits)
    pool.close()


@pytest.mark.parametrize("strategy", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("block_size", [288, 512, 1024])
def test_refused_block_sizes_take_no_page(cuda, pbm_mod, strategy, block_size):
    """Blocks larger than the walks are built for: the call is refused and the pool, the outputs and the
    counters are as before it, with a budget and without one; the next call is served."""
    torch, pbm = cuda, pbm_mod
    n = 40000
    pool = pbm.Pool(1 << 16, 64)
    pool.prefill(0.6, 4)   # pages are listed in a pool at least half full
    before = pool.read_bitmap()
    for fail_fast in (1, 0):
        ids = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        steps = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        with pytest.raises(pbm.PbmError) as e:
            pool.alloc(pbm.walk_config(strategy, fail_fast=fail_fast, block_size=block_size), n, 3, ids, steps)
        assert e.value.rc == pbm.ERR_CUDA
        torch.cuda.synchronize()
        assert np.array_equal(pool.read_bitmap(), before)
        assert (ids == -9).all() and (steps == -9).all()
        s = pool.stats()
        assert (s.successes, s.failures, s.steps) == (0, 0, 0)
    ids = torch.full((100,), -9, dtype=torch.int32, device="cuda")
    pool.alloc(pbm.walk_config(strategy, fail_fast=1), 100, 3, ids)
    assert (ids >= 0).all()
    pool.close()


@pytest.mark.parametrize("keep", [True, False])
@pytest.mark.parametrize("capture_mode", ["global", "thread_local", "relaxed"])
def test_captured_budget_launches_of_many_graphs(cuda, pbm_mod, keep, capture_mode):
    """Graph after graph of one pool, kept or thrown away, more than any fixed number of workspaces: every
    captured launch hands the free pages out in order, with a walk that could not find them."""
    torch, pbm = cuda, pbm_mod
    T, n, per, graphs = 1 << 14, 9000, 7, 40
    pool = pbm.Pool(T, 64)
    pool.prefill(0.6, 5)
    before = pool.read_bitmap()
    free = np.nonzero(np.unpackbits(before.view(np.uint8), bitorder="little")[:T] == 0)[0]
    want = np.concatenate([free, np.full(n - len(free), -1)])
    cfg = pbm.walk_config(pbm.RANDOM_WALK, fail_fast=1, max_steps=1)
    kept = []
    s = torch.cuda.Stream()
    for k in range(graphs):
        ids = torch.full((per, n), -9, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s, capture_error_mode=capture_mode):
            for j in range(per):
                pool.alloc(cfg, n, j, ids[j], stream=s.cuda_stream)
                pool.free(cfg, n, ids[j], stream=s.cuda_stream)
        if keep:
            kept.append((g, ids))
        for _ in range(2):
            ids.fill_(-9)
            g.replay()
            torch.cuda.synchronize()
            assert (ids.cpu().numpy() == want).all()
        if not keep:
            g.reset()
    for g, ids in kept:
        ids.fill_(-9)
    torch.cuda.synchronize()
    for g, ids in kept:
        g.replay()
    torch.cuda.synchronize()
    for g, ids in kept:
        assert (ids.cpu().numpy() == want).all()
    assert np.array_equal(pool.read_bitmap(), before)
    pool.close()


def test_captured_budget_launches_outlive_their_pool(cuda, pbm_mod):
    """A graph that is thrown away after its pool returns its workspace to nobody."""
    torch, pbm = cuda, pbm_mod
    s = torch.cuda.Stream()
    for _ in range(3):
        pool = pbm.Pool(1 << 12, 64)
        ids = torch.empty(100, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            pool.alloc(pbm.walk_config(pbm.RANDOM_WALK, fail_fast=1), 100, 1, ids, stream=s.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert (ids >= 0).all()
        pool.close()
        g.reset()
        torch.cuda.synchronize()


@pytest.mark.parametrize("parts,max_steps", [(1, 512), (1, 4096), (3, 4096)])
@pytest.mark.parametrize("block_size", [32, 256])
@pytest.mark.parametrize("T,occ", [(3000, 0.0), (65536, 0.5), (1 << 20, 0.5), (1 << 20, 0.9), ((1 << 24) - 5, 0.5),
                                   (1 << 24, 0.9), (1 << 22, 0.98)])
def test_clock_sweep_serves_every_free_page(cuda, pbm_mod, orc, T, occ, block_size, parts, max_steps):
    """Launches that ask for exactly the free pages, in one call or in several, get all of them; the next request
    finds none; and again, once a third of them has come back."""
    torch, pbm = cuda, pbm_mod
    pool = pbm.Pool(T, 64)
    pool.prefill(occ, 3)
    free = T - pool.used()
    if parts > 1 and occ > 0.95:
        max_steps = 1 << 16        # pages that the first launches passed lie far apart
    cfg = pbm.walk_config(pbm.SINGLE_CLOCK, max_steps=max_steps, block_size=block_size)
    ids = torch.empty(free, dtype=torch.int32, device="cuda")
    steps = torch.empty(free, dtype=torch.int32, device="cuda")
    cut = np.linspace(0, free, parts + 1).astype(np.int64)
    for lo, hi in zip(cut[:-1], cut[1:]):
        pool.alloc(cfg, int(hi - lo), 7, ids[lo:], steps[lo:])
    assert int((ids < 0).sum()) == 0 and pool.used() == T
    chk = pool.check(ids, free)
    assert (chk.n_duplicates, chk.n_not_marked, chk.n_out_of_range) == (0, 0, 0)
    assert int(steps.min()) >= 1 and int(steps.max()) <= max_steps
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    pool.alloc(cfg, 1, 7, one)
    assert one.item() == -1
    k = free // 3
    pool.free(cfg, k, ids)
    pool.alloc(pbm.walk_config(pbm.SINGLE_CLOCK, max_steps=1 << 20, block_size=block_size), k, 9, ids)
    assert int((ids < 0).sum()) == 0 and pool.used() == T
    assert pool.check(ids, free).n_duplicates == 0
    pool.close()


def test_clock_sweeps_side_by_side_serve_their_requests(cuda, pbm_mod):
    """Launches in several streams that ask for three quarters of the free pages between them."""
    torch, pbm = cuda, pbm_mod
    T, streams = 1 << 20, [torch.cuda.Stream() for _ in range(3)]
    pool = pbm.Pool(T, 64)
    cfg = pbm.walk_config(pbm.SINGLE_CLOCK)
    for k in range(10):
        pool.reset()
        pool.prefill(0.7, k)
        free = T - pool.used()
        n = 3 * free // 4
        ids = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        cut = np.linspace(0, n, 4).astype(np.int64)
        torch.cuda.synchronize()
        for s, lo, hi in zip(streams, cut[:-1], cut[1:]):
            pool.alloc(cfg, int(hi - lo), k, ids[lo:], stream=s.cuda_stream)
        torch.cuda.synchronize()
        assert int((ids < 0).sum()) == 0 and pool.used() == T - free + n
        assert pool.check(ids, n).n_duplicates == 0
    pool.close()


@pytest.mark.parametrize("n", [100, 40000, 200000])
def test_free_list_gets_and_puts_in_two_streams(cuda, pbm_mod, n):
    """Gets of one stream beside puts of another, on a list so short that pages come straight back: in the end the
    bitmap marks exactly the pages that are held."""
    torch, pbm = cuda, pbm_mod
    T = 3 * n
    pool = pbm.Pool(T, 64)
    cfg = pbm.walk_config(pbm.LINKED_LIST)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    held = torch.full((2, n), -1, dtype=torch.int32, device="cuda")
    pool.alloc(cfg, n, 0, held[0])
    pool.alloc(cfg, n, 0, held[1])
    torch.cuda.synchronize()
    for k in range(60):
        new = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        pool.free(cfg, n, held[k % 2], stream=a.cuda_stream)
        pool.alloc(cfg, n, k, new, stream=b.cuda_stream)
        torch.cuda.synchronize()
        assert (new >= 0).all()
        held[k % 2] = new
        ids = np.sort(held.cpu().numpy().ravel())
        assert np.unique(ids).size == 2 * n
        bits = np.unpackbits(pool.read_bitmap().view(np.uint8), bitorder="little")[:T]
        assert np.array_equal(np.nonzero(bits)[0], ids)
    pool.close()


@pytest.mark.parametrize("T", [17_100_000, 17_200_001, 40_000_003])
def test_budget_pass_with_several_words_a_thread(cuda, pbm_mod, T):
    """Pools around and past a word for every thread of the pass: request r gets the r-th free page."""
    torch, pbm = cuda, pbm_mod
    pool = pbm.Pool(T, 64)
    pool.prefill(0.93, 6)
    words = pool.read_bitmap()
    free = np.nonzero(np.unpackbits(words.view(np.uint8), bitorder="little")[:T] == 0)[0]
    cfg = pbm.walk_config(pbm.COLLAB_RW_BM, fail_fast=1)
    for n in ((len(free) + 1) // 2, len(free) - 1, len(free) + 9):
        pool.write_bitmap(words)
        ids = torch.full((n,), -9, dtype=torch.int32, device="cuda")
        pool.alloc(cfg, n, 3, ids)
        k = min(n, len(free))
        assert np.array_equal(ids.cpu().numpy(), np.concatenate([free[:k], np.full(n - k, -1)]))
        assert pool.used() == T - len(free) + k
    pool.close()
