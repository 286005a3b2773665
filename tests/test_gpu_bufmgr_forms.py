"""Buffer-manager rounds at the sizes where the launch changes form: blocks of 64 and 256
threads, frames copied in one or several pieces, releases merged over a block.  Whole
numbers and bytes, compared exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frame_size", [16, 48, 1040, 4096, 4112, 12304])
@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("by_page", [True, False])
def test_every_copied_frame_holds_its_page(cuda, pbm_mod, frame_size, policy, by_page):
    torch, pbm = cuda, pbm_mod
    n_logical, n_frames, R, rounds = 6000, 1500, 333, 12
    gen = torch.Generator(device="cuda")
    gen.manual_seed(frame_size)
    words = frame_size // 4
    backing = torch.randint(-2**31, 2**31 - 1, (n_logical, words), generator=gen, device="cuda", dtype=torch.int32)
    bm = pbm.BufferManager(n_logical, n_frames, frame_size=frame_size, policy=policy, n_arms=R if policy else 1,
                           backing=backing)
    rng = np.random.default_rng(1)
    prev = idx = None
    for r in range(rounds):
        # some pages asked for by many requests of the round, and some ids that name no page
        pages = np.where(rng.random(R) < 0.3, rng.integers(0, 5, R), rng.integers(0, n_logical, R)).astype(np.int32)
        pages[rng.random(R) < 0.02] = -1
        d = torch.from_numpy(pages).cuda()
        frames = torch.empty(R, dtype=torch.int32, device="cuda")
        held = torch.empty(R, dtype=torch.int32, device="cuda")
        k = 0 if prev is None else R
        if by_page:
            bm.round_pages(prev, idx, k, d, R, r * R, frames, held)
            assert np.array_equal(held.cpu().numpy(), np.where(pages >= 0, pages, -1))
        else:
            bm.round(prev, idx, k, d, R, r * R, frames)
        out = torch.empty(R, words, dtype=torch.int32, device="cuda")
        bm.gather(frames, R, frame_size, out)
        ok = d >= 0
        assert torch.equal(frames >= 0, ok)
        assert torch.equal(out[ok], backing[d[ok].long()])
        prev, idx = (held if by_page else frames), torch.randperm(R, device="cuda").to(torch.int32)
    if by_page:
        bm.round_pages(prev, idx, R, None, 0, 0, None)
    else:
        bm.round(prev, idx, R, None, 0, 0, None)
    c, chk = bm.counters(), bm.check()
    assert (c.bad_unpins, c.timeouts, c.failures, chk.mismatches, chk.loading, chk.pins) == (0, 0, 0, 0, 0, 0)
    assert c.hits + c.misses == c.unpins and c.evictions > 0
    bm.close()


@pytest.mark.parametrize("extra", [0, 1, 5000])
@pytest.mark.parametrize("frame_size", [16, 2048, 4112])
@pytest.mark.parametrize("policy", [0, 1])
def test_large_copying_rounds_hold_their_pages(cuda, pbm_mod, frame_size, policy, extra):
    """Rounds on both sides of three blocks of 64 fetches an SM, where the staging buffers halve."""
    torch, pbm = cuda, pbm_mod
    R = 3 * 64 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n_logical, n_frames, words = 60000, 40000, frame_size // 4
    gen = torch.Generator(device="cuda")
    gen.manual_seed(frame_size + extra)
    backing = torch.randint(-2**31, 2**31 - 1, (n_logical, words), generator=gen, device="cuda", dtype=torch.int32)
    bm = pbm.BufferManager(n_logical, n_frames, frame_size=frame_size, policy=policy, n_arms=R if policy else 1,
                           backing=backing)
    prev = idx = None
    for r in range(3):
        d = torch.randint(0, n_logical, (R,), generator=gen, device="cuda", dtype=torch.int32)
        frames = torch.empty(R, dtype=torch.int32, device="cuda")
        bm.round(prev, idx, R if r else 0, d, R, r * R, frames)
        out = torch.empty(R, words, dtype=torch.int32, device="cuda")
        bm.gather(frames, R, frame_size, out)
        assert (frames >= 0).all() and torch.equal(out, backing[d.long()])
        prev, idx = frames, torch.randperm(R, generator=gen, device="cuda").to(torch.int32)
    c, chk = bm.counters(), bm.check()
    assert (c.bad_unpins, c.timeouts, c.failures, chk.mismatches, chk.loading, chk.pins) == (0, 0, 0, 0, 0, R)
    assert c.hits + c.misses == 3 * R and c.evictions > 0
    bm.close()


@pytest.mark.parametrize("n", [1, 33, 511, 513, 5000, 80001])
@pytest.mark.parametrize("by_page", [True, False])
def test_release_rounds_move_exactly_the_listed_pins(cuda, pbm_mod, n, by_page):
    """Each page is fetched several times and released in parts: after every part the pins of every page
    are what the host counts; releases of pins that are not held are refused and counted."""
    torch, pbm = cuda, pbm_mod
    n_logical, n_frames = 4096, 4096
    rng = np.random.default_rng(n)
    pages = np.minimum(rng.zipf(1.3, n) - 1, n_logical - 1).astype(np.int32)
    bm = pbm.BufferManager(n_logical, n_frames)
    d = torch.from_numpy(pages).cuda()
    frames = torch.empty(n, dtype=torch.int32, device="cuda")
    held = torch.empty(n, dtype=torch.int32, device="cuda")
    bm.round_pages(None, None, 0, d, n, 0, frames, held)
    order = torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda()
    pins = np.bincount(pages, minlength=n_logical)
    for lo, hi in ((0, n // 3), (n // 3, n)):
        if hi == lo:
            continue
        if by_page:
            bm.round_pages(held, order[lo:], hi - lo, None, 0, 0, None)
        else:
            bm.round(frames, order[lo:], hi - lo, None, 0, 0, None)
        pins = pins - np.bincount(pages[order[lo:hi].cpu().numpy()], minlength=n_logical)
        assert np.array_equal(bm.read_tables()[1], pins)
    c = bm.counters()
    assert (c.unpins, c.bad_unpins) == (n, 0) and not pins.any()
    extra = torch.tensor([0], dtype=torch.int32, device="cuda")
    if by_page:
        bm.round_pages(held, extra, 1, None, 0, 0, None)
    else:
        bm.round(frames, extra, 1, None, 0, 0, None)
    c = bm.counters()
    assert (c.unpins, c.bad_unpins) == (n, 1) and not bm.read_tables()[1].any()
    bm.close()


@pytest.mark.parametrize("page_size,nbytes", [(4, 4), (16, 16), (64, 60), (96, 96), (100, 96), (4096, 4096), (4096, 16)])
@pytest.mark.parametrize("shift", [0, 1])
def test_gather_copies_rows(cuda, pbm_mod, page_size, nbytes, shift):
    """Whole and partial rows, 16-byte pieces and 4-byte ones (odd page sizes, an output off a 16-byte
    boundary), ids that name no page."""
    torch, pbm = cuda, pbm_mod
    T, n = 1000, 777
    pool = pbm.Pool(T, page_size, materialize=True)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    full = page_size // 4 * 4
    pool.claim_write_free(n, 3, ids, payload_bytes=full, hold=True)
    ask = ids.clone()
    ask[5], ask[6] = -1, T
    buf = torch.full((n * nbytes // 4 + 8,), -7, dtype=torch.int32, device="cuda")
    out = buf[shift:shift + n * nbytes // 4]
    pool.gather_pages(ask, n, nbytes, out)
    want = torch.arange(n, dtype=torch.int32, device="cuda").repeat_interleave(nbytes // 4).view(n, -1)
    want[5], want[6] = 0, 0
    assert torch.equal(out.view(n, -1), want)
    assert (buf[:shift] == -7).all() and (buf[shift + n * nbytes // 4:] == -7).all()
    pool.close()


@pytest.mark.parametrize("frame_size,R", [(16, 333), (4112, 333), (4096, 30000)])
@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("by_page", [True, False])
def test_backing_store_in_host_memory(cuda, pbm_mod, frame_size, R, policy, by_page):
    """Pages filled from pinned host memory, which the device reads over the link."""
    torch, pbm = cuda, pbm_mod
    n_logical, n_frames, words = 4 * R, 2 * R, frame_size // 4
    gen = torch.Generator(device="cuda")
    gen.manual_seed(frame_size)
    want = torch.randint(-2**31, 2**31 - 1, (n_logical, words), generator=gen, device="cuda", dtype=torch.int32)
    backing = want.cpu().pin_memory()
    bm = pbm.BufferManager(n_logical, n_frames, frame_size=frame_size, policy=policy, n_arms=R if policy else 1,
                           backing=backing)
    prev = idx = None
    for r in range(4):
        d = torch.randint(0, n_logical, (R,), generator=gen, device="cuda", dtype=torch.int32)
        frames, held = (torch.empty(R, dtype=torch.int32, device="cuda") for _ in range(2))
        if by_page:
            bm.round_pages(prev, idx, R if r else 0, d, R, r * R, frames, held)
        else:
            bm.round(prev, idx, R if r else 0, d, R, r * R, frames)
        out = torch.empty(R, words, dtype=torch.int32, device="cuda")
        bm.gather(frames, R, frame_size, out)
        assert (frames >= 0).all() and torch.equal(out, want[d.long()])
        prev, idx = (held if by_page else frames), torch.randperm(R, generator=gen, device="cuda").to(torch.int32)
    c, chk = bm.counters(), bm.check()
    assert (c.bad_unpins, c.timeouts, c.failures, chk.mismatches, chk.loading, chk.pins) == (0, 0, 0, 0, 0, R)
    assert c.hits + c.misses == 4 * R and c.evictions > 0
    bm.close()


@pytest.mark.parametrize("per_sm", [128, 256])
@pytest.mark.parametrize("extra", [-1, 0, 4000])
@pytest.mark.parametrize("policy", [0, 1])
def test_rounds_where_the_blocks_grow(cuda, pbm_mod, per_sm, extra, policy):
    """Rounds on both sides of the sizes from which blocks are larger, with hot pages and ids that name none: every
    request holds the frame of its page, and the pins are what the host counts."""
    torch, pbm = cuda, pbm_mod
    R = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n_logical, n_frames = 300000, 150000
    rng = np.random.default_rng(R)
    bm = pbm.BufferManager(n_logical, n_frames, policy=policy, n_arms=R if policy else 1)
    prev = idx = None
    for r in range(3):
        pages = np.where(rng.random(R) < 0.3, rng.integers(0, 5, R), rng.integers(0, n_logical, R)).astype(np.int32)
        pages[rng.random(R) < 0.02] = -1
        d = torch.from_numpy(pages).cuda()
        frames, held = (torch.empty(R, dtype=torch.int32, device="cuda") for _ in range(2))
        bm.round_pages(prev, idx, R if r else 0, d, R, r * R, frames, held)
        assert np.array_equal(held.cpu().numpy(), np.where(pages >= 0, pages, -1))
        frame_of, pins, of_frame = bm.read_tables()[0], bm.read_tables()[1], frames.cpu().numpy()
        ok = pages >= 0
        assert np.array_equal(frame_of[pages[ok]], of_frame[ok])
        assert np.array_equal(pins, np.bincount(pages[ok], minlength=n_logical))
        prev, idx = held, torch.randperm(R, device="cuda").to(torch.int32)
    c, chk = bm.counters(), bm.check()
    assert (c.bad_unpins, c.timeouts, c.failures, chk.mismatches, chk.loading) == (0, 0, 0, 0, 0)
    bm.close()
