"""The forms that the allocation kernels take for whole warps and blocks, at the
sizes where they can go wrong, against the oracle's sequential replay or the
walk's own probe sequence.  All comparisons are of whole numbers, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

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
