"""Workloads of the page and buffer manager, as a program that uses it runs them.

Every case goes through the Python binding of the C ABI (`pbm.py`), on pools,
graphs and buffer managers that the program made beforehand.  Parallel walks
race for pages, so which page a request gets is not determined; what a pass
returns is what every correct run agrees on: which requests were served, the
bytes read back through the pages, the pages the buffer manager holds, and the
pool's whole bitmap once the pass has released what it took.  Where one warp
serves the call, or the pages are handed out in order, the ids themselves come
back too.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("parallel-db-buffer-management_gb300"))

import pbm  # noqa: E402

WALKS = {"page": pbm.RANDOM_WALK, "word": pbm.RANDOM_WALK_BM, "collab": pbm.COLLAB_RW_BM,
         "clustered": pbm.CLUSTERED_RW_BM, "list": pbm.LINKED_LIST, "clock": pbm.SINGLE_CLOCK,
         "dist": pbm.DIST_CLOCK}


# ---- the cases --------------------------------------------------------------

def listed():
    return [
        # A query operator asks for a warp's worth of scratch pages and gives them back: the latency
        # of one small call.
        {"name": "alloc_collab_32", "kind": "alloc", "walk": "collab", "bits": 32, "width": 32, "fail_fast": 0,
         "pages": 1 << 16, "occupancy": 0.5, "n": 32},
        # Hash-table partitions written into small pages: 16,384 workers each claim a 64 B page of a
        # half-full pool, write it, read it back and free it.
        {"name": "page_io_16k_64b", "kind": "page_io", "pages": 1 << 16, "page_size": 64, "payload": 64,
         "occupancy": 0.5, "n": 1 << 14},
        # A parallel operator's million page requests on the 64 GiB pool's bitmap at 90%.
        {"name": "alloc_collab_1m", "kind": "alloc", "walk": "collab", "bits": 32, "width": 32, "fail_fast": 0,
         "pages": 1 << 24, "occupancy": 0.9, "n": 1 << 20},
        # The plain per-thread page probe on a ragged, crowded pool: long walks.
        {"name": "alloc_page_250k", "kind": "alloc", "walk": "page", "bits": 32, "width": 32, "fail_fast": 0,
         "pages": 5000011, "occupancy": 0.9, "n": 250007},
        # The free-list strategy, for callers that want pages back in release order.
        {"name": "alloc_list_1m", "kind": "alloc", "walk": "list", "bits": 32, "width": 32, "fail_fast": 0,
         "pages": 1 << 24, "occupancy": 0.5, "n": 1 << 20},
        # The shared clock arm, an odd number of requests.
        {"name": "alloc_clock_300k", "kind": "alloc", "walk": "clock", "bits": 32, "width": 32, "fail_fast": 0,
         "pages": 1 << 22, "occupancy": 0.75, "n": 300007},
        # A load that asks for more pages than are left (2^22 requests at 90%): fail-fast launches
        # hand out what there is and refuse the rest at once.
        {"name": "alloc_failfast_4m", "kind": "alloc", "walk": "collab", "bits": 32, "width": 32, "fail_fast": 1,
         "pages": 1 << 24, "occupancy": 0.9, "n": 1 << 22},
        # One cycle of a batch executor: 256 callers' uneven groups are allocated, swapped and freed
        # by a replayed graph, the pool going from 81% to 90% and back.
        {"name": "batch_graph_1500k", "kind": "batch", "form": "graph", "walk": "collab", "bits": 32, "width": 64,
         "pages": 1 << 24, "occupancy": 0.81, "groups": 256, "requests": 1500000},
        # Eight rounds of a table scan mix through the buffer manager: Zipf(0.99) page references,
        # pins held for a geometric number of rounds, frames for a sixteenth of the pages.
        {"name": "bufmgr_128k", "kind": "bufmgr", "policy": "single", "logical": 1 << 24, "frames": 1 << 20,
         "round": 1 << 17, "frame_size": 0},
        # The same with 4 KiB frames filled from a backing store, each request reading its record.
        {"name": "bufmgr_copy_16k", "kind": "bufmgr", "policy": "single", "logical": 1 << 20, "frames": 1 << 17,
         "round": 1 << 14, "frame_size": 4096},
        # Variable-size blocks (16 B .. 64 KiB) of 256 callers, allocated and freed by a replayed graph.
        {"name": "malloc_runs_512k", "kind": "malloc", "backend": "runs", "pages": 1 << 22, "groups": 256,
         "requests": 1 << 19},
        # A burst of 64 tenants' alloc / free / fetch requests through the serving loop.
        {"name": "serve_1000", "kind": "serve", "pages": 1 << 22, "tenants": 64, "requests": 1000,
         "max_pages": 4096},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more workload of the same ranges: every strategy, word width, hand policy and backend."""
    kind = rng.choice(["alloc", "alloc", "alloc", "alloc", "failfast", "page_io", "batch", "batch", "bufmgr",
                       "copy", "malloc", "malloc", "spans", "serve"])
    occ = rng.choice([0.02, 0.25, 0.5, 0.75, 0.9, 0.95])
    if kind == "alloc":
        walk = rng.choice(sorted(WALKS))
        pages = log_int(rng, 1 << 14, 1 << 24)
        return {"kind": "alloc", "walk": walk, "bits": rng.choice([32, 64]), "width": rng.choice([8, 16, 32]),
                "fail_fast": 0, "pages": pages, "occupancy": occ,
                "n": log_int(rng, 1, min(1 << 20, pages * (1 - occ) * 0.5))}
    if kind == "failfast":
        pages = log_int(rng, 1 << 16, 1 << 24)
        occ = rng.choice([0.6, 0.75, 0.9, 0.95])
        free = pages * (1 - occ)
        return {"kind": "alloc", "walk": rng.choice(["collab", "word", "page"]), "bits": 32, "width": 32,
                "fail_fast": 1, "pages": pages, "occupancy": occ,
                "n": min(1 << 22, int(free * rng.uniform(0.6, 2.5)) + 64)}
    if kind == "page_io":
        pages = log_int(rng, 1 << 12, 1 << 18)
        size = rng.choice([64, 96, 256, 1024, 4096])
        occ = min(occ, 0.9)
        return {"kind": "page_io", "pages": pages, "page_size": size, "payload": rng.choice([4, 60, 64, size]) if size > 64
                else rng.choice([4, 60, 64]), "occupancy": occ, "n": log_int(rng, 8, pages * (1 - occ) * 0.6)}
    if kind == "batch":
        pages = log_int(rng, 1 << 18, 1 << 24)
        walk = rng.choice(["collab", "collab", "collab", "word", "page"])
        occ = min(occ, 0.9)
        return {"kind": "batch", "form": rng.choice(["graph", "launch", "inline"]), "walk": walk,
                "bits": rng.choice([32, 64]), "width": rng.choice([16, 32, 64]) if walk == "collab" else 32,
                "pages": pages, "occupancy": occ, "groups": log_int(rng, 1, 256),
                "requests": log_int(rng, 1 << 9, min(1500000, pages * (1 - occ) * 0.6))}
    if kind in ("bufmgr", "copy"):
        copy = kind == "copy"
        logical = log_int(rng, 1 << 14, (1 << 20) if copy else (1 << 24))
        frames = logical // rng.choice([4, 8, 16])
        policy = rng.choice(["single", "single", "dist"])
        most = min(1 << 17, frames // 8)
        return {"kind": "bufmgr", "policy": policy, "logical": logical, "frames": frames,
                "round": log_int(rng, max(48, most // 64) if policy == "dist" else 48, most),
                "frame_size": rng.choice([64, 512, 4096]) if copy else 0}
    if kind == "malloc":
        requests = log_int(rng, 1 << 8, 1 << 19)
        return {"kind": "malloc", "backend": rng.choice(["runs", "queue"]), "pages": max(1 << 13, requests * 8),
                "groups": log_int(rng, 1, 256), "requests": requests}
    if kind == "spans":
        n = log_int(rng, 64, 1 << 17)
        return {"kind": "spans", "pages": max(1 << 16, n * 64), "max_run": rng.choice([4, 32, 48]), "n": n}
    return {"kind": "serve", "pages": log_int(rng, 1 << 21, 1 << 23), "tenants": rng.choice([8, 64]),
            "requests": log_int(rng, 40, 1000), "max_pages": log_int(rng, 64, 4096)}


# ---- what a program has in hand before the call -----------------------------

class _DeviceWords:
    """The pool's bitmap as an array of 32-bit words (keeps the pool alive)."""

    def __init__(self, pool):
        self.pool = pool
        self.__cuda_array_interface__ = {"shape": (pool.bitmap_bytes // 4,), "typestr": "<i4",
                                         "data": (pool.bitmap_ptr, False), "version": 3}


def bitmap_of(pool):
    return torch.as_tensor(_DeviceWords(pool), device="cuda")


def log_uniform(gen, n, lo, hi):
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.exp(u * math.log((hi + 1) / lo)).mul_(lo).floor_().clamp_(lo, hi).to(torch.int32)


def zipf(gen, n, items, s=0.99):
    """Zipf(s) references: the inverse of the continuous distribution, through a random permutation."""
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    rank = (u * ((items + 1) ** (1 - s) - 1) + 1).pow_(1 / (1 - s)).floor_().clamp_(1, items).to(torch.int64) - 1
    return torch.randperm(items, generator=gen, device="cuda", dtype=torch.int32)[rank].contiguous()


def group_counts(seed, groups, requests):
    """LogU[1, 65536] group sizes scaled to `requests` in all."""
    rng = np.random.default_rng(seed)
    w = np.exp(rng.uniform(0, math.log(65536), groups))
    c = np.floor(w * (requests / w.sum())).astype(np.int64)
    c[np.argmax(c)] += requests - c.sum()
    return c


def group_table(op, counts):
    t = np.zeros(len(counts), dtype=[("op", "<i4"), ("count", "<u4"), ("offset", "<u8")])
    t["op"], t["count"] = op, counts
    t["offset"] = np.concatenate([[0], np.cumsum(counts)[:-1]])
    return t


def on_device(table):
    return torch.from_numpy(table.view(np.uint8).reshape(-1).copy()).cuda()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": case, "seed": (seed * 2654435761 + 12345) % (1 << 31),
         "stream": torch.cuda.current_stream().cuda_stream}
    globals()["prepare_" + case["kind"]](case, seed, gen, s)
    torch.cuda.synchronize()
    return s


def prepare_alloc(c, seed, gen, s):
    s["pool"] = pbm.Pool(c["pages"])
    s["pool"].prefill(c["occupancy"], seed)
    s["cfg"] = pbm.walk_config(WALKS[c["walk"]], word_bits=c["bits"], collab_width=c["width"],
                               fail_fast=c["fail_fast"])
    s["ids"] = torch.empty(c["n"], dtype=torch.int32, device="cuda")
    s["steps"] = torch.empty(c["n"], dtype=torch.int32, device="cuda")
    s["bitmap"] = bitmap_of(s["pool"])
    # one warp serves the call, or the free pages are handed out in order
    s["ordered"] = c["fail_fast"] == 1 or (c["walk"] == "collab" and c["width"] == 32 and c["n"] <= 32)


def prepare_page_io(c, seed, gen, s):
    s["pool"] = pbm.Pool(c["pages"], c["page_size"], materialize=True)
    s["pool"].prefill(c["occupancy"], seed)
    s["cfg"] = pbm.walk_config(pbm.RANDOM_WALK)
    s["ids"] = torch.empty(c["n"], dtype=torch.int32, device="cuda")
    s["data"] = torch.empty(c["n"], c["payload"] // 4, dtype=torch.int32, device="cuda")
    s["bitmap"] = bitmap_of(s["pool"])


def prepare_batch(c, seed, gen, s):
    n, groups = c["requests"], c["groups"]
    s["pool"] = pbm.Pool(c["pages"])
    s["pool"].prefill(c["occupancy"], seed)
    s["cfg"] = pbm.walk_config(WALKS[c["walk"]], word_bits=c["bits"], collab_width=c["width"], blocks_per_sm=5)
    counts = group_counts(seed, groups, n)
    tables = [group_table(op, counts) for op in (pbm.OP_ALLOC, pbm.OP_SWAP, pbm.OP_FREE)]
    s["arena"] = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    s["results"] = torch.empty(n, dtype=torch.int32, device="cuda")
    s["d_tables"] = [on_device(t) for t in tables]
    s["h_tables"] = [pbm.groups_array([(int(g["op"]), int(g["count"]), int(g["offset"])) for g in t]) for t in tables]
    if c["form"] == "graph":
        s["d_all"] = torch.cat(s["d_tables"])
        s["graph"] = s["pool"].graph(s["cfg"], s["d_all"], groups, 3, s["arena"], n, s["seed"], results=s["results"])
    s["bitmap"] = bitmap_of(s["pool"])


ROUNDS = 8       # rounds of one buffer-manager pass
TRACE = 64       # rounds of references the program replays


def prepare_bufmgr(c, seed, gen, s):
    n, fsz = c["round"], c["frame_size"]
    s["trace"] = zipf(gen, TRACE * n, c["logical"])
    if fsz:
        s["backing"] = torch.randint(-2**31, 2**31 - 1, (c["logical"] * fsz // 4,), generator=gen, device="cuda",
                                     dtype=torch.int32)
        s["record"] = min(fsz, 256)
        s["data"] = torch.empty(ROUNDS * n, s["record"] // 4, dtype=torch.int32, device="cuda")
    dist = c["policy"] == "dist"
    s["bm"] = pbm.BufferManager(c["logical"], c["frames"], frame_size=fsz,
                                policy=pbm.BM_DIST_CLOCK if dist else pbm.BM_SINGLE_CLOCK, n_arms=n if dist else 1,
                                backing=s.get("backing"))
    s["frames"] = torch.empty(ROUNDS * n, dtype=torch.int32, device="cuda")
    s["held"] = torch.empty(ROUNDS * n, dtype=torch.int32, device="cuda")
    # each reference keeps its pin for a geometric (p = 0.25) number of rounds,
    # the last ones until the end of the pass
    u = torch.rand(ROUNDS * n, generator=gen, device="cuda", dtype=torch.float64)
    hold = torch.floor(torch.log1p(-u) / math.log(0.75)).to(torch.int64) + 1
    due = (torch.arange(ROUNDS * n, device="cuda") // n + hold).clamp_(max=ROUNDS)
    s["release"] = torch.sort(due, stable=True).indices.to(torch.int32)
    ends = np.concatenate([[0], np.cumsum(torch.bincount(due, minlength=ROUNDS + 1).cpu().numpy())])
    s["ends"] = [int(e) for e in ends]
    s["at"] = 0
    # a manager in use: every frame holds some page
    fill = torch.randperm(c["logical"], generator=gen, device="cuda", dtype=torch.int32)[:c["frames"]].contiguous()
    got = torch.empty_like(fill)
    held = torch.empty_like(fill)
    index = torch.arange(c["frames"], dtype=torch.int32, device="cuda")
    chunk = n if dist else 1 << 16
    for lo in range(0, c["frames"], chunk):
        k = min(chunk, c["frames"] - lo)
        s["bm"].round_pages(None, None, 0, fill[lo:], k, 0, got[lo:], held[lo:])
        s["bm"].round_pages(held, index[lo:], k, None, 0, 0, None)


def prepare_malloc(c, seed, gen, s):
    n, groups = c["requests"], c["groups"]
    s["pool"] = pbm.Pool(c["pages"], 4096, materialize=True)
    s["sizes"] = log_uniform(gen, n, 16, 65536)
    # slots without a request in this step carry size 0
    s["sizes"][torch.rand(n, generator=gen, device="cuda") < 0.05] = 0
    s["ptrs"] = torch.zeros(n, dtype=torch.int64, device="cuda")
    counts = group_counts(seed, groups, n)
    tables = torch.cat([on_device(group_table(op, counts)) for op in (pbm.OP_MALLOC, pbm.OP_MFREE)])
    s["tables"] = tables
    if c["backend"] == "queue":
        s["pool"].qmalloc_init(1 << 20)
        make = s["pool"].qmalloc_graph
    else:
        s["pool"].malloc_init()
        make = s["pool"].malloc_graph
    s["graph"] = make(tables, groups, 2, s["sizes"], s["ptrs"], n, s["seed"])
    s["bitmap"] = bitmap_of(s["pool"])


def prepare_spans(c, seed, gen, s):
    s["pool"] = pbm.Pool(c["pages"])
    s["pool"].prefill(0.02, seed)
    s["npages"] = log_uniform(gen, c["n"], 1, c["max_run"])
    s["ids"] = torch.empty(c["n"], dtype=torch.int32, device="cuda")
    s["bitmap"] = bitmap_of(s["pool"])


def prepare_serve(c, seed, gen, s):
    rng = np.random.default_rng(seed)
    n, tenants = c["requests"], c["tenants"]
    s["pool"] = pbm.Pool(c["pages"])
    s["pool"].prefill(0.5, seed)
    s["fetch"] = zipf(gen, 1 << 16, 1 << 18)
    s["bm"] = pbm.BufferManager(1 << 18, 1 << 17, policy=pbm.BM_DIST_CLOCK, n_arms=4096)
    s["server"] = pbm.Server(s["pool"], tenants, 1 << 16, n_streams=4, max_batch_requests=256, max_occupancy=0.95,
                             bufmgr=s["bm"], fetch_pages=s["fetch"], max_fetch_pages=1 << 15)
    u = rng.uniform(size=n)
    s["ops"] = np.where(u < 0.45, pbm.REQ_ALLOC, np.where(u < 0.9, pbm.REQ_FREE, pbm.REQ_FETCH)).tolist()
    s["tenants"] = rng.integers(0, tenants, n).tolist()
    s["counts"] = np.floor(np.exp(rng.uniform(0, math.log(c["max_pages"] + 1), n))).astype(np.int64).tolist()
    # the burst ends with every tenant giving its pages back
    s["ops"] += [pbm.REQ_FREE] * tenants
    s["tenants"] += list(range(tenants))
    s["counts"] += [1 << 30] * tenants
    s["arrivals"] = [0.0] * len(s["ops"])
    s["bitmap"] = bitmap_of(s["pool"])


# ---- one pass ---------------------------------------------------------------

def run(state):
    state["seed"] = (state["seed"] + 1) % (1 << 31)
    return globals()["run_" + state["case"]["kind"]](state["case"], state)


def run_alloc(c, s):
    n, pool, ids, steps = c["n"], s["pool"], s["ids"], s["steps"]
    pool.alloc(s["cfg"], n, s["seed"], ids, steps, stream=s["stream"])
    pool.free(s["cfg"], n, ids, stream=s["stream"])
    if s["ordered"]:
        return {"ids": ids, "steps": steps, "bitmap": s["bitmap"]}
    return {"served": ids >= 0, "bitmap": s["bitmap"]}


def run_page_io(c, s):
    n, pool, ids = c["n"], s["pool"], s["ids"]
    pool.claim_write_free(n, s["seed"], ids, payload_bytes=c["payload"], hold=True, stream=s["stream"])
    pool.gather_pages(ids, n, c["payload"], s["data"], stream=s["stream"])
    pool.free(s["cfg"], n, ids, stream=s["stream"])
    return {"data": s["data"], "bitmap": s["bitmap"]}


def run_batch(c, s):
    n, groups = c["requests"], c["groups"]
    for k in range(3):                       # allocate, swap, free
        if c["form"] == "graph":
            s["graph"].replay(s["stream"])
        else:
            inline = c["form"] == "inline"
            s["pool"].batch(s["cfg"], None if inline else s["d_tables"][k], s["h_tables"][k] if inline else None,
                            groups, s["arena"], n, s["seed"] + 7 * k, pbm.LAUNCH_PERSISTENT, stream=s["stream"],
                            results=s["results"])
    return {"released": s["results"] >= 0, "bitmap": s["bitmap"]}


def run_bufmgr(c, s):
    n, bm, ends, stream = c["round"], s["bm"], s["ends"], s["stream"]
    trace, frames, held, release = (s[k].data_ptr() for k in ("trace", "frames", "held", "release"))
    for r in range(ROUNDS):
        lo = 4 * r * n
        k = ends[r + 1] - ends[r]
        bm.round_pages(held, release + 4 * ends[r], k, trace + 4 * s["at"] * n, n, s["at"] * n, frames + lo, held + lo,
                       stream=stream)
        if c["frame_size"]:
            bm.gather(frames + lo, n, s["record"], s["data"].data_ptr() + r * n * s["record"], stream=stream)
        s["at"] = (s["at"] + 1) % TRACE
    bm.round_pages(held, release + 4 * ends[ROUNDS], ends[ROUNDS + 1] - ends[ROUNDS], None, 0, 0, None, stream=stream)
    return {"held": s["held"], "data": s["data"]} if c["frame_size"] else {"held": s["held"]}


def run_malloc(c, s):
    s["graph"].replay(s["stream"])
    served = s["ptrs"] != 0
    s["graph"].replay(s["stream"])
    out = {"served": served, "ptrs": s["ptrs"]}
    if c["backend"] == "runs":               # queued blocks stay with their class
        out["bitmap"] = s["bitmap"]
    return out


def run_spans(c, s):
    n, pool, ids = c["n"], s["pool"], s["ids"]
    pool.alloc_spans(n, s["npages"], s["seed"], ids, stream=s["stream"])
    pool.free_runs(n, ids, s["npages"], stream=s["stream"])
    return {"served": ids >= 0, "bitmap": s["bitmap"]}


def run_serve(c, s):
    res, _, _ = s["server"].run(s["arrivals"], s["tenants"], s["ops"], s["counts"])
    got = np.frombuffer(res, dtype=[("t", "<f8", 4), ("pages", "<u8"), ("status", "<i4"), ("pad", "<u4")])
    return {"pages": got["pages"].astype(np.int64), "status": got["status"].copy(), "bitmap": s["bitmap"]}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """Bytes: every id, page, pointer and record read once and written once, and one read and one write of the
    bitmap word (or page-table entry) that a claim, a release, a pin or an unpin changes."""
    c, k = case, case["kind"]
    if k == "alloc":
        granted = min(c["n"], int(c["pages"] * (1 - c["occupancy"])))
        scan = c["pages"] // 8 if c["fail_fast"] else 0
        return {"bytes": 12 * c["n"] + 16 * granted + scan, "flops": 0}
    if k == "page_io":
        return {"bytes": c["n"] * (12 + 16 + 3 * c["payload"]), "flops": 0}
    if k == "batch":
        # allocate: slot and result written; swap: slot read and written; free: slot read; 4 bitmap words changed
        return {"bytes": c["requests"] * (8 + 12 + 8 + 4 * 8) + 3 * 16 * c["groups"], "flops": 0}
    if k == "bufmgr":
        n = ROUNDS * c["round"]
        # page, release index, held page; two outputs; one 8-byte entry read and written by the pin and by the unpin
        copy = n * (0.3 * 2 * c["frame_size"] + 2 * min(c["frame_size"], 256)) if c["frame_size"] else 0
        return {"bytes": n * (12 + 8 + 32) + copy, "flops": 0}
    if k == "malloc":
        # size, pointer written, read and cleared; the run's first page, length and count; two bitmap words changed
        return {"bytes": c["requests"] * (4 + 24 + 18 + 16), "flops": 0}
    if k == "spans":
        return {"bytes": c["n"] * (8 + 8 + 16), "flops": 0}
    mean = c["max_pages"] / math.log(c["max_pages"] + 1)
    return {"bytes": c["requests"] * 0.9 * mean * 12, "flops": 0}


def exact(case, seed):
    """Every output is a whole number, compared value for value: there is nothing to round."""
    return None
