"""Device memory of a context: the search workspace that it keeps gives way to whatever else the context has
to allocate.  The device's memory is played by epik2_test_memory_limit, so nothing is filled up."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu

GIB = 1 << 30


@pytest.fixture(scope="module")
def big():
    rng = np.random.default_rng(3)
    return rng.integers(0, 3, (8192, 1024), dtype=np.uint8), (rng.random(8192) < 0.5).astype(np.uint8)


@pytest.fixture(scope="module")
def small():
    return O.gen_hwe(41, 600, 300, 280)


@pytest.mark.parametrize("call", ["dump", "tables", "load", "replicates"])
def test_workspace_gives_way(big, small, call):
    """About 1 GiB of workspace is left by a search of 1024 x 8192; the next call needs most of it."""
    g, p = small
    with epik2.Context(0) as c:
        did = c.load(*big)
        sid = c.load(g, p)
        want = c.scan(did)
        held = c.info(did)["device_bytes"] + c.info(sid)["device_bytes"]
        c.test_memory_limit(held + int(1.15 * GIB))
        if call == "dump":  # 300 SNPs: 0.98 GB of tables
            r = O.scan(g, p, with_tables=True)
            t, s = c.dump_tables(sid)
            assert np.array_equal(t, r["tables"]) and np.array_equal(s.view(np.uint32), r["scores"].view(np.uint32))
        elif call == "tables":
            trip = np.tile(np.array([[0, 1, 2], [5, 100, 299]], np.uint32), (2200000, 1))  # 1.0 GB
            t = c.tables(sid, trip)
            cell = 9 * g[:, 5].astype(int) + 3 * g[:, 100] + g[:, 299]
            assert np.array_equal(t[1::2][-1], np.concatenate([np.bincount(cell[p == v], minlength=27) for v in (0, 1)]))
            assert np.array_equal(t[1], t[-1])
        elif call == "load":
            m = np.zeros((1000, 7000), np.uint8)  # pair margins 0.8 GB
            c.unload(c.load(m, (np.arange(1000) % 2).astype(np.uint8)))
        else:
            reps = np.stack([np.random.default_rng(t).permutation(p) for t in range(2)])
            for q, b in zip(reps, c.scan_replicates(sid, reps)):
                r = O.scan(g, q)
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
        got = c.scan(did)  # its workspace no longer fits beside the rest or is allocated anew
        assert got.ijk == want.ijk and got.score == want.score
        c.test_memory_limit(0)
        got = c.scan(did)
        assert got.ijk == want.ijk and got.score == want.score


def _kernel_ms(c, f):
    f()
    got = f()
    return got, c.stats()["last_scan_kernel_ms"]


def test_replicates_in_groups_that_leave_room_for_their_search():
    """Memory for 12 of 16 replicates and 1 GiB: the search's own rows, margins and planes need most of that
    GiB, so a group of 12 could only take the form that shares all-sample counts, at three times the time."""
    g, p = O.gen_hwe(5, 2000, 1536, 900)
    reps = np.stack([np.random.default_rng(t).permutation(p) for t in range(16)])
    with epik2.Context(0) as c:
        did = c.load(g, p)
        want, free_ms = _kernel_ms(c, lambda: c.scan_replicates(did, reps))
        per = int(epik2.library().epik2_replicate_bytes(2000, 1536))
    with epik2.Context(0) as c:
        did = c.load(g, p)
        c.test_memory_limit(c.info(did)["device_bytes"] + 12 * per + GIB + (1 << 20))
        got, ms = _kernel_ms(c, lambda: c.scan_replicates(did, reps))
    assert [(b.ijk, b.score) for b in got] == [(b.ijk, b.score) for b in want]
    assert ms <= 1.5 * free_ms, (ms, free_ms)


def test_batch_in_parts_whose_searches_fit():
    """12 datasets of 100 x 2000, 0.4 GB of packed margins together: with room for the planes of a search and
    half of the margins the batch is searched in two parts, not on the other kernels."""
    data = [O.gen_hwe(60 + t, 100, 2000, 50) for t in range(12)]
    with epik2.Context(0) as c:
        ids = [c.load(g, p) for g, p in data]
        want, free_ms = _kernel_ms(c, lambda: c.scan_batch(ids))
        held = sum(c.info(d)["device_bytes"] for d in ids)
    with epik2.Context(0) as c:
        ids = [c.load(g, p) for g, p in data]
        c.test_memory_limit(held + int(1.05 * GIB) + (250 << 20))
        got, ms = _kernel_ms(c, lambda: c.scan_batch(ids))
        pinned, pinned_ms = _kernel_ms(c, lambda: c.scan_batch(ids, engine=epik2.ENGINE_TC_FP4, stage_words=8, pair_tile=32, overlap=1))
    assert [(b.ijk, b.score) for b in got] == [(b.ijk, b.score) for b in want]
    assert [(b.ijk, b.score) for b in pinned] == [(b.ijk, b.score) for b in want]
    assert ms <= 1.25 * free_ms, (ms, free_ms, pinned_ms)


@pytest.mark.parametrize("rescore", [0, 1])
def test_no_room_for_the_workspace(rescore):
    """Without room for its workspace every form takes the other kernels, with equal results."""
    g, p = O.gen_hwe(71, 3000, 400, 1300, planted=[(2, 150, 390)], effects=[0.8])
    reps = np.stack([np.random.default_rng(t).permutation(p) for t in range(4)])

    def calls(limit):
        out = []
        with epik2.Context(0) as c:
            a, b = c.load(g, p), c.load(np.ascontiguousarray(g[:, :200]), p)
            held = c.info(a)["device_bytes"] + c.info(b)["device_bytes"]
            if limit:  # planes of the split search: 68 MB for a, 19 MB for b, four times that for the replicates
                c.test_memory_limit(held + (10 << 20))
            c.scan(a)
            c.reset_stats()
            out += [c.scan(a), c.scan(a, snp_begin=10, snp_end=300)]
            launches = c.stats()["kernel_launches"]
            out += c.scan_topk(a, 32) + c.scan_batch([a, b]) + c.scan_replicates(b, reps)
            fp64 = [x.score_fp64 for x in c.scan_topk(a, 32, rescore_fp64=1) + c.scan_batch([a, b], rescore_fp64=1) +
                    c.scan_replicates(b, reps, rescore_fp64=1)] if rescore else []
            if limit:  # the tables, and nothing beside them
                c.test_memory_limit(held + 200 * 199 * 198 // 6 * 220 + (1 << 20))
            t, s = c.dump_tables(b)
        return [(x.ijk, x.score) for x in out], fp64, t, s, launches
    want, got = calls(False), calls(True)
    assert got[0] == want[0] and got[1] == want[1]
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[3].view(np.uint32), want[3].view(np.uint32))
    assert got[4] != want[4]  # other kernels: another number of launches
