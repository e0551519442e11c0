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
