"""Small searches, which take the integer engine, single FP4 CTAs or the genotype-split search by their size
(triplets x samples 3e6, 4e7 and 2.5e8, samples 64, 1000 and 4096), on both sides of each line and as whole
searches, parts and batches: best triplet, tables and FP32 scores must equal the oracle's bit for bit."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu

SHAPES = [(64, 67), (64, 68), (65, 67), (65, 68), (64, 287), (64, 288), (1000, 27), (1000, 28), (1001, 26), (1001, 63),
          (1000, 63), (1000, 116), (4096, 73), (4097, 73), (4096, 72), (700, 3), (5, 30), (1, 3)]


@pytest.mark.parametrize("engine", [epik2.ENGINE_AUTO, epik2.ENGINE_TC_FP4])
def test_whole_searches_and_parts(engine):
    with epik2.Context(0, engine=engine) as c:
        for S, M in SHAPES:
            g, p = O.gen_hwe(S + M, S, M, S // 3)
            r = O.scan(g, p, with_tables=True)
            did = c.load(g, p)
            b = c.scan(did)
            assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"]), (S, M)
            if M < 150:
                t, s = c.dump_tables(did)
                assert np.array_equal(t, r["tables"]) and np.array_equal(s.view(np.uint32), r["scores"].view(np.uint32))
            tri = np.array(O.triplet_list(M))
            for a, e in ((0, 1), (M // 3, M // 3 + 2), (M - 3, M)):
                rows = np.flatnonzero((tri[:, 0] >= a) & (tri[:, 0] < e))
                if len(rows) == 0:
                    continue
                w = rows[np.argmin(r["scores"][rows])]
                b = c.scan(did, snp_begin=a, snp_end=e)
                assert b.ijk == tuple(int(x) for x in tri[w]) and f32_bits(b.score) == f32_bits(r["scores"][w]), (S, M, a, e)
            with pytest.raises(epik2.Epik2Error) as err:
                c.scan(did, snp_begin=M - 2, snp_end=M)
            assert err.value.status == epik2.E_INVALID
            c.unload(did)


@pytest.mark.parametrize("n,S,M", [(1, 64, 5), (3, 4096, 70), (3, 4097, 30), (40, 300, 31), (17, 1500, 80)])
def test_batches(n, S, M):
    rng = np.random.default_rng(n)
    with epik2.Context(0) as c:
        data = [O.gen_hwe(10 * n + t, max(1, S - 7 * t), max(3, M - t % 5), S // 4) for t in range(n)]
        ids = [c.load(g, p) for g, p in data]
        for rescore in (0, 1):
            for (g, p), b in zip(data, c.scan_batch(ids, rescore_fp64=rescore)):
                r = O.scan(g, p)
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
        # a new phenotype follows into the next calls (shapes seen once, a new plan, its replay), and
        # other shapes between them
        for _ in range(4):
            q = rng.permutation(data[0][1])
            c.set_pheno(ids[0], q)
            r = O.scan(data[0][0], q)
            for got in (c.scan_batch(ids)[0], c.scan_batch(ids[::-1])[-1], c.scan_batch(ids + ids[:1])[-1]):
                assert got.ijk == r["ijk"] and f32_bits(got.score) == f32_bits(r["score"])
