"""Tiles of a single pipeline stage: a class without samples and at most 128 or 256 in the other.  The
overlapped kernel's producing warps can then run several tiles ahead of its scoring warps, which must still
find their descriptors (the autotuner times that kernel, so AUTO meets it where the genotype-split search
gives way: here nearly constant SNPs).  Many tiles per CTA pair; every form against the integer engine,
and the smaller one against the oracle."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


def _data(S, M, cases, maf, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(*maf, M)
    u = rng.random((S, M))
    g = (u >= (1 - p) ** 2).astype(np.uint8) + (u >= 1 - p * p).astype(np.uint8)
    return g, np.full(S, 1 if cases else 0, np.uint8)


@pytest.mark.parametrize("S", [1, 31, 80, 128, 129, 256, 257])
@pytest.mark.parametrize("cases", [False, True])
def test_overlapped_kernel(S, cases):
    g, p = _data(S, 300, cases, (0.05, 0.5), S)
    with epik2.Context(0) as c:
        did = c.load(g, p)
        want = c.scan(did, engine=epik2.ENGINE_INT)
        small = c.load(np.ascontiguousarray(g[:, :90]), p)
        r = O.scan(np.ascontiguousarray(g[:, :90]), p, with_tables=True)
        for words in (4, 8):
            kw = dict(engine=epik2.ENGINE_TC_FP4, stage_words=words, pair_tile=64, overlap=2)
            for _ in range(3):
                b = c.scan(did, **kw)
                assert b.ijk == want.ijk and f32_bits(b.score) == f32_bits(want.score)
            for b, w in zip(c.scan_batch([did, small, did], **kw), (want, None, want)):
                ijk, score = (w.ijk, w.score) if w else (r["ijk"], r["score"])
                assert b.ijk == ijk and f32_bits(b.score) == f32_bits(score)
            with epik2.Context(0, **kw) as k:
                d = k.load(np.ascontiguousarray(g[:, :90]), p)
                t, s = k.dump_tables(d)
                assert np.array_equal(t, r["tables"]) and np.array_equal(s.view(np.uint32), r["scores"].view(np.uint32))


@pytest.mark.parametrize("S,M", [(80, 407), (40, 500), (200, 407)])
@pytest.mark.parametrize("cases", [False, True])
def test_default_on_nearly_constant_snps(S, M, cases):
    g, p = _data(S, M, cases, (0.0005, 0.01), S + M)
    with epik2.Context(0) as c:
        did = c.load(g, p)
        want = c.scan(did, engine=epik2.ENGINE_INT)
        for b in (c.scan(did), c.scan(did), c.scan_batch([did, did])[1], c.scan_replicates(did, p[None, :])[0]):
            assert b.ijk == want.ijk and f32_bits(b.score) == f32_bits(want.score)
        c.autotune(did)
