"""Parts of a search by first SNP: the genotype-split search lays out rows and margins from the part's first
SNP on (whole groups of 128), so the parts begin and end on both sides of such groups, in ascending,
descending and repeated order on one context.  Triplet and score must equal the integer engine's, and the
best of adjacent parts the whole search's."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,M,cases", [(4500, 300, 2000), (5003, 517, 1100)])
def test_parts_equal_the_integer_engine(S, M, cases):
    g, p = O.gen_hwe(S, S, M, cases, planted=[(M // 2, M // 2 + 40, M - 2)], effects=[0.7])
    cuts = [0, 1, 30, 31, 95, 126, 127, 128, 129, 254, 255, 256, M - 5, M - 3, M - 2]
    parts = [(a, b) for a, b in zip(cuts, cuts[1:])] + [(5, M), (127, M), (128, 260), (255, M)]
    with epik2.Context(0) as c:
        did = c.load(g, p)
        want = {ab: c.scan(did, snp_begin=ab[0], snp_end=ab[1], engine=epik2.ENGINE_INT) for ab in parts}
        for order in (parts, parts[::-1], parts):
            got = {ab: c.scan(did, snp_begin=ab[0], snp_end=ab[1]) for ab in order}
            for ab in parts:
                assert got[ab].ijk == want[ab].ijk and f32_bits(got[ab].score) == f32_bits(want[ab].score), ab
        top = c.scan_topk(did, 32, snp_begin=127, snp_end=M, rescore_fp64=1)
        ref = c.scan_topk(did, 32, snp_begin=127, snp_end=M, rescore_fp64=1, engine=epik2.ENGINE_INT)
        assert [(b.ijk, b.score_fp64) for b in top] == [(b.ijk, b.score_fp64) for b in ref]
        whole = c.scan(did)
        best = min((got[ab] for ab in zip(cuts, cuts[1:])), key=lambda b: (b.score, b.ijk))
        assert best.ijk == whole.ijk and best.score == whole.score
