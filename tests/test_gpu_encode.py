"""Encoding and single margins of matrices on both sides of the vector encoder's rule (SNP counts
that are multiples of 16 with at least 16384 threads' work), with class sizes off the word size and
genotype values beyond 2: the 27-cell tables of listed triplets, counted from the planes, and of a
search's winner must equal counts made with numpy."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


def _table(g, p, t):
    cell = 9 * np.minimum(g[:, t[0]], 2) + 3 * np.minimum(g[:, t[1]], 2) + np.minimum(g[:, t[2]], 2)
    return np.concatenate([np.bincount(cell[p != 1], minlength=27), np.bincount(cell[p == 1], minlength=27)])


@pytest.mark.parametrize("S,M,cases", [(8191, 1024, 0.5), (16389, 512, 0.3), (8150, 1040, 0.7), (65000, 144, 0.02),
                                       (2048, 128, 0.5), (8191, 1025, 0.5)])
def test_tables_from_planes(S, M, cases):
    rng = np.random.default_rng(S + M)
    g = rng.choice(np.array([0, 1, 2, 3, 255], np.uint8), size=(S, M), p=[0.4, 0.3, 0.2, 0.05, 0.05])
    p = (rng.random(S) < cases).astype(np.uint8)
    trip = np.sort(np.array([rng.choice(M, 3, replace=False) for _ in range(150)]), axis=1)
    trip[0], trip[1] = (0, 1, 2), (M - 3, M - 2, M - 1)
    with epik2.Context(0) as ctx:
        did = ctx.load(g, p)
        got = ctx.tables(did, trip)
        best = ctx.scan(did, snp_begin=0, snp_end=2)
        one = ctx.scan(did, snp_begin=0, snp_end=2, engine=epik2.ENGINE_INT)
    for t, tab in zip(trip, got):
        assert np.array_equal(tab, _table(g, p, t)), t
    assert best.ijk == one.ijk and best.score == one.score


@pytest.mark.parametrize("M", [3, 32, 33, 64, 65, 66, 97, 176, 177, 178, 16500])
def test_pair_margin_tiles(M):
    """The tile list of the pair margins (64 SNPs j x 112 SNPs k; from 16385 SNPs more blocks than a
    block of its kernel has threads): the last 24 SNPs' tables, which complete from their margins, and
    for a small dataset all of them.  Counts, so exact."""
    rng = np.random.default_rng(M)
    S = 70
    g = rng.integers(0, 3, (S, M)).astype(np.uint8)
    p = (rng.random(S) < 0.5).astype(np.uint8)
    b = max(0, M - 24)
    want = O.scan(np.ascontiguousarray(g[:, b:]), p)
    with epik2.Context(0) as c:
        did = c.load(g, p)
        got = c.scan(did, snp_begin=b, snp_end=M)
        assert tuple(x - b for x in got.ijk) == tuple(want["ijk"]) and f32_bits(got.score) == f32_bits(want["score"])
        if M < 1000:
            assert c.scan(did).score == np.float32(O.scan(g, p)["score"])
        c.set_pheno(did, 1 - p)
        want = O.scan(np.ascontiguousarray(g[:, b:]), 1 - p)
        got = c.scan(did, snp_begin=b, snp_end=M)
        assert f32_bits(got.score) == f32_bits(want["score"])
