"""The genotype-split search (the library's choice for classes of at most 65535 samples) where it
can go wrong: edges of its tiles (56 SNPs j x 128 SNPs k), of its sample groups (quads of 128,
groups without samples, each genotype the most frequent one), class splits from empty to full,
equal scores, and the limit of its 16-bit cells.  Tables and FP32 scores must equal the oracle's bit for
bit, and the screened search must return the oracle's triplet and score."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def auto():
    c = epik2.Context(0)
    yield c
    c.close()


def _check(ctx, g, p, tables=True):
    r = O.scan(g, p, with_tables=tables)
    did = ctx.load(g, p)
    try:
        b = ctx.scan(did)
        assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
        if tables:
            t, s = ctx.dump_tables(did)
            assert np.array_equal(t, r["tables"])
            assert np.array_equal(s.view(np.uint32), r["scores"].view(np.uint32))
    finally:
        ctx.unload(did)


def _genotypes(rng, S, M, share):
    """Genotypes with the shares (g0, g1, g2)."""
    return rng.choice(3, size=(S, M), p=share).astype(np.uint8)


@pytest.mark.parametrize("M", [3, 4, 5, 57, 58, 59, 129, 130, 131, 186, 187])
def test_tile_edges(auto, M):
    g, p = O.gen_hwe(900 + M, 700, M, 301)
    _check(auto, g, p)


@pytest.mark.parametrize("S", [1, 2, 63, 127, 128, 129, 255, 257, 383, 385, 511, 1024])
def test_sample_group_edges(auto, S):
    rng = np.random.default_rng(S)
    for share in ((0.5, 0.3, 0.2), (0.2, 0.6, 0.2), (0.1, 0.2, 0.7)):  # each genotype dropped
        g = _genotypes(rng, S, 20, share)
        p = (rng.random(S) < 0.4).astype(np.uint8)
        _check(auto, g, p)


def test_groups_of_whole_quads_and_empty_groups(auto):
    S = 1024
    p = np.tile(np.array([0, 1], np.uint8), S // 2)
    g = np.zeros((S, 12), np.uint8)      # constant SNPs: both counted groups empty
    g[:256, 1] = 1                       # groups of exactly 128 samples per class
    g[256:512, 1] = 2
    g[:, 2] = 2
    g[:, 3] = 1
    g[:258, 4] = 1                       # 129 per class
    g[:, 5:] = np.random.default_rng(5).integers(0, 3, (S, 7))
    _check(auto, g, p)


@pytest.mark.parametrize("cases", [0, 1, 7, 150, 1499, 1500])
def test_class_splits(auto, cases):
    rng = np.random.default_rng(cases)
    g = _genotypes(rng, 1500, 70, (0.6, 0.3, 0.1))
    p = np.zeros(1500, np.uint8)
    p[rng.permutation(1500)[:cases]] = 1
    _check(auto, g, p)


def _even(S, cases):
    """The class split whose screening bound has p = 1/2."""
    return 1.115 * S * abs((S - cases + 13.5) / (S + 27.0) - 0.5) ** 3 <= 1.0


@pytest.mark.parametrize("S", [150, 1000, 9000])
@pytest.mark.parametrize("top_k", [1, 32])
def test_even_and_uneven_classes(auto, S, top_k):
    """The last even split and the first uneven one on either side, and an even and an uneven dataset in
    one batch: triplets and scores as the oracle's (exact, the scores are FP32 sums in its order)."""
    rng = np.random.default_rng(S)
    g = _genotypes(rng, S, 40, (0.5, 0.35, 0.15))
    few = next(c for c in range(S) if _even(S, c))
    many = next(c for c in range(S, 0, -1) if _even(S, c))
    splits = [few, few - 1, many, many + 1]
    dids = []
    try:
        for cases in splits:
            p = np.zeros(S, np.uint8)
            p[rng.permutation(S)[:cases]] = 1
            r = O.scan(g, p, with_tables=True)
            did = auto.load(g, p)
            dids.append((did, r))
            if top_k == 1:
                b = auto.scan(did)
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
            else:
                best = np.sort(r["scores"].astype(np.float64))[:top_k]
                got = [x.score for x in auto.scan_topk(did, top_k)]
                assert np.array_equal(np.sort(np.float32(got)), best.astype(np.float32))
        if top_k == 1:
            for (_, r), b in zip(dids, auto.scan_batch([d for d, _ in dids])):
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
    finally:
        for did, _ in dids:
            auto.unload(did)


def test_rare_alleles_and_strong_effects(auto):
    """Scores far from the bulk, sparse tables: where the screening bound is loosest."""
    rng = np.random.default_rng(17)
    for S, cases, share in ((400, 0.5, (0.96, 0.035, 0.005)), (3000, 0.1, (0.9, 0.09, 0.01)), (900, 0.8, (0.3, 0.4, 0.3))):
        g = _genotypes(rng, S, 90, share)
        carrier = (g[:, 4] > 0) | (g[:, 50] > 0) | (g[:, 88] == 2)
        p = np.where(carrier, rng.random(S) < 0.97, rng.random(S) < cases / 4).astype(np.uint8)
        _check(auto, g, p)


def test_equal_scores_break_to_the_lowest_triplet(auto):
    rng = np.random.default_rng(23)
    g = _genotypes(rng, 600, 80, (0.4, 0.4, 0.2))
    g[:, 60] = g[:, 3]
    g[:, 71] = g[:, 3]
    g[:, 77] = g[:, 30]
    p = ((g[:, 3] + g[:, 30] + rng.integers(0, 3, 600)) > 3).astype(np.uint8)
    _check(auto, g, p)
    _check(auto, np.zeros((300, 130), np.uint8), (np.arange(300) % 2).astype(np.uint8))  # every score equal


@pytest.mark.parametrize("n0,n1", [(65535, 40), (40, 65535), (65536, 40), (65535, 65535)])
def test_limit_of_the_16_bit_cells(auto, n0, n1):
    g, p = O.gen_hwe(77, n0 + n1, 20, n1)
    _check(auto, g, p)


def test_ranges_and_topk_agree_with_the_integer_engine(auto):
    g, p = O.gen_hwe(31, 1501, 200, 640, planted=[(4, 100, 190)], effects=[0.8])
    did = auto.load(g, p)
    try:
        want = auto.scan_topk(did, 32, engine=epik2.ENGINE_INT, rescore_fp64=1)
        got = auto.scan_topk(did, 32, rescore_fp64=1)
        assert [(b.ijk, f32_bits(b.score), b.score_fp64) for b in got] == \
               [(b.ijk, f32_bits(b.score), b.score_fp64) for b in want]
        assert [b.ijk for b in auto.scan_topk(did, 32)] == [b.ijk for b in auto.scan_topk(did, 32, engine=epik2.ENGINE_INT)]
        for a, b in ((0, 1), (5, 61), (61, 200), (197, 198)):
            x, y = auto.scan(did, snp_begin=a, snp_end=b), auto.scan(did, snp_begin=a, snp_end=b, engine=epik2.ENGINE_INT)
            assert x.ijk == y.ijk and f32_bits(x.score) == f32_bits(y.score)
        with pytest.raises(epik2.Epik2Error) as e:
            auto.scan(did, snp_begin=198, snp_end=200)
        assert e.value.status == epik2.E_INVALID
    finally:
        auto.unload(did)


def test_batch_and_replicates_equal_separate_searches(auto):
    """Datasets of many shapes, and phenotypes of very different class sizes, in one search each."""
    data = [O.gen_hwe(40 + t, S, M, c) for t, (S, M, c) in enumerate(
        [(300, 20, 140), (64, 3, 32), (2047, 70, 1500), (500, 131, 250), (40, 12, 0), (3001, 33, 3000), (129, 187, 64)])]
    ids = [auto.load(g, p) for g, p in data]
    try:
        for rescore in (0, 1):
            got = auto.scan_batch(ids, rescore_fp64=rescore)
            for (g, p), b in zip(data, got):
                r = O.scan(g, p)
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
                if rescore:
                    assert b.score_fp64 == O.k2_fp64(O.scan(g, p, with_tables=True)["tables"][_index(g.shape[1], *b.ijk)])
    finally:
        for d in ids:
            auto.unload(d)
    g, p = O.gen_hwe(90, 900, 66, 400)
    rng = np.random.default_rng(3)
    reps = np.stack([rng.permutation(p), np.zeros_like(p), np.ones_like(p), (rng.random(900) < 0.03).astype(np.uint8)])
    did = auto.load(g, p)
    try:
        for q, b in zip(reps, auto.scan_replicates(did, reps)):
            r = O.scan(g, q)
            assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
    finally:
        auto.unload(did)


def _index(m, i, j, k):
    before_i = sum((m - 1 - a) * (m - 2 - a) // 2 for a in range(i))
    before_j = sum(m - 1 - b for b in range(i + 1, j))
    return before_i + before_j + k - j - 1
