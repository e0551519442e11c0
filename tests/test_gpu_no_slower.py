"""Searches that the library's own choice of kernel must not make slower than the kernels it chooses from:
data and shapes where the genotype-split search has least to gain.  Each is timed (fastest of 9 calls)
against the fastest pinned configuration; both sides' results must be equal.  The bound of 1.3 is far above
the run-to-run spread (a few per cent) and below what a wrong choice costs (1.4 to 100 times); a comparison
that a busy host disturbed is made again, twice at most."""
import time

import numpy as np
import pytest

import epik2

pytestmark = pytest.mark.gpu

PINNED = ({"engine": epik2.ENGINE_INT}, {"engine": epik2.ENGINE_TC, "stage_words": 4},
          {"engine": epik2.ENGINE_TC_FP4, "stage_words": 8, "pair_tile": 32, "overlap": 1},
          {"engine": epik2.ENGINE_TC_FP4, "stage_words": 16, "pair_tile": 64, "overlap": 1})


@pytest.fixture(scope="module")
def auto():
    c = epik2.Context(0)
    yield c
    c.close()


def _hwe(S, M, maf, cases, seed=1):
    rng = np.random.default_rng(seed)
    p = rng.uniform(*maf, M)
    u = rng.random((S, M), dtype=np.float32)
    g = (u >= (1 - p) ** 2).astype(np.uint8) + (u >= 1 - p * p).astype(np.uint8)
    ph = np.zeros(S, np.uint8)
    ph[rng.permutation(S)[:cases]] = 1
    return g, ph


def _time(f, n=9):
    f()
    f()
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        r = f()
        t.append(time.perf_counter() - t0)
    return min(t), r


def _compare(call, pinned=PINNED, slack=1.3):
    for attempt in range(3):
        ours, got = _time(call)
        best = None
        for kw in pinned:
            t, want = _time(lambda: call(**kw))
            got_l, want_l = (got, want) if isinstance(got, list) else ([got], [want])
            assert [(b.ijk, b.score) for b in got_l] == [(b.ijk, b.score) for b in want_l]
            best = t if best is None else min(best, t)
        if ours <= slack * best:
            return
    assert ours <= slack * best, (ours * 1e3, best * 1e3)


def _with(auto, g, p, slack=1.3, **kw):
    did = auto.load(g, p)
    try:
        _compare(lambda **pin: auto.scan(did, **kw, **pin), slack=slack)
    finally:
        auto.unload(did)


@pytest.mark.parametrize("S,M,maf,cases", [(2000, 512, (0.005, 0.02), 100), (4000, 1024, (0.02, 0.05), 200),
                                           (4000, 512, (0.05, 0.5), 40), (1000, 1024, (0.001, 0.005), 500),
                                           (8192, 512, (0.05, 0.5), 5)])
def test_rare_alleles_and_uneven_classes(auto, S, M, maf, cases):
    _with(auto, *_hwe(S, M, maf, cases))


@pytest.mark.parametrize("S,M", [(50, 4), (100, 8), (50, 100), (50, 200), (500, 32), (500, 64), (1000, 64), (2048, 40)])
def test_small_searches(auto, S, M):
    _with(auto, *_hwe(S, M, (0.05, 0.5), S // 2))


@pytest.mark.parametrize("n,S,M", [(3, 100, 8), (512, 100, 8), (256, 500, 32), (200, 500, 64)])
def test_batches_of_small_datasets(auto, n, S, M):
    ids = [auto.load(*_hwe(S, M, (0.05, 0.5), S // 2, seed=t)) for t in range(n)]
    try:
        _compare(lambda **kw: auto.scan_batch(ids, **kw), PINNED[1:])
    finally:
        for d in ids:
            auto.unload(d)


@pytest.mark.parametrize("S,M", [(2000, 4096), (500, 12000)])
def test_parts_of_a_large_search(auto, S, M):
    """Also the last first SNPs, whose triplets are few beside the matrix."""
    rng = np.random.default_rng(M)
    g = rng.integers(0, 3, (S, M), dtype=np.uint8)
    did = auto.load(g, (rng.random(S) < 0.5).astype(np.uint8))
    try:
        for a, e in ((M - 10, M), (M - 100, M), (M // 2, M // 2 + 1), (M // 2, M // 2 + 8), (0, 1)):
            _compare(lambda **kw: auto.scan(did, snp_begin=a, snp_end=e, **kw), PINNED[1:] if e < M else PINNED, slack=1.6)
    finally:
        auto.unload(did)


@pytest.mark.parametrize("S,M,constant", [(200, 700, 1.0), (1000, 1024, 1.0), (2000, 1024, 1.0), (4000, 1024, 0.95),
                                          (8192, 512, 1.0), (9500, 512, 1.0), (1000, 1024, 0.4)])
def test_constant_snps(auto, S, M, constant):
    g, p = _hwe(S, M, (0.05, 0.5), S // 2)
    g[:, np.random.default_rng(2).permutation(M)[:int(constant * M)]] = 0
    _with(auto, g, p)


def test_nearly_constant_snps(auto):
    _with(auto, *_hwe(500, 700, (0.0002, 0.001), 250))


def test_constant_snps_after_another_dataset_and_as_replicates(auto):
    """The count of nearly constant SNPs belongs to its dataset, also after a new phenotype."""
    a = auto.load(*_hwe(1000, 700, (0.05, 0.5), 500))
    g = np.zeros((1000, 700), np.uint8)
    p = (np.arange(1000) % 2).astype(np.uint8)
    b = auto.load(g, p)
    try:
        auto.set_pheno(a, p)
        _compare(lambda **kw: auto.scan(a, **kw))
        _compare(lambda **kw: auto.scan(b, **kw))
        auto.set_pheno(b, 1 - p)
        _compare(lambda **kw: auto.scan(b, **kw))
        one = auto.scan(b, engine=epik2.ENGINE_INT)
        for r in auto.scan_replicates(b, np.stack([1 - p, 1 - p])):
            assert r.ijk == one.ijk and r.score == one.score
        _compare(lambda **kw: auto.scan_batch([a, b], **kw), PINNED[1:], slack=1.6)
    finally:
        auto.unload(a)
        auto.unload(b)
