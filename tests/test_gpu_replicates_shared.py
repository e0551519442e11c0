"""The replicate form that shares the all-sample counts of a tile (its cases are counted for every
replicate, its controls are the totals less them).  It serves classes of more than 65535 samples, and
matrices whose split search finds no room for its workspace; each replicate must equal the oracle's search
of its phenotype bit for bit.  Also the captured launch of batches, which pinned options take."""
import numpy as np
import pytest

import epik2
import oracle as O
from conftest import f32_bits

pytestmark = pytest.mark.gpu


def _check(g, reps, got, only=None):
    for t, (q, b) in enumerate(zip(reps, got)):
        if only is None or t in only:
            r = O.scan(g, q)
            assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"]), t


def test_classes_beyond_65535():
    """A class of 70000; replicates with a planted triplet in the first tile, without cases, without controls,
    and with class sizes on both sides of the line (a group with one such replicate takes this form)."""
    S, M = 140003, 19
    g, p = O.gen_hwe(151, S, M, 70001, planted=[(0, 1, 2)], effects=[0.7])
    rng = np.random.default_rng(5)
    few = np.zeros(S, np.uint8)
    few[rng.permutation(S)[:65000]] = 1
    reps = np.stack([p, np.zeros_like(p), np.ones_like(p), rng.permutation(p), few])
    with epik2.Context(0) as c:
        did = c.load(g, p)
        for rescore in (0, 1):
            got = c.scan_replicates(did, reps, rescore_fp64=rescore)
            _check(g, reps, got)
            if rescore:
                for q, b in zip(reps[:2], got):
                    i, j, k = b.ijk
                    cell = 9 * g[:, i].astype(int) + 3 * g[:, j] + g[:, k]
                    t = np.concatenate([np.bincount(cell[q != 1], minlength=27), np.bincount(cell[q == 1], minlength=27)])
                    assert b.score_fp64 == O.k2_fp64(t.astype(np.uint32))


@pytest.mark.parametrize("S,M,R", [(1000, 150, 7), (777, 97, 33), (2049, 70, 300)])
def test_without_room_for_the_split_search(S, M, R):
    g, p = O.gen_hwe(S, S, M, S // 3, planted=[(0, 1, M - 1)], effects=[0.8])
    rng = np.random.default_rng(M)
    reps = np.stack([rng.permutation(p) for _ in range(R)])
    reps[0], reps[1], reps[2] = p, 0, 1
    with epik2.Context(0) as c:
        did = c.load(g, p)
        c.reset_stats()
        want = c.scan_replicates(did, reps)
        launches = c.stats()["kernel_launches"]
        held = c.info(did)["device_bytes"]
    with epik2.Context(0) as c:
        # the allocation that a one-call search of 100 x 2000 leaves holds all the replicates; beside it there
        # is room for a tile list, not for the planes of a split search
        did = c.load(g, p)
        c.scan_u8(np.zeros((100, 2000), np.uint8), np.zeros(100, np.uint8), engine=epik2.ENGINE_INT, snp_begin=0, snp_end=1)
        spare = int(epik2.library().epik2_dataset_bytes(100, 2000))
        c.test_memory_limit(held + spare + (200 << 10))
        c.reset_stats()
        got = c.scan_replicates(did, reps)
        assert c.stats()["kernel_launches"] != launches  # another form
    assert [(b.ijk, b.score) for b in got] == [(b.ijk, b.score) for b in want]
    _check(g, reps, got, only=(0, 1, 2, R // 2, R - 1))


@pytest.mark.parametrize("kw", [dict(engine=epik2.ENGINE_TC, stage_words=8), dict(engine=epik2.ENGINE_TC_FP4, stage_words=16, pair_tile=64, overlap=1),
                                dict(engine=epik2.ENGINE_TC_FP4, stage_words=8, pair_tile=64, overlap=2)],
                         ids=["int8", "pairs", "overlapped"])
def test_captured_batch_follows_phenotypes_and_takes_512(kw):
    g, p = O.gen_hwe(161, 500, 40, 240)
    rng = np.random.default_rng(9)
    with epik2.Context(0) as c:
        ids = [c.load(g, p), c.load(np.ascontiguousarray(g[:, ::-1]), p)]
        for _ in range(3):  # the first builds the plan, the others replay it
            q = [rng.permutation(p) for _ in ids]
            for d, x in zip(ids, q):
                c.set_pheno(d, x)
            for h, x, b in zip((g, g[:, ::-1]), q, c.scan_batch(ids, **kw)):
                r = O.scan(np.ascontiguousarray(h), x)
                assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
        tiny = [c.load(np.ascontiguousarray(g[t:t + 40, :3 + t % 9]), p[t:t + 40]) for t in range(256)]
        many = tiny + tiny
        for t, b in enumerate(c.scan_batch(many, **kw)):
            r = O.scan(np.ascontiguousarray(g[t % 256:t % 256 + 40, :3 + t % 256 % 9]), p[t % 256:t % 256 + 40])
            assert b.ijk == r["ijk"] and f32_bits(b.score) == f32_bits(r["score"])
