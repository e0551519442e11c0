"""Performance cases of the exhaustive third-order K2 search: what a user of this library has it
do, through the public entry points of the Python mirror of the C ABI.

listed() holds the named cases, draw() gives further ones of the same ranges, prepare() makes what
a program has in hand before the call (matrix, phenotype, resident datasets on one context), run()
is one pass, work() the bytes and operations no implementation can do without, exact() the scores
in 64 bits by plain torch where that takes seconds.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cross-dpc-episdet_b200"))
import epik2  # noqa: E402
from epik2 import sharding, workloads  # noqa: E402

# kinds of call:
#   one_call    matrix and phenotype in host memory -> best triplet (upload, encode, search)
#   scan        best triplet of a resident dataset
#   shard       the same over one of eight equal-work ranges of the first index (one GPU's share)
#   topk        the 32 best triplets, rescored in double precision
#   batch       best triplet of each of many resident datasets, one call
#   replicates  best triplet of phenotype permutations of one resident matrix, one call
#   permute     a new phenotype for a resident matrix, then its best triplet
#   region      every table and score of a small set of SNPs


def _case(name, kind, snps, samples, cases=0.5, data="hwe", **more):
    c = {"kind": kind, "snps": snps, "samples": samples, "cases": cases, "data": data, **more}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: the reference program's own data (uniform genotypes) at its smallest size
        _case("one call 128 x 2048", "one_call", 128, 2048, data="uniform"),
        # an ordinary study of candidate SNPs, nothing a multiple of anything, a third are cases
        _case("one call 333 x 3001", "one_call", 333, 3001, cases=1 / 3),
        # the small benchmark workload, resident
        _case("plain small 512 x 2048", "scan", 512, 2048),
        # the two matrices of the serving workload
        _case("resident A 1024 x 8192", "scan", 1024, 8192),
        _case("resident B 3072 x 4096", "scan", 3072, 4096),
        # the benchmark's step: an eighth of the large workload
        _case("plain large shard 4096 x 16384", "shard", 4096, 16384, part=2),
        # the precision workload: 32 best, double precision, rare alleles among them
        _case("precision 2048 x 8192", "topk", 2048, 8192, maf_lo=0.01),
        # datasets of many sizes in one call
        _case("batch of 16", "batch", 1536, 12000, count=16),
        # permutation test of a resident matrix, one call
        _case("replicates 8 of 1024 x 8192", "replicates", 1024, 8192, count=8),
        # permutation test driven by the caller: one phenotype after the other
        _case("permute 601 x 5003", "permute", 601, 5003, cases=0.4),
        # a biobank's sample count on a candidate set
        _case("many samples 256 x 100000", "scan", 256, 100000),
        # every table of a region
        _case("region 96 x 3001", "region", 96, 3001),
    ]


def _triplets(m):
    return m * (m - 1) * (m - 2) // 6


def draw(rng):
    """One more case: sizes over their logarithms, odd ones, case fractions from 0.25 to 0.75."""
    kind = rng.choice(["one_call", "one_call", "scan", "scan", "scan", "shard", "topk", "batch", "replicates", "permute",
                       "region"])
    frac = round(rng.uniform(0.25, 0.75), 3)
    data = rng.choice(["hwe", "hwe", "hwe", "uniform"])
    if kind == "region":
        return _case("", kind, rng.randint(40, 120), rng.randint(500, 6000), frac, data)
    if kind == "batch":
        return _case("", kind, 1536, 12000, 0.5, "hwe", count=rng.randint(5, 16), first=rng.randint(0, 79))
    count = rng.randint(3, 9) if kind == "replicates" else 1
    top = 1.2e13 / (0.125 if kind == "shard" else count)
    while True:
        m = round(math.exp(rng.uniform(math.log(128), math.log(4096))))
        s = round(math.exp(rng.uniform(math.log(1000), math.log(40000))))
        if _triplets(m) * s <= top and (kind != "shard" or m >= 1000):
            break
    more = {"count": count} if kind == "replicates" else {"part": rng.randrange(8)} if kind == "shard" else {}
    return _case("", kind, m, s, frac, data, **more)


def _matrix(gen, snps, samples, case_fraction, data, maf_lo=0.05):
    """Genotypes uint8 [samples][snps] and phenotype uint8 [samples] on the GPU: Hardy-Weinberg at
    minor-allele frequencies uniform in [maf_lo, 0.5], or uniform genotypes as the reference program
    makes; carriers of one planted triplet are cases more often."""
    dev = "cuda"
    u = torch.rand(samples, snps, generator=gen, device=dev)
    if data == "uniform":
        g = (u * 3).to(torch.uint8).clamp_(max=2)
    else:
        p = maf_lo + (0.5 - maf_lo) * torch.rand(snps, generator=gen, device=dev)
        q2 = (1 - p) ** 2
        g = (u >= q2).to(torch.uint8)
        g += (u >= q2 + 2 * p * (1 - p)).to(torch.uint8)
    a, b, c = snps // 7, snps // 2, snps - 3
    carrier = (g[:, a] > 0) & (g[:, b] > 0) & (g[:, c] > 0)
    lean = torch.rand(samples, generator=gen, device=dev) + 0.25 * carrier
    ph = torch.zeros(samples, dtype=torch.uint8, device=dev)
    ph[lean.topk(round(case_fraction * samples)).indices] = 1
    return g, ph


_context = None


def _ctx():
    """The one context a program keeps for all its searches."""
    global _context
    if _context is None:
        _context = epik2.Context(0)
    return _context


class _Resident:
    """Datasets that stay on the GPU as long as the state that holds them."""

    def __init__(self, ids):
        self.ids = ids

    def __del__(self):
        for d in self.ids:
            try:
                _ctx().unload(d)
            except Exception:
                pass


def _specs(case):
    return workloads.batched_specs()[case.get("first", 0):][: case["count"]]


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "batch":
        return [_matrix(gen, s["n_snps"], s["n_samples"], s["n_cases"] / s["n_samples"], "hwe") for s in _specs(case)]
    g, ph = _matrix(gen, case["snps"], case["samples"], case["cases"], case["data"], case.get("maf_lo", 0.05))
    if case["kind"] in ("replicates", "permute"):
        n = case.get("count", 1)
        perm = torch.stack([ph[torch.randperm(len(ph), generator=gen, device="cuda")] for _ in range(n)])
        return g, ph, perm
    return g, ph


def prepare(case, seed):
    kind = case["kind"]
    host = [[t.cpu().numpy() for t in x] for x in (_inputs(case, seed) if kind == "batch" else [_inputs(case, seed)])]
    torch.cuda.empty_cache()
    state = {"kind": kind, "opts": {}}
    if kind == "one_call":
        state["geno"], state["pheno"] = host[0]
        return state
    state["held"] = _Resident([_ctx().load(h[0], h[1]) for h in host])
    if kind in ("replicates", "permute"):
        state["phenos"] = host[0][2]
    if kind == "shard":
        a, b = sharding.shard_bounds(case["snps"], 8)[case["part"]]
        state["opts"] = {"snp_begin": a, "snp_end": b}
    return state


def _of(bests):
    return {"score": np.array([b.score for b in bests], dtype=np.float32),
            "ijk": np.array([b.ijk for b in bests], dtype=np.int64)}


def run(state):
    c, kind = _ctx(), state["kind"]
    if kind == "one_call":
        return _of([c.scan_u8(state["geno"], state["pheno"])])
    ids = state["held"].ids
    if kind in ("scan", "shard"):
        return _of([c.scan(ids[0], **state["opts"])])
    if kind == "topk":
        top = c.scan_topk(ids[0], 32, rescore_fp64=1)
        return {**_of(top), "score64": np.array([b.score_fp64 for b in top])}
    if kind == "batch":
        return _of(c.scan_batch(ids))
    if kind == "replicates":
        return _of(c.scan_replicates(ids[0], state["phenos"]))
    if kind == "permute":
        c.set_pheno(ids[0], state["phenos"][0])
        return _of([c.scan(ids[0])])
    tables, scores = c.dump_tables(ids[0])
    return {"tables": tables, "scores": scores}


def work(case):
    """Bytes: the matrix, the phenotype(s) and the results once.  Operations: for every triplet its
    54 counts' worth of score (27 cells, 8 operations each) and, for every sample, the four products
    of the two smaller genotype groups of its first SNP (on average 0.41 of the samples for these
    allele frequencies, 2/3 for uniform genotypes)."""
    kind = case["kind"]
    sets = ([(s["n_snps"], s["n_samples"], 1) for s in _specs(case)] if kind == "batch"
            else [(case["snps"], case["samples"], case.get("count", 1))])
    share = 2 / 3 if case["data"] == "uniform" else 0.41
    b = f = 0.0
    for m, s, n in sets:
        t = _triplets(m) * n * (0.125 if kind == "shard" else 1.0)
        b += m * s + n * s + 32 * n + (220 * t if kind == "region" else 0)
        f += t * (216 + 8 * share * s)
    return {"bytes": b, "flops": f}


def _all_scores(g, ph, keep):
    """The `keep` lowest K2 scores of all triplets in 64 bits (sorted): counts by 0/1 products (exact
    in 32 bits), ln n! by lgamma."""
    s, m = g.shape
    f = torch.lgamma(torch.arange(s + 2, dtype=torch.float64, device=g.device) + 1)
    cls = [g[ph == 0], g[ph == 1]]
    best = torch.empty(0, dtype=torch.float64, device=g.device)
    for i in range(m - 2):
        w = m - 1 - i
        step = max(1, (1 << 22) // w)
        hot = [torch.stack([(c[:, i + 1:] == v) for v in range(3)]).to(torch.float32) for c in cls]  # [3][S_c][w]
        for j0 in range(0, w, step):
            j1 = min(w, j0 + step)
            tot = torch.zeros(j1 - j0, w, dtype=torch.float64, device=g.device)
            for a in range(3):
                part = []
                for c, h in zip(cls, hot):
                    rows = c[:, i] == a
                    ha = h[:, rows]
                    part.append((ha, ha[:, :, j0:j1]))
                for b in range(3):
                    for d in range(3):
                        n = [(left[b].T @ full[d]).round().to(torch.int64) for full, left in part]
                        tot += f[n[0] + n[1] + 1] - f[n[0]] - f[n[1]]
            rows = torch.arange(j0, j1, device=g.device)[:, None]
            tot = tot[torch.arange(w, device=g.device)[None, :] > rows]
            best = torch.cat([best, tot])
            if len(best) > (1 << 24):
                best = best.topk(keep, largest=False).values
    return best.topk(min(keep, len(best)), largest=False).values.cpu().numpy()


def _region(g, ph):
    """Every score of a region in 64 bits, in the order of the triplets."""
    s, m = g.shape
    f = torch.lgamma(torch.arange(s + 2, dtype=torch.float64, device=g.device) + 1)
    tri = torch.combinations(torch.arange(m, device=g.device), 3)
    out = []
    hot = [torch.stack([(g[ph == c] == v) for v in range(3)]).to(torch.float32) for c in (0, 1)]
    for i in range(m - 2):
        t = tri[tri[:, 0] == i]
        tot = torch.zeros(len(t), dtype=torch.float64, device=g.device)
        for a in range(3):
            for b in range(3):
                for d in range(3):
                    n = [((h[b] * h[a][:, i:i + 1]).T @ h[d])[t[:, 1], t[:, 2]].round().to(torch.int64) for h in hot]
                    tot += f[n[0] + n[1] + 1] - f[n[0]] - f[n[1]]
        out.append(tot)
    return torch.cat(out).cpu().numpy()


def exact(case, seed):
    kind, m = case["kind"], case["snps"]
    cost = _triplets(m) * (case["samples"] + 3000) * case.get("count", 1)
    if kind in ("shard", "batch") or cost > 2.5e12:
        return None
    torch.backends.cuda.matmul.allow_tf32 = False
    x = _inputs(case, seed)
    if kind == "region":
        return {"tables": None, "scores": _region(*x)}
    if kind == "replicates":
        return {"score": np.concatenate([_all_scores(x[0], p, 1) for p in x[2]]), "ijk": None}
    top = _all_scores(x[0], x[2][0] if kind == "permute" else x[1], 32 if kind == "topk" else 1)
    if kind == "topk":
        return {"score": top, "ijk": None, "score64": top}
    return {"score": top, "ijk": None}
