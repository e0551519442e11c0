// Genotype-split tensor-core search (tcgen05 block-scaled FP4 on CTA pairs, sm_100a).
//
// Same result as k_scan_tc, the integer engine and the reference's kernel_epi
// (GPU/v4.cpp:295-594): exact tables, K2 in the reference's FP32 order, lowest (score, i, j, k).
//
// Two things make it cheaper than counting the 8 cells of (i, j, k) over all samples:
//
// 1. For a fixed first SNP i the samples of a class are sorted by their genotype of i, and only
//    the two rarer genotypes are counted:
//      D_g[(k, c)][(j, b)] = sum over the samples of group g of x_c(k) x_b(j),  b, c in {0, 1},
//    four products per triplet and sample of a counted group instead of eight per sample.  The
//    counted groups hold at most 2/3 of the samples (0.41 on average for minor-allele frequencies
//    uniform in [0.05, 0.5]); the cells of the most frequent genotype follow from the (j, k)
//    margins by inclusion-exclusion, as the cells with genotype 2 of j or k do.  No operand holds
//    a product of two SNPs any more: both are plain indicator rows.  The sorting itself is one
//    pass of bit transposes per i (k_split_lists, k_split_planes), 1-7 % of a search.
// 2. A triplet's 27 cells are first put through a lower bound of K2 (screen_constants in
//    host_data.cpp: one reciprocal per cell and a few FP32 operations, no table).  Only where the
//    bound does not exceed the best score found so far (of the whole launch) is the score computed
//    in the reference's arithmetic.  The bound is below the score by 1 to 2 on average, by 3 to 6
//    where cases are 5 % or fewer.
//
// Warp roles of a CTA (512 threads), concurrent from tile to tile:
//   warps 0-5   produce: expand the compacted bit planes into the operand ring (warps 0-3 the 64
//               SNPs k of this CTA, 4-5 its 28 SNPs j), a quad of 128 samples per stage, 8 stages; half of
//               them take the even, half the odd stages
//   warp 6      fences the stored stages and issues the products (even CTA)
//   warp 7      schedules: takes tiles from the queue, publishes descriptor, record and job
//   warps 8-15  score: copy a tile's four accumulators out of tensor memory into a 16-bit staging
//               buffer (class 0 in the low, class 1 in the high half of a word), which frees them
//               for the next tile, then complete, screen and select while that tile counts
// Classes of at most 65535 samples (the 16-bit halves).
//
// What bounds it: the scoring warps (about 330 instructions per 32 triplets, 27 more where the classes
// are not even: screen_constants) up to about 8192 samples: the loop alone takes 340 clocks per
// scheduler and 32 triplets, in the kernel 430 to 530, for the producing warps issue beside it.  From
// there on also the round trip of a ring stage (stores, fence and arrival in the even CTA, products,
// commit).  What the parts of that round trip cost sets the roles and hand-offs (clocks, measured
// alone): a commit of four products 560; an arrival in the other CTA 133, and 447 with a cluster-scope
// release; issuing four products and their commit 330 from a converged warp, 610 from a lane-0 branch;
// a wait on a barrier that is complete 111, which passes during the issue of the stage before.
// Whole calls against what the other kernels take in their fastest configuration: 1024 x 8192 12.9 -> 3.94
// ms, 3072 x 4096 224 -> 79.2, 2048 x 8192 97 -> 26.9, an eighth of 4096 x 16384 141 -> 32.5.
//
// A step that is scored (exact_score) costs four times a screened one.  Usual data score 1e-5 to 2e-3
// of the steps, the more the fewer triplets there are to learn the threshold from; data whose scores
// are equal (constant or equal SNPs) all of them: split_screens in api.cu keeps most of those away.
//
// Every mbarrier wait is bounded; on expiry the kernel sets an error word and ends.  A producing warp then
// goes on to the end of its tile and may overwrite a stage that is still to be multiplied: counts that come
// of it are wrong, but 16 bits wide, and the ln n! table can be read for any such (dataset_layout).
#include <atomic>
#include <cfloat>
#include <type_traits>

#include "epik2_internal.h"
#include "scan_common.cuh"
#include "tc_ptx.cuh"

namespace epik2 {

// ------------------------------------------------------------------ sorting by genotype of i

// 32 x 32 bit transpose across a warp: lane l, bit b -> lane b, bit l.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(kFull, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

// What a search needs once, for job blockIdx.y, by ranges of blockIdx.x (a part of a search: from its
// first SNP on):
// [0, row_blocks): rows[32w + b][q] from planes[w][32q ..], one warp per class word and four 32-SNP
// columns;
// [row_blocks, row_blocks + pair_blocks): the pair margins packed, class 0 in the low, class 1 in the
// high half of each count (16 bytes per pair instead of 32: one load and no packing per triplet, half
// the traffic; bound by memory);
// the last block: the row of no genotypes behind the others; the job's slots (and, by job 0, the
// candidate lists) emptied.
__global__ void __launch_bounds__(256) k_split_setup(const SplitJob* __restrict__ jobs, int row_blocks, int pair_blocks,
                                                     BestSlot* __restrict__ slots, int per_job,
                                                     BestSlot* __restrict__ cand, int n_cand) {
  const SplitJob& J = jobs[blockIdx.y];
  const int lane = threadIdx.x & 31;
  if ((int)blockIdx.x < row_blocks) {
    const int64_t m_pad = J.m_pad, words = (int64_t)J.w0 + J.w1;
    const int mwp = J.mwp, nq = mwp / 4;
    const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int64_t w = unit / nq;
    const int q = 4 * (int)(unit - w * nq);
    if (w >= words) return;
    uint2 v[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int64_t snp = 32 * (int64_t)(J.q0 + q + t) + lane;
      v[t] = snp < m_pad ? __ldg(J.planes + w * m_pad + snp) : make_uint2(0, 0);
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
      v[t].x = transpose32(v[t].x, lane);
      v[t].y = transpose32(v[t].y, lane);
    }
    uint4* dst = reinterpret_cast<uint4*>(J.rows + (32 * w + lane) * (int64_t)mwp + q);
    dst[0] = make_uint4(v[0].x, v[0].y, v[1].x, v[1].y);
    dst[1] = make_uint4(v[2].x, v[2].y, v[3].x, v[3].y);
  } else if ((int)blockIdx.x < row_blocks + pair_blocks) {
    const uint4* __restrict__ src = J.pairs;
    uint4* __restrict__ dst = J.pairs16;
    for (int64_t x = J.pair0 + (int64_t)((int)blockIdx.x - row_blocks) * 256 + threadIdx.x; x < J.tri; x += (int64_t)pair_blocks * 256) {
      const uint4 a = __ldg(src + x), b = __ldg(src + J.tri + x);
      dst[x] = make_uint4(a.x | (b.x << 16), a.y | (b.y << 16), a.z | (b.z << 16), a.w | (b.w << 16));
    }
  } else {
    for (int x = threadIdx.x; x < J.mwp; x += 256) J.rows[32 * ((int64_t)J.w0 + J.w1) * J.mwp + x] = make_uint2(0, 0);
    BestSlot empty{};
    empty.score = FLT_MAX;
    empty.key = ~0ull;
    for (int x = threadIdx.x; x < per_job; x += 256) slots[(int64_t)blockIdx.y * per_job + x] = empty;
    if (blockIdx.y == 0)
      for (int x = threadIdx.x; x < n_cand; x += 256) cand[x] = empty;
  }
}

// First of a search's chunk: blocks [0, 2n) make the sample lists of record b / 2, class b % 2; the
// others the tile queue (split_tiles).
//
// Lists: the row numbers of each group's samples, up to the end of its last quad the empty row's.  Bound
// by latency: a thread takes a class word of 32 samples and the rows meet in shared memory, from where
// they leave side by side (256 x 100000: 34 us; written from where they were found, 64).
//
// Tile queue: one block per run of records and j block u; the run's tiles of that j block follow one
// another record by record, so the CTAs working at the same time share the (j, k) margins through L2.
// The blocks take their place in the queue from the cursor (any order is correct).
constexpr int kListThreads = 256;

__device__ void split_tiles(const SplitJob* __restrict__ jobs, const SplitRec* __restrict__ recs, const SplitRun run,
                            int u, uint64_t* __restrict__ tiles, unsigned* __restrict__ cursor) {
  __shared__ unsigned s_warp[kListThreads / 32], s_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = jobs[recs[run.rec0].job].m, i0 = recs[run.rec0].i;  // the run's records are i0, i0 + 1, ...
  auto count = [&](int i) { return (unsigned)tiles_of_pair_block((int64_t)i + 1 + kSplitJ * u, m, kSplitK); };
  if (count(i0) == 0) return;  // the run's smallest i has the most tiles
  for (int r0 = 0; r0 < run.n; r0 += kListThreads) {
    const int r = r0 + tid;
    const unsigned n = r < run.n ? count(i0 + r) : 0u;
    unsigned x = n;  // inclusive sum over the block
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned y = __shfl_up_sync(kFull, x, off);
      if (lane >= off) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    unsigned before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kListThreads / 32; w++) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
    if (tid == 0) s_base = atomicAdd(cursor, total);
    __syncthreads();
    const unsigned at = s_base + before + x - n;
    for (unsigned t = 0; t < n; t++) tiles[at + t] = pack_split_tile((uint32_t)(run.rec0 + r), (uint32_t)u, t);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kListThreads)
    k_split_lists(const SplitJob* __restrict__ jobs, SplitRec* __restrict__ recs, int n_recs, int32_t* __restrict__ lists,
                  const SplitRun* __restrict__ runs, int max_blocks, uint64_t* __restrict__ tiles,
                  unsigned* __restrict__ cursor) {
  __shared__ uint2 s_sum[kListThreads / 32];
  __shared__ int s_rows[32 * kListThreads];
  if (blockIdx.x >= 2u * (unsigned)n_recs) {
    const int b = (int)(blockIdx.x - 2u * (unsigned)n_recs);
    split_tiles(jobs, recs, runs[b / max_blocks], b % max_blocks, tiles, cursor);
    return;
  }
  SplitRec& rec = recs[blockIdx.x >> 1];
  const int c = (int)(blockIdx.x & 1u);
  const SplitJob& J = jobs[rec.job];
  const int i = rec.i, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int n[2][3];
#pragma unroll
  for (int x = 0; x < 2; x++) {
    n[x][0] = (int)J.singles[((int64_t)x * J.m_pad + i) * 2];
    n[x][1] = (int)J.singles[((int64_t)x * J.m_pad + i) * 2 + 1];
    n[x][2] = (x ? J.n1 : J.n0) - n[x][0] - n[x][1];
  }
  const int t0 = n[0][0] + n[1][0], t1 = n[0][1] + n[1][1], t2 = n[0][2] + n[1][2];
  const int gC = (t0 >= t1 && t0 >= t2) ? 0 : (t1 >= t2 ? 1 : 2);
  const int gA = gC == 0 ? 1 : 0, gB = gC == 2 ? 1 : 2;
  int qend[4], q = 0;
#pragma unroll
  for (int g = 0; g < 4; g++) {
    const int* nc = n[g >> 1];
    const int want = (g & 1) ? gB : gA;
    const int cnt = want == 0 ? nc[0] : want == 1 ? nc[1] : nc[2];
    q += cnt > 0 ? (cnt + 127) / 128 : 1;
    qend[g] = q;
  }
  if (c == 0 && tid == 0) {
#pragma unroll
    for (int g = 0; g < 4; g++) rec.qend[g] = qend[g];
    rec.genos = gA | (gB << 2) | (gC << 4);
  }
  int32_t* list = lists + rec.list_off;
  const int words = c ? J.w1 : J.w0, wb = c ? J.w0 : 0, ncls = c ? J.n1 : J.n0;
  int posA = 128 * (c ? qend[1] : 0), posB = 128 * (c ? qend[2] : qend[0]);
  for (int base = 0; base < words; base += kListThreads) {
    const int w = base + tid;
    uint32_t ma = 0, mb = 0;
    if (w < words) {
      const uint2 v = __ldg(J.planes + (int64_t)(wb + w) * J.m_pad + i);
      const int left = ncls - 32 * w;
      const uint32_t valid = left >= 32 ? kFull : ((1u << left) - 1u);
      const uint32_t m2 = ~(v.x | v.y) & valid;
      ma = gA == 0 ? v.x : v.y;
      mb = gB == 1 ? v.y : m2;
    }
    const int ca = __popc(ma), cb = __popc(mb);
    int xa = ca, xb = cb;  // inclusive sums over the block
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int ya = __shfl_up_sync(kFull, xa, off), yb = __shfl_up_sync(kFull, xb, off);
      if (lane >= off) {
        xa += ya;
        xb += yb;
      }
    }
    if (lane == 31) s_sum[warp] = make_uint2((uint32_t)xa, (uint32_t)xb);
    __syncthreads();
    int ba = 0, bb = 0, ta = 0, tb = 0;
#pragma unroll
    for (int x = 0; x < kListThreads / 32; x++) {
      const uint2 v = s_sum[x];
      if (x < warp) {
        ba += (int)v.x;
        bb += (int)v.y;
      }
      ta += (int)v.x;
      tb += (int)v.y;
    }
    int pa = ba + xa - ca, pb = ta + bb + xb - cb;  // in the staging buffer: A's, then B's
    const int row = 32 * (wb + w);
    while (ma) {
      s_rows[pa++] = row + __ffs(ma) - 1;
      ma &= ma - 1;
    }
    while (mb) {
      s_rows[pb++] = row + __ffs(mb) - 1;
      mb &= mb - 1;
    }
    __syncthreads();
    for (int x = tid; x < ta; x += kListThreads) list[posA + x] = s_rows[x];
    for (int x = tid; x < tb; x += kListThreads) list[posB + x] = s_rows[ta + x];
    posA += ta;
    posB += tb;  // (the next round's first barrier comes before its rows)
  }
  const int endA = 128 * (c ? qend[2] : qend[0]), endB = 128 * (c ? qend[3] : qend[1]);
  const int empty = 32 * (J.w0 + J.w1);
  for (int x = posA + tid; x < endA; x += kListThreads) list[x] = empty;
  for (int x = posB + tid; x < endB; x += kListThreads) list[x] = empty;
}

// 32 x 32 bit transpose inside a thread: word s, bit b -> word b, bit s (16 exchanges per step: two
// byte permutes each for the steps of 16 and 8 bits, four shifts and selects for the others).
__device__ __forceinline__ void transpose_words(uint32_t (&a)[32]) {
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint32_t x = a[k], y = a[k + 16];
    a[k] = prmt(x, y, 0x5410u);
    a[k + 16] = prmt(x, y, 0x7632u);
  }
#pragma unroll
  for (int k = 0; k < 32; k++)
    if (!(k & 8)) {
      const uint32_t x = a[k], y = a[k + 8];
      a[k] = prmt(x, y, 0x6240u);
      a[k + 8] = prmt(x, y, 0x7351u);
    }
#pragma unroll
  for (int j = 4; j > 0; j >>= 1) {
    const uint32_t m = j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int k = 0; k < 32; k++)
      if (!(k & j)) {
        const uint32_t x = a[k], y = a[k + j];
        a[k] = (x & m) | ((y << j) & ~m);
        a[k + j] = ((x >> j) & m) | (y & ~m);
      }
  }
}

// Compacted planes: per record and quad of 128 samples, the four words of g0 and of g1 of every SNP
// (32 bytes, so that a warp of the search reads 1 KiB).  A block of four warps takes 32 pieces of 32
// SNPs each (a piece: one quad and one 32-SNP column; as many quads as columns are short of 32);
// warp w makes word w: each lane reads the row words of its column for the 32 samples (coalesced
// across the lanes) and transposes them in its registers.  The words meet in shared memory, [plane,
// w][bit][piece] with rows of 33, and leave as whole SNPs.  Bound by the transposes (integer pipe):
// 1024 x 8192 with uniform genotypes takes 267 us per search, 450 with transposes by shuffles across
// the lanes.
constexpr int kPlaneThreads = 128;
__global__ void __launch_bounds__(kPlaneThreads) k_split_planes(const SplitJob* __restrict__ jobs, const SplitRec* __restrict__ recs,
                                                                const int32_t* __restrict__ lists, uint4* __restrict__ cp) {
  __shared__ uint32_t s_word[8 * 32 * 33];
  const SplitRec& rec = recs[blockIdx.y];
  const int mlen = rec.mlen, ncol = mlen / 32, nq = rec.qend[3];
  const int span = ncol > 16 ? 32 : ncol > 8 ? 16 : ncol > 4 ? 8 : 4;  // columns of a block
  const int sets = 32 / span, cblocks = (ncol + span - 1) / span;      // quads of a block; blocks across
  const int quad0 = (int)(blockIdx.x / (unsigned)cblocks) * sets, col0 = (int)(blockIdx.x % (unsigned)cblocks) * span;
  if (quad0 >= nq) return;
  const SplitJob& J = jobs[rec.job];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  {
    const int quad = quad0 + lane / span, col = col0 + lane % span;
    const bool on = quad < nq && col < ncol;
    const int4* list = reinterpret_cast<const int4*>(lists + rec.list_off + 128 * (on ? quad : quad0) + 32 * w);
    const uint2* rows = J.rows + (rec.qlo - J.q0) + (on ? col : col0);
    const int mwp = J.mwp;
    uint32_t x[32], y[32];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const int4 s = __ldg(list + t);
      const uint2 r0 = __ldg(rows + (int64_t)s.x * mwp), r1 = __ldg(rows + (int64_t)s.y * mwp);
      const uint2 r2 = __ldg(rows + (int64_t)s.z * mwp), r3 = __ldg(rows + (int64_t)s.w * mwp);
      x[4 * t] = r0.x; x[4 * t + 1] = r1.x; x[4 * t + 2] = r2.x; x[4 * t + 3] = r3.x;
      y[4 * t] = r0.y; y[4 * t + 1] = r1.y; y[4 * t + 2] = r2.y; y[4 * t + 3] = r3.y;
    }
    transpose_words(x);
#pragma unroll
    for (int b = 0; b < 32; b++) s_word[(w * 32 + b) * 33 + lane] = x[b];
    transpose_words(y);
#pragma unroll
    for (int b = 0; b < 32; b++) s_word[((4 + w) * 32 + b) * 33 + lane] = y[b];
  }
  __syncthreads();
  for (int piece = w; piece < 32; piece += kPlaneThreads / 32) {  // lane = SNP of the piece's column
    const int quad = quad0 + piece / span, col = col0 + piece % span;
    if (quad >= nq || col >= ncol) continue;
    const uint32_t* p = s_word + lane * 33 + piece;
    uint4* dst = cp + rec.cp_off + 2 * ((int64_t)quad * mlen + 32 * col + lane);
    dst[0] = make_uint4(p[0], p[32 * 33], p[2 * 32 * 33], p[3 * 32 * 33]);
    dst[1] = make_uint4(p[4 * 32 * 33], p[5 * 32 * 33], p[6 * 32 * 33], p[7 * 32 * 33]);
  }
}

// ------------------------------------------------------------------ the search kernel

constexpr int kSProd = 6;            // producing warps
constexpr int kSScore = 8;           // scoring warps (the last ones): four pairs of warps
constexpr int kSPairs = kSScore / 2;
constexpr int kSPairJ = 28;          // SNPs j scored by a pair (x 32 SNPs k)
constexpr int kSFirstScore = kSProd + 2;
constexpr int kSThreads = 32 * (kSFirstScore + kSScore);
constexpr int kSStages = 8;
constexpr int kSRaw = 2;             // raw slots of a producing warp
constexpr int kSRowBytes = 64;       // a quad: 4 words of 32 samples, E2M1
constexpr uint32_t kSSbo = 8 * kSRowBytes;
constexpr int kSHalfJ = kSplitJ / 2; // SNPs j expanded by each CTA
constexpr int kSStageA = 128 * kSRowBytes;
constexpr int kSStageBytes = (128 + 2 * kSHalfJ) * kSRowBytes;
constexpr int kSStagingOff = kSStages * kSStageBytes;  // E[c][j][k]: uint4 words (u, b) = (A,0) (A,1) (B,0) (B,1)
constexpr int kSStagingBytes = 2 * kSplitJ * 64 * 16;
// Per pair of scoring warps: the margins of its SNPs j.
constexpr int kSPairOff = kSStagingOff + kSStagingBytes;
constexpr int kMargWords = 20;       // forms of (A, g_j), (B, g_j) for each g_j, then of each (C, g_j); row j of the pair table
constexpr int kSPairBytes = kSPairJ * kMargWords * 4;
constexpr int kSRawOff = kSPairOff + kSPairs * kSPairBytes;  // raw words: per producing warp kSRaw slots of 1 KiB
constexpr int kSSlotOff = kSRawOff + kSProd * kSRaw * 1024;
constexpr int kSSlotBytes = 64 + 128 + 16;        // record, job, descriptor
constexpr int kSBarOff = kSSlotOff + kSplitSlots * kSSlotBytes;
constexpr int kSSmemBytes = kSBarOff + 256;
static_assert(kSSmemBytes <= 232448 - 1024, "shared memory of one CTA");
static_assert(kSPairBytes % 16 == 0 && kSStagingOff % 128 == 0, "alignment");

constexpr int kCFull = 0, kCEmpty = 8, kCAcc = 16, kCDrained = 17, kCHand = 18, kCDesc = 21, kCRel = 24, kCFinal = 27;
// Accumulators of group g: columns [112g, 112g + 112).  Scale factors (UE8M0, per row and K group):
// columns [448, 480) for the first two K groups of a quad (2 and 1), [480, 512) for the others (1/2).
constexpr uint32_t kSSfCol = 448;
constexpr uint32_t kScale01 = 0x7F807F80u, kScale23 = 0x7E7E7E7Eu;
// kind::mxf4, M = 256 (pair), N = 112, K = 64; E2M1 operands, UE8M0 scales, FP32 accumulators
constexpr uint32_t kSIdesc = (1u << 7) | (1u << 10) | ((112u >> 3) << 17) | (1u << 23) | ((256u >> 4) << 24);

// Issued by one elected lane of a converged warp with warp-uniform operands: an instruction then
// takes 8 clocks to issue; from a lane-0 branch it takes 44 (every operand is moved to the uniform
// registers first), and the products of a stage 610 clocks instead of 330.
__device__ __forceinline__ void split_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate, uint32_t sfa,
                                          uint32_t sfb) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n\t}\n" ::"r"(
          d_tmem),
      "l"(a), "l"(b), "r"(kSIdesc), "r"(accumulate), "r"(sfa), "r"(sfb));
}
// Arrival on a barrier of the other CTA.  What it announces are stores to this CTA's own shared
// memory for its own tensor core (fence.proxy.async before) or completed reads of its own tensor
// memory, so no cluster-scope release: that one waits for earlier accesses of the thread and costs
// several hundred clocks.
__device__ __forceinline__ void bar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void split_commit(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}\n" ::"r"(
          bar),
      "h"((uint16_t)3)
      : "memory");
}

__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// 128 sample bits of one SNP and genotype -> four K groups of 32 E2M1 elements.  Group q holds bit q
// of every nibble of the four words: 0.5, 1 and 2 for q = 0, 1, 2 without a shift, and q = 3 moved
// to 2 (bit 3 is the sign).  Both operands hold the same values, so the products are 1/4, 1, 4 and
// 4; the scale factors of the K groups (kScale01, kScale23) make them 1.
__device__ __forceinline__ void store_quad(uint32_t at, uint4 w) {
  sts128(at, make_uint4(w.x & 0x11111111u, w.y & 0x11111111u, w.z & 0x11111111u, w.w & 0x11111111u));
  sts128(at + 128, make_uint4(w.x & 0x22222222u, w.y & 0x22222222u, w.z & 0x22222222u, w.w & 0x22222222u));
  sts128(at + 256, make_uint4(w.x & 0x44444444u, w.y & 0x44444444u, w.z & 0x44444444u, w.w & 0x44444444u));
  sts128(at + 384, make_uint4((w.x >> 1) & 0x44444444u, (w.y >> 1) & 0x44444444u, (w.z >> 1) & 0x44444444u,
                              (w.w >> 1) & 0x44444444u));
}

__device__ __forceinline__ bool bar_test(uint32_t bar, uint32_t parity) {  // without waiting
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint4 lds128(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr));
  return v;
}

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// w.lo * coef.byte0 + w.hi * coef.byte1 + c, unsigned halves, signed bytes
__device__ __forceinline__ int dot2(uint32_t w, uint32_t coef, int c) {
  int r;
  asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(coef), "r"(c));
  return r;
}

// The two linear forms of a cell (a controls, b cases) that the screening bound needs, as the bits of
// FP32 numbers: n = 2^20 + N with N = a + b + 1 (a step of the bits is 1/8), and d = 1.5 * 2^23 + 64 D
// with 64 D = 64 (a + 1/2) - kp N.  N stays below 2^18 and 64 D below 2^22 for 16-bit counts, so adding
// and subtracting the bits adds and subtracts the numbers, and one FP32 subtraction converts (an integer
// conversion takes twice the pipe time); that of n leaves N + 7/16, the number the bound wants, whose
// sixteenths 2^20 - 7/16 can hold.  A margin over x cells holds the sums of its cells' bits modulo 2^32,
// so that cells complete by integer subtraction.
constexpr uint32_t kBitsN = 0x49800000u, kBitsD = 0x4B400000u;
constexpr float kLessN = 1048576.0f - kScreenShift;
struct Form {
  uint32_t n, d;
};
__device__ __forceinline__ Form operator-(Form x, Form y) { return Form{x.n - y.n, x.d - y.d}; }
struct FormOf {  // counts (class 0 low half, class 1 high half) of a sum over `cells` cells -> forms
  uint32_t coef;   // bytes (64 - kp, -kp)
  int bias;        // 32 - kp
  __device__ __forceinline__ Form operator()(uint32_t w, int cells) const {
    return Form{(uint32_t)dot2(w, 0x0808u, (int)((kBitsN + 8u) * (uint32_t)cells)),
                (uint32_t)dot2(w, coef, (int)((kBitsD + (uint32_t)bias) * (uint32_t)cells))};
  }
};

// Lower bound of K2 (screen_constants in host_data.cpp), cell by cell: per cell one reciprocal, six
// FP32 operations (five for even classes, where theta1 is 0) and half an integer addition.
template <bool kEven>
struct Screen {
  float theta1, theta2;  // of 64 D
  float acc;
  uint32_t bits;         // sum of the cells' log2 (N + 7/16), from below, in units of 2^-23
  template <int kN>
  __device__ __forceinline__ void cells(const Form (&f)[kN]) {
    float D[kN], M[kN], r[kN];
#pragma unroll
    for (int x = 0; x < kN; x++) {
      D[x] = __uint_as_float(f[x].d) - 12582912.0f;
      M[x] = __uint_as_float(f[x].n) - kLessN;
    }
#pragma unroll
    for (int x = 0; x < kN; x++) {
      const float P = fmaf(fabsf(D[x]), -theta2, M[x]);
      r[x] = rcp_approx(kEven ? P : fmaf(D[x], -theta1, P));
    }
    // (the order of the sums is the faster one of either form: 4096 x 16384 with the other one 2 % slower,
    // 1136 x 18638 with a third of cases 1.5 %)
    if (kEven) {
#pragma unroll
      for (int x = 0; x + 1 < kN; x += 2) bits += __float_as_uint(M[x]) + __float_as_uint(M[x + 1]);
      if (kN & 1) bits += __float_as_uint(M[kN - 1]);
#pragma unroll
      for (int x = 0; x < kN; x++) acc = fmaf(D[x] * r[x], D[x], acc);
    } else {
#pragma unroll
      for (int x = 0; x < kN; x++) {
        acc = fmaf(D[x] * r[x], D[x], acc);
        bits += __float_as_uint(M[x]);
      }
    }
  }
};

// The other cells of one genotype of j, from those with g_k = 0 and 1 (f[0], f[1]: A; f[3], f[4]: B;
// f[6], f[7]: C) and the margins (A, j), (B, j), (C, j): one subtraction of three terms per form.
__device__ __forceinline__ void row_forms(Form ijA, Form ijB, Form ijC, Form (&f)[9]) {
  f[2] = ijA - f[0] - f[1];
  f[5] = ijB - f[3] - f[4];
  f[8] = ijC - f[6] - f[7];
}

// Cells of one counted genotype of i from its four counts: t[3b + c].
__device__ __forceinline__ void counted_cells(uint32_t t00, uint32_t t01, uint32_t t10, uint32_t t11, uint32_t ij0,
                                              uint32_t ij1, uint32_t ij2, uint32_t ik0, uint32_t ik1, uint32_t (&t)[9]) {
  t[0] = t00;
  t[1] = t01;
  t[2] = ij0 - t00 - t01;
  t[3] = t10;
  t[4] = t11;
  t[5] = ij1 - t10 - t11;
  t[6] = ik0 - t00 - t10;
  t[7] = ik1 - t01 - t11;
  t[8] = ij2 - t[6] - t[7];
}

// Cells of the genotype of i that was not counted: (j, k) margins less the counted cells' sums.
__device__ __forceinline__ void dropped_cells(uint4 jk, uint32_t nj0, uint32_t nj1, uint32_t nj2, uint32_t nk0,
                                              uint32_t nk1, const uint32_t (&a)[9], const uint32_t (&b)[9],
                                              uint32_t (&t)[9]) {
  const uint32_t m02 = nj0 - jk.x - jk.y, m12 = nj1 - jk.z - jk.w;
  const uint32_t m20 = nk0 - jk.x - jk.z, m21 = nk1 - jk.y - jk.w, m22 = nj2 - m20 - m21;
  t[0] = jk.x - a[0] - b[0];
  t[1] = jk.y - a[1] - b[1];
  t[2] = m02 - a[2] - b[2];
  t[3] = jk.z - a[3] - b[3];
  t[4] = jk.w - a[4] - b[4];
  t[5] = m12 - a[5] - b[5];
  t[6] = m20 - a[6] - b[6];
  t[7] = m21 - a[7] - b[7];
  t[8] = m22 - a[8] - b[8];
}

// Counts (g_i = g, g_x = 0 and 1) from the packed counts c of the pair (i, x) and the singles of x.
__device__ __forceinline__ void by_genotype(uint4 c, uint32_t n0, uint32_t n1, int g, uint32_t& x0, uint32_t& x1) {
  x0 = g == 0 ? c.x : g == 1 ? c.z : n0 - c.x - c.z;
  x1 = g == 0 ? c.y : g == 1 ? c.w : n1 - c.y - c.w;
}

// K2 of triplet (i, j, k) in the reference's arithmetic and order from its eight staged words per
// class (e0: g_k = 0, e1: g_k = 1) and the margins in device memory; its table where one is
// wanted.  Not inlined: the search takes it for one triplet in a thousand or fewer.
__device__ __noinline__ float exact_score(uint4 e0, uint4 e1, const SplitJob* J, int i, int j, int k, int genos,
                                          uint32_t* table) {
  const int gA = genos & 3, gB = (genos >> 2) & 3, gC = genos >> 4;
  const int64_t m_pad = J->m_pad;
  auto single = [&](int x, uint32_t& n0, uint32_t& n1) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(J->singles) + x), b = __ldg(reinterpret_cast<const uint2*>(J->singles) + m_pad + x);
    n0 = a.x | (b.x << 16);
    n1 = a.y | (b.y << 16);
  };
  const uint32_t all = (uint32_t)J->n0 | ((uint32_t)J->n1 << 16);
  uint32_t ni[3], nj[3], nk[3];
  single(i, ni[0], ni[1]);
  single(j, nj[0], nj[1]);
  single(k, nk[0], nk[1]);
  ni[2] = all - ni[0] - ni[1];
  nj[2] = all - nj[0] - nj[1];
  const uint4 ij = __ldg(J->pairs16 + tri_offset(m_pad, i, j)), ik = __ldg(J->pairs16 + tri_offset(m_pad, i, k));
  const uint4 jk = __ldg(J->pairs16 + tri_offset(m_pad, j, k));
  uint32_t t[3][9], x0, x1, y0, y1;
  by_genotype(ij, nj[0], nj[1], gA, x0, x1);
  by_genotype(ik, nk[0], nk[1], gA, y0, y1);
  counted_cells(e0.x, e1.x, e0.y, e1.y, x0, x1, (gA == 0 ? ni[0] : ni[1]) - x0 - x1, y0, y1, t[0]);
  by_genotype(ij, nj[0], nj[1], gB, x0, x1);
  by_genotype(ik, nk[0], nk[1], gB, y0, y1);
  counted_cells(e0.z, e1.z, e0.w, e1.w, x0, x1, (gB == 1 ? ni[1] : ni[2]) - x0 - x1, y0, y1, t[1]);
  dropped_cells(jk, nj[0], nj[1], nj[2], nk[0], nk[1], t[0], t[1], t[2]);
  const float* __restrict__ lut = J->lut;
  float score = 0.0f;
#pragma unroll
  for (int g = 0; g < 3; g++) {
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const uint32_t w = g == gC ? t[2][c] : ((g == 0 || (g == 1 && gC == 0)) ? t[0][c] : t[1][c]);
      const uint32_t a = w & 0xFFFFu, b = w >> 16;
      const float d = __fsub_rn(__ldg(lut + a + b + 1), __ldg(lut + a));
      score = __fadd_rn(score, __fsub_rn(d, __ldg(lut + b)));
      if (table) {
        table[9 * g + c] = a;
        table[27 + 9 * g + c] = b;
      }
    }
  }
  return fabsf(score);
}

template <bool kDump, bool kTopK, bool kEven>
__global__ void __launch_bounds__(kSThreads, 1) k_scan_split(const SplitParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ long long s_hand[kSplitSlots];  // odd CTA: descriptors handed over by the even CTA
  __shared__ int s_abort, s_fail[kSPairs];         // s_fail: one per pair of scoring warps
  const int tid = threadIdx.x, warp = __shfl_sync(kFull, tid >> 5, 0), lane = tid & 31;
  const uint32_t crank = cluster_rank();
  const bool even = crank == 0;
  const uint32_t sbase = smem_u32(smem), bar0 = sbase + kSBarOff;
  auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };
  auto slot_rec = [&](uint32_t t) { return reinterpret_cast<const SplitRec*>(smem + kSSlotOff + (t % kSplitSlots) * kSSlotBytes); };
  auto slot_job = [&](uint32_t t) { return reinterpret_cast<const SplitJob*>(smem + kSSlotOff + (t % kSplitSlots) * kSSlotBytes + 64); };
  auto slot_desc = [&](uint32_t t) { return reinterpret_cast<volatile long long*>(smem + kSSlotOff + (t % kSplitSlots) * kSSlotBytes + 192); };
  const long long wl = p.wait_limit > 0 ? p.wait_limit : kWaitLimit;
  volatile int* abort_flag = &s_abort;

  if (tid == 0) {
    for (int s = 0; s < kSStages; s++) {
      // + the odd CTA's issuing warp, + some that never come (test hook)
      bar_init(bar(kCFull + s), kSProd / 2 + (even ? 1 : 0) + (s == 0 && p.test_withhold == (int)blockIdx.x + 1 ? 1000 : 0));
      bar_init(bar(kCEmpty + s), 1);
    }
    bar_init(bar(kCAcc), 1);
    bar_init(bar(kCDrained), 2 * kSScore);  // both CTAs' scoring warps arrive in the even one
    for (int s = 0; s < kSplitSlots; s++) {
      bar_init(bar(kCHand + s), 1);
      bar_init(bar(kCDesc + s), 1);
      bar_init(bar(kCRel + s), kSScore);
    }
    bar_init(bar(kCFinal), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
    for (int x = 0; x < kSPairs; x++) s_fail[x] = 0;
  }
  cluster_sync_all();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(kFull, s_tmem, 0);
  if (warp < 4) {
    const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) + kSSfCol;
    tmem_st16_fill(ta, kScale01);
    tmem_st16_fill(ta + 16, kScale01);
    tmem_st16_fill(ta + 32, kScale23);
    tmem_st16_fill(ta + 48, kScale23);
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();

  if (warp < kSProd) {
    // ================= producing warps =================
    // A: rows 64c + kk of this CTA's 64 SNPs k; B: rows 28b + jj of its 28 SNPs j.  A warp takes
    // one quad (4 words) of a stage for 32 SNPs: 32 bytes loaded, 8 x 16 bytes stored per lane.  The
    // words come by cp.async through the lane's own two raw slots, a stage ahead; the proxy fence
    // that the stores need is left to the issuing warp, since a fence here would wait for them.
    const bool isA = warp < 4;
    const int sub = isA ? warp >> 1 : warp - 4;
    const int x = isA ? 32 * (warp & 1) + lane : lane;           // row of genotype 0
    const int row1 = x + (isA ? 64 : kSHalfJ);                   // row of genotype 1
    const bool on = isA || lane < kSHalfJ;
    const uint32_t raw0 = sbase + kSRawOff + (uint32_t)(warp * kSRaw * 1024 + 16 * lane);
    const uint32_t off_base = isA ? 0u : (uint32_t)kSStageA;
    const uint32_t off0 = off_base + (uint32_t)(x >> 3) * kSSbo + (uint32_t)(x & 7) * 16;
    const uint32_t off1 = off_base + (uint32_t)(row1 >> 3) * kSSbo + (uint32_t)(row1 & 7) * 16;
    const uint32_t zero = (uint32_t)(wl >> 63);  // 0, unknown to the compiler
    uint32_t stage = 0;  // of the ring, counted over all tiles
    for (uint32_t t = 0;; t++) {
      const bool got = bar_wait(bar(kCDesc + (int)(t % kSplitSlots)), (t / kSplitSlots) & 1u, wl);
      if (__any_sync(kFull, !got)) {
        *abort_flag = 1;
        break;
      }
      const long long desc = *slot_desc(t);
      if (desc < 0) break;
      const SplitRec* R = slot_rec(t);
      const int nq = R->qend[3], mlen = R->mlen, first = (int)((stage + (uint32_t)sub) & 1u);
      const int j0 = R->i + 1 + kSplitJ * (int)(((uint64_t)desc >> 24) & 0x3FFFF);
      const int k0 = j0 + 1 + kSplitK * (int)(((uint64_t)desc >> 42) & 0xFFFF);
      const int snp = (isA ? k0 + 64 * (int)crank : j0 + kSHalfJ * (int)crank) + x - 32 * R->qlo;
      // (words past a row's end belong to no SNP that is scored; the buffer has room behind its last row)
      const uint4* next = p.cp + R->cp_off + 2 * ((int64_t)snp + (int64_t)first * mlen);
      const int64_t step = 4 * (int64_t)mlen;
      const int mine = (nq - first + 1) / 2;  // quads of this warp
      auto load = [&](int st, uint32_t after) {  // this lane's words of the warp's quad st into its raw slot
        if (st < mine) {
          const uint32_t to = raw0 + 1024u * (uint32_t)(st & 1) + after;
          cp_async16(to, next);
          cp_async16(to + 512u, next + 1);
          next += step;
        }
        cp_async_commit();
      };
      load(0, 0);
      load(1, 0);
      bool bad = false;
      for (int st = 0; st < mine; st++) {
        cp_async_wait<1>();
        const uint32_t from = raw0 + 1024u * (uint32_t)(st & 1);
        const uint4 va = lds128(from), vb = lds128(from + 512u);
        const uint32_t g = stage + (uint32_t)(first + 2 * st), slot = g % kSStages;
        const uint32_t phase = (g / kSStages & 1u) ^ 1u;  // the first round finds every slot empty
        const bool empty = bar_test(bar(kCEmpty) + 8u * slot, phase);
        load(st + 2, (va.w | vb.w) & zero);  // into the slot just read: not issued before the words are here
        if (!bad && !empty) bad = !bar_wait(bar(kCEmpty) + 8u * slot, phase, wl);
        if (on) {
          const uint32_t at = sbase + slot * (uint32_t)kSStageBytes;
          store_quad(at + off0, va);
          store_quad(at + off1, vb);
        }
        __syncwarp();
        if (lane == 0) bar_arrive(bar(kCFull) + 8u * slot);
      }
      stage += (uint32_t)nq;
      if (__any_sync(kFull, bad)) {
        *abort_flag = 1;
        break;
      }
    }
  } else if (warp == kSProd) {
    // ================= issuing warp =================
    // Fences the stored stages for the async proxy; the odd CTA's then tells the even one's, which
    // issues the products.  Everything it needs per stage stays in uniform registers: slot and phase
    // of the ring, and the accumulator column and rest of the current sample group.
    uint32_t slot = 0, phase = 0;
    bool ready = false;  // stage `slot` was found full already
    for (uint32_t t = 0;; t++) {
      bool bad = !bar_wait(bar(kCDesc + (int)(t % kSplitSlots)), (t / kSplitSlots) & 1u, wl);
      if (__any_sync(kFull, bad)) {
        *abort_flag = 1;
        break;
      }
      if (__shfl_sync(kFull, *slot_desc(t), 0) < 0) break;
      const SplitRec* R = slot_rec(t);
      const int e0 = __shfl_sync(kFull, R->qend[0], 0), e1 = __shfl_sync(kFull, R->qend[1], 0);
      const int e2 = __shfl_sync(kFull, R->qend[2], 0), nq = __shfl_sync(kFull, R->qend[3], 0);
      if (!even) {
        for (int q = 0; q < nq && !bad; q++) {
          if (!ready) bad = __any_sync(kFull, !bar_wait(bar(kCFull) + 8u * slot, phase, wl));
          fence_proxy_async();
          if (lane == 0) bar_arrive_remote(map_cta(bar(kCFull) + 8u * slot, 0));
          slot = slot + 1 == kSStages ? 0 : slot + 1;
          phase ^= slot == 0;
          ready = __all_sync(kFull, bar_test(bar(kCFull) + 8u * slot, phase));
        }
        if (bad) {
          *abort_flag = 1;
          break;
        }
        continue;
      }
      // the previous tile's accumulators have been copied out of both CTAs
      if (t > 0) bad = __any_sync(kFull, !bar_wait(bar(kCDrained), (t - 1) & 1u, wl));
      uint32_t d = tmem, acc = 0;
      int end = e0;  // of the current group
      for (int q = 0; q < nq && !bad; q++) {
        if (!ready) bad = __any_sync(kFull, !bar_wait(bar(kCFull) + 8u * slot, phase, wl));
        if (bad) break;
        fence_proxy_async();
        tc_fence_after();
        const uint32_t slot1 = slot + 1 == kSStages ? 0 : slot + 1, phase1 = phase ^ (slot1 == 0);
        const bool next = bar_test(bar(kCFull) + 8u * slot1, phase1);  // its latency passes during the issue
        const uint32_t sA = sbase + slot * (uint32_t)kSStageBytes;
        const uint64_t da = smem_desc(sA, kSSbo), db = smem_desc(sA + kSStageA, kSSbo);
        split_mma(d, da, db, acc, tmem + kSSfCol, tmem + kSSfCol + 16);
        split_mma(d, da + 16u, db + 16u, 1u, tmem + kSSfCol + 32, tmem + kSSfCol + 48);
        acc = 1;
        if (q + 1 == end) {  // every group has a quad, so the ends are distinct
          end = end == e0 ? e1 : (end == e1 ? e2 : nq);
          d += 112u;
          acc = 0;
        }
        split_commit(bar(kCEmpty) + 8u * slot);
        ready = __all_sync(kFull, next);
        slot = slot1;
        phase = phase1;
      }
      if (bad) {
        *abort_flag = 1;
        break;
      }
      split_commit(bar(kCAcc));
    }
  } else if (warp == kSProd + 1) {
    // ================= scheduling warp =================
    // Even CTA: ticket -> descriptor, handed to the odd CTA; both publish descriptor, record and
    // job of tile t in slot t % 3, free again once tile t - 3 has been scored.
    const unsigned n_tiles = *reinterpret_cast<const volatile unsigned*>(p.n_tiles);
    for (uint32_t t = 0;; t++) {
      const int sl = (int)(t % kSplitSlots);
      const uint32_t ph = (t / kSplitSlots) & 1u;
      long long d = -1;
      bool bad = false;
      if (lane == 0) {
        if (!even) {
          if (bar_wait_cluster(bar(kCHand + sl), ph, wl)) d = *reinterpret_cast<volatile long long*>(&s_hand[sl]);
          else bad = true;
        }
        if (t >= kSplitSlots && !bad) bad = !bar_wait(bar(kCRel + sl), ph ^ 1u, wl);
        if (even && !bad) {
          const unsigned ticket = atomicAdd(p.counter, 1u);
          if (ticket < n_tiles && !*abort_flag) d = (long long)__ldg(p.tiles + ticket);
        }
      }
      bad = __any_sync(kFull, bad);
      if (bad) {
        *abort_flag = 1;
        d = -1;
      }
      d = __shfl_sync(kFull, d, 0);
      if (even && lane == 0) {
        st_cluster_s64(map_cta(smem_u32(&s_hand[sl]), 1), d);
        bar_arrive_cluster(map_cta(bar(kCHand + sl), 1));
      }
      uint32_t* sw = reinterpret_cast<uint32_t*>(smem + kSSlotOff + sl * kSSlotBytes);
      if (d >= 0) {
        const SplitRec* R = p.recs + ((uint64_t)d & 0xFFFFFF);
        if (lane < 16) sw[lane] = reinterpret_cast<const uint32_t*>(R)[lane];
        const SplitJob* J = p.jobs + R->job;
        sw[16 + lane] = reinterpret_cast<const uint32_t*>(J)[lane];
      }
      if (lane == 0) *slot_desc(t) = d;
      __syncwarp();
      if (lane == 0) bar_arrive(bar(kCDesc + sl));
      if (d < 0) break;
    }
  } else if (warp >= kSFirstScore) {
    // ================= scoring warps =================
    // Warp (c, kh, part): drains rows c of the SNPs k 32kh.. and columns of half of the SNPs
    // j; the pair of warps with the same (kh, part) shares its part of the staging buffer and its margins
    // and nothing else, so the pairs go from tile to tile by themselves (less than a tile apart).
    const int sw = warp - kSFirstScore;
    const int quarter = warp & 3, kh = quarter & 1, c = quarter >> 1, part = sw >> 2;
    const int pt = 32 * c + lane;  // thread of the pair
    const int pair = kh + 2 * part, pbar = 1 + pair;
    const int pj = 28 * part, nj = 28;  // its SNPs j in the tile
    volatile int* const fail = &s_fail[pair];
    int* const marg = reinterpret_cast<int*>(smem + kSPairOff + pair * kSPairBytes);
    float best_s = FLT_MAX, list_s = FLT_MAX;
    unsigned long long best_k = ~0ull, list_k = ~0ull;
    unsigned thr = 0x7F7F7F7Fu, known = thr;  // bits of the score to reach; of the one last read
    if (kTopK) {  // continue the lists of the earlier launches of this search
      const BestSlot& e = p.cand[((int64_t)blockIdx.x * kSScore + sw) * 32 + lane];
      list_s = e.score;
      list_k = e.key;
    }
    int cur_job = -1;
    auto flush_job = [&](int jb) {  // this warp's best of job jb into its slot
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const float os = __shfl_xor_sync(kFull, best_s, off);
        const unsigned long long ok = __shfl_xor_sync(kFull, best_k, off);
        if (better(os, ok, best_s, best_k)) {
          best_s = os;
          best_k = ok;
        }
      }
      if (lane == 0) {
        BestSlot& slot = p.job_slots[((int64_t)jb * gridDim.x + blockIdx.x) * kSScore + sw];
        if (better(best_s, best_k, slot.score, slot.key)) {
          slot.score = best_s;
          slot.key = best_k;
        }
      }
      best_s = FLT_MAX;
      best_k = ~0ull;
    };
    long long desc = -1;
    bool got = bar_wait(bar(kCDesc), 0, wl);
    if (got) desc = *slot_desc(0);
    for (uint32_t t = 0;; t++) {
      bool ok = got;
      const SplitRec* R = slot_rec(t);
      const SplitJob* J = slot_job(t);
      int i = 0, m = 0, jp = 0, kb = 0;  // first SNP, SNPs; first SNP j and k of the pair
      // margins of this thread's SNP k and, in the pair's first threads, of a SNP j: in flight while the
      // tile's products complete and its accumulators are copied
      uint4 ik, ij;
      uint2 sk0, sk1, sj0, sj1, si0, si1;
      if (ok && desc >= 0) {
        i = R->i;
        m = J->m;
        jp = i + 1 + kSplitJ * (int)(((uint64_t)desc >> 24) & 0x3FFFF);
        kb = jp + 1 + kSplitK * (int)(((uint64_t)desc >> 42) & 0xFFFF) + 64 * (int)crank + 32 * kh;
        jp += pj;
        const int64_t m_pad = J->m_pad;
        const uint4* pi = J->pairs16 + tri_offset(m_pad, i, i + 1) - (i + 1);  // + x: pair (i, x)
        const uint2* si = reinterpret_cast<const uint2*>(J->singles);
        const int xk = min(kb + lane, m - 1), xj = min(jp + (pt < nj ? pt : 0), m - 1);  // both > i
        ik = __ldg(pi + xk);
        sk0 = __ldg(si + xk);
        sk1 = __ldg(si + m_pad + xk);
        ij = __ldg(pi + xj);
        sj0 = __ldg(si + xj);
        sj1 = __ldg(si + m_pad + xj);
        si0 = __ldg(si + i);
        si1 = __ldg(si + m_pad + i);
        if (lane == 0) known = *reinterpret_cast<volatile unsigned*>(p.thr + R->job);
        ok = bar_wait(bar(kCAcc), t & 1u, wl);
      }
      // Both warps leave together or not at all: the pair's flag is written only before this
      // barrier and read only between it and the next one.
      if (!ok) *abort_flag = 1;
      if (!ok || *abort_flag) *fail = 1;
      pair_sync(pbar);  // both warps are done with the staging buffer and the margins
      if (desc < 0 || *fail) break;
      known = __shfl_sync(kFull, known, 0);
      if (R->job != cur_job) {
        if (cur_job >= 0) flush_job(cur_job);
        cur_job = R->job;
        thr = known;
      }
      thr = min(thr, known);
      const int genos = R->genos, gA = genos & 3, gB = (genos >> 2) & 3;
      tc_fence_after();
      // accumulators -> staging
      const uint32_t Ek = sbase + kSStagingOff + (uint32_t)((pj * 64 + 32 * kh + lane) * 16);
      {
        const uint32_t ta = tmem + ((uint32_t)(32 * quarter) << 16);
        const uint32_t dst = Ek + (uint32_t)(c * kSplitJ * 64 * 16);
        // Eight SNPs j per wait, then four: the loads' latency is paid four times instead of seven
        // (3072 x 4096 82.9 -> 79.1 ms).
        auto drain = [&](int jj, auto quads) {
          constexpr int kQ = decltype(quads)::value;
          const uint32_t tc = ta + (uint32_t)(2 * kSHalfJ * part + jj);  // SNP j of half h: 28h further
          uint32_t v[kQ][4][2][4];
#pragma unroll
          for (int h = 0; h < kQ; h++)
#pragma unroll
            for (int g = 0; g < 4; g++)
#pragma unroll
              for (int b = 0; b < 2; b++) tmem_ld4(tc + (uint32_t)(112 * g + kSHalfJ * b + 4 * h), v[h][g][b]);
          tmem_wait_ld();
          const float magic = 8388608.0f;
#pragma unroll
          for (int q = 0; q < 4 * kQ; q++) {
            uint32_t w[4];
#pragma unroll
            for (int ub = 0; ub < 4; ub++) {
              const uint32_t lo = __float_as_uint(__uint_as_float(v[q >> 2][ub >> 1][ub & 1][q & 3]) + magic);
              const uint32_t hi = __float_as_uint(__uint_as_float(v[q >> 2][2 + (ub >> 1)][ub & 1][q & 3]) + magic);
              w[ub] = prmt(lo, hi, 0x5410u);
            }
            sts128(dst + (uint32_t)((jj + q) * 64 * 16), make_uint4(w[0], w[1], w[2], w[3]));
          }
        };
        static_assert(kSPairJ == 28 && kSHalfJ == 28, "a pair's SNPs j are one half of the tile's");
#pragma unroll 1
        for (int jj = 0; jj < 24; jj += 8) drain(jj, std::integral_constant<int, 2>());
        drain(24, std::integral_constant<int, 1>());
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (even) bar_arrive(bar(kCDrained));
        else bar_arrive_remote(map_cta(bar(kCDrained), 0));
      }
      // margins as forms: per j into shared memory, per k (this thread's) in registers
      const uint32_t ntot = (uint32_t)J->n0 | ((uint32_t)J->n1 << 16);
      const FormOf form{J->coef, J->bias};
      if (pt < nj) {
        const uint32_t i0 = si0.x | (si1.x << 16), i1 = si0.y | (si1.y << 16);
        const uint32_t nA = gA == 0 ? i0 : i1, nB = gB == 1 ? i1 : ntot - i0 - i1;
        const uint32_t n0 = sj0.x | (sj1.x << 16), n1 = sj0.y | (sj1.y << 16);
        uint32_t wA[3], wB[3];
        const uint32_t wj[3] = {n0, n1, ntot - n0 - n1};
        by_genotype(ij, n0, n1, gA, wA[0], wA[1]);
        by_genotype(ij, n0, n1, gB, wB[0], wB[1]);
        wA[2] = nA - wA[0] - wA[1];
        wB[2] = nB - wB[0] - wB[1];
        int* o = marg + kMargWords * pt;
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const Form x = form(wA[b], 3), y = form(wB[b], 3), z = form(wj[b] - wA[b] - wB[b], 3);
          *reinterpret_cast<uint4*>(o + 4 * b) = make_uint4(x.n, x.d, y.n, y.d);
          *reinterpret_cast<uint2*>(o + 12 + 2 * b) = make_uint2(z.n, z.d);
        }
        const int64_t j = min(jp + pt, m - 1);
        *reinterpret_cast<const uint4**>(o + 18) = J->pairs16 + (j * (J->m_pad - 1) - (j * (j - 1)) / 2 - j - 1);
      }
      Form kA0, kA1, kB0, kB1, kC0, kC1;
      {
        const uint32_t n0 = sk0.x | (sk1.x << 16), n1 = sk0.y | (sk1.y << 16);
        uint32_t a0, a1, b0, b1;
        by_genotype(ik, n0, n1, gA, a0, a1);
        by_genotype(ik, n0, n1, gB, b0, b1);
        kA0 = form(a0, 3);
        kA1 = form(a1, 3);
        kB0 = form(b0, 3);
        kB1 = form(b1, 3);
        kC0 = form(n0 - a0 - b0, 3);
        kC1 = form(n1 - a1 - b1, 3);
      }
      pair_sync(pbar);  // staging rows and margins are in place
      // complete, screen, select: lane = k, this warp's j = c, c + 2, ...
      // SNP jj of the pair makes a triplet with this lane's k if jj < lane_end (j < k < m)
      const int k = kb + lane;
      const int lane_end = k < m ? min(nj, k - jp) : 0, warp_end = min(nj, min(m - 1, kb + 31) - jp);
      Screen<kEven> scr;
      scr.theta1 = J->theta1;
      scr.theta2 = J->theta2;
      const float coef = -J->c, base = J->base;
      float limit = __uint_as_float(thr) - base;
      uint4 jk;
      // (j, k) margins of the pair's row jj
      auto load_jk = [&](int jj, uint4& a) {
        a = make_uint4(0, 0, 0, 0);
        if (jj < lane_end)
          a = __ldg(*reinterpret_cast<const uint4* const*>(marg + kMargWords * jj + 18) + k);
      };
      load_jk(c, jk);
      if (kb < m) {
#pragma unroll 1
        for (int jj = c; jj < warp_end; jj += 2) {
          const int j = jp + jj;
          const bool valid = jj < lane_end;
          const uint4 e0 = lds128(Ek + (uint32_t)(jj * 64 * 16));
          const uint4 e1 = lds128(Ek + (uint32_t)((kSplitJ + jj) * 64 * 16));
          bool want = valid;
          if (kDump) {
            load_jk(jj + 2, jk);
          } else {
            const Form q00 = form(jk.x, 3), q01 = form(jk.y, 3), q10 = form(jk.z, 3), q11 = form(jk.w, 3);
            load_jk(jj + 2, jk);
            const uint4* mj = reinterpret_cast<const uint4*>(marg + kMargWords * jj);
            auto margins = [&](int b, Form& ijA, Form& ijB, Form& ijC) {
              const uint4 x = mj[b];
              const uint2 y = *(reinterpret_cast<const uint2*>(mj + 3) + b);
              ijA = Form{x.x, x.y};
              ijB = Form{x.z, x.w};
              ijC = Form{y.x, y.y};
            };
            scr.acc = 0.0f;
            scr.bits = 0u;
            Form ijA, ijB, ijC, r0[9], r1[9], r2[9];
            margins(0, ijA, ijB, ijC);
            r0[0] = form(e0.x, 1);
            r0[1] = form(e1.x, 1);
            r0[3] = form(e0.z, 1);
            r0[4] = form(e1.z, 1);
            r0[6] = q00 - r0[0] - r0[3];
            r0[7] = q01 - r0[1] - r0[4];
            row_forms(ijA, ijB, ijC, r0);
            scr.cells(r0);
            margins(1, ijA, ijB, ijC);
            r1[0] = form(e0.y, 1);
            r1[1] = form(e1.y, 1);
            r1[3] = form(e0.w, 1);
            r1[4] = form(e1.w, 1);
            r1[6] = q10 - r1[0] - r1[3];
            r1[7] = q11 - r1[1] - r1[4];
            row_forms(ijA, ijB, ijC, r1);
            scr.cells(r1);
            margins(2, ijA, ijB, ijC);
            r2[0] = kA0 - r0[0] - r1[0];
            r2[1] = kA1 - r0[1] - r1[1];
            r2[3] = kB0 - r0[3] - r1[3];
            r2[4] = kB1 - r0[4] - r1[4];
            r2[6] = kC0 - r0[6] - r1[6];
            r2[7] = kC1 - r0[7] - r1[7];
            row_forms(ijA, ijB, ijC, r2);
            scr.cells(r2);
            // sum of logs: bits - 27 * 127 * 2^23 (modulo 2^32) in units of 2^-23 log2, half of it in ln
            const float lg = __uint2float_rn(scr.bits - 27u * 0x3F800000u);
            const float low = fmaf(kScreenLog, lg, coef * scr.acc);
            want = valid && !(low >= limit);  // not a number: take the exact path
          }
          if (!__any_sync(kFull, want)) continue;
          float sc = FLT_MAX;
          unsigned long long key = ~0ull;
          if (want) {
            uint32_t table[kDump ? 54 : 1];
            sc = exact_score(e0, e1, J, R->i, j, k, R->genos, kDump ? table : nullptr);
            const int i1 = R->i;
            key = pack_key((uint64_t)i1, (uint64_t)j, (uint64_t)k);
            if (kDump) {
              const int64_t ti = triplet_index(m, i1, j, k);
#pragma unroll
              for (int x = 0; x < 54; x++) p.dump_tables[ti * 54 + x] = table[kDump ? x : 0];
              p.dump_scores[ti] = sc;
            }
            if (better(sc, key, best_s, best_k)) {
              best_s = sc;
              best_k = key;
            }
          }
          unsigned reach = __float_as_uint(sc);  // FLT_MAX where not wanted
          if (kTopK) {
            const float ts = __shfl_sync(kFull, list_s, 31);
            const unsigned long long tk = __shfl_sync(kFull, list_k, 31);
            unsigned todo = __ballot_sync(kFull, want && better(sc, key, ts, tk));
            while (todo) {
              const int src = __ffs(todo) - 1;
              todo &= todo - 1;
              const float cs = __shfl_sync(kFull, sc, src);
              const unsigned long long ck = __shfl_sync(kFull, key, src);
              const float ts2 = __shfl_sync(kFull, list_s, 31);
              const unsigned long long tk2 = __shfl_sync(kFull, list_k, 31);
              if (better(cs, ck, ts2, tk2)) warp_list_insert(list_s, list_k, cs, ck, lane);
            }
            // 32 triplets reach this warp's last entry: no triplet above it is among the best 32
            reach = __float_as_uint(__shfl_sync(kFull, list_s, 31));
          }
          reach = __reduce_min_sync(kFull, reach);
          // Also without an improvement the lowest score known by now is read: early in a search the warps
          // learn from one another within a tile.  Only a lower one is written: an atomic at every such
          // step took 1.97 ms instead of 1.73 for 512 x 8192 constant SNPs, which are all scored.
          const unsigned now = *reinterpret_cast<volatile unsigned*>(p.thr + cur_job);
          if (lane == 0 && reach < now) atomicMin(p.thr + cur_job, reach);
          thr = min(reach, now);
          limit = __uint_as_float(thr) - base;
        }
      }
      __syncwarp();
      if (lane == 0) bar_arrive(bar(kCRel + (int)(t % kSplitSlots)));  // done with tile t's slot
      got = bar_wait(bar(kCDesc + (int)((t + 1) % kSplitSlots)), ((t + 1) / kSplitSlots) & 1u, wl);
      desc = got ? *slot_desc(t + 1) : -1;
    }
    if (cur_job >= 0) flush_job(cur_job);
    if (kTopK) {
      BestSlot& e = p.cand[((int64_t)blockIdx.x * kSScore + sw) * 32 + lane];
      e.score = list_s;
      e.key = list_k;
    }
  }

  // ---- teardown: every role has left its loop; tensor memory is released only after every
  // product has completed (bounded wait on one more commit)
  if (warp == kSProd && lane == 0) {
    if (even) mma_commit_pair(bar(kCFinal));
    if (!bar_wait(bar(kCFinal), 0, wl)) s_abort = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (s_abort && tid == 0) atomicExch(p.err, 1);
  cluster_sync_all();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

int split_score_warps() { return kSScore; }

template <bool kD, bool kT, bool kE>
static cudaError_t split_set_smem() {
  return cudaFuncSetAttribute(k_scan_split<kD, kT, kE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSSmemBytes);
}

cudaError_t split_configure() {
  static std::atomic<uint64_t> configured{0};  // bit per device: the attribute belongs to one
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (configured.load() & bit) return cudaSuccess;
  e = split_set_smem<false, false, false>();
  if (e == cudaSuccess) e = split_set_smem<false, false, true>();
  if (e == cudaSuccess) e = split_set_smem<true, false, false>();
  if (e == cudaSuccess) e = split_set_smem<false, true, false>();
  if (e == cudaSuccess) e = split_set_smem<false, true, true>();
  if (e == cudaSuccess) configured |= bit;
  return e;
}

// Candidates that can be among the best 32 in double precision: those within `margin` (twice the
// most that FP32 and FP64 scores differ by) of the score that 32 candidates of one warp reach.
__global__ void __launch_bounds__(256) k_split_collect(const BestSlot* __restrict__ cand, int n,
                                                       const unsigned* __restrict__ thr, float margin,
                                                       BestSlot* __restrict__ out, unsigned* __restrict__ count) {
  const int x = (int)(blockIdx.x * 256 + threadIdx.x);
  if (x >= n) return;
  const BestSlot c = cand[x];
  if (c.key != ~0ull && c.score <= __uint_as_float(*thr) + margin) out[atomicAdd(count, 1u)] = c;
}

cudaError_t launch_split_collect(const BestSlot* cand, int n, const unsigned* thr, float margin, BestSlot* out,
                                 unsigned* count, cudaStream_t stream) {
  k_split_collect<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(cand, n, thr, margin, out, count);
  return cudaGetLastError();
}

cudaError_t launch_split_setup(const SplitJob* jobs, int n_jobs, int64_t max_units, int64_t max_tri, BestSlot* slots,
                               int per_job, BestSlot* cand, int n_cand, cudaStream_t stream) {
  if (n_jobs <= 0) return cudaSuccess;
  const int row_blocks = (int)((max_units + 7) / 8);
  const int pair_blocks = (int)(max_tri / 256 < 4095 ? max_tri / 256 + 1 : 4096);
  k_split_setup<<<dim3((unsigned)(row_blocks + pair_blocks + 1), (unsigned)n_jobs), 256, 0, stream>>>(
      jobs, row_blocks, pair_blocks, slots, per_job, cand, n_cand);
  return cudaGetLastError();
}

cudaError_t launch_split_prepare(const SplitJob* jobs, SplitRec* recs, int n, int max_quads, int max_cols,
                                 int32_t* lists, uint4* cp, const SplitRun* runs, int n_runs, int max_blocks,
                                 uint64_t* tiles, unsigned* cursor, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int64_t blocks = 2 * (int64_t)n + (int64_t)n_runs * max_blocks;
  k_split_lists<<<(unsigned)blocks, kListThreads, 0, stream>>>(jobs, recs, n, lists, runs, max_blocks, tiles, cursor);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // blocks of a record: at most those of max_cols columns (fewer columns take more quads per block)
  const int span = max_cols > 16 ? 32 : max_cols > 8 ? 16 : max_cols > 4 ? 8 : 4;
  const int64_t units = (int64_t)((max_quads + 32 / span - 1) / (32 / span)) * ((max_cols + span - 1) / span);
  for (int at = 0; at < n; at += 65535) {
    const int c = n - at < 65535 ? n - at : 65535;
    k_split_planes<<<dim3((unsigned)units, (unsigned)c), kPlaneThreads, 0, stream>>>(jobs, recs + at, lists, cp);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <bool kD, bool kT, bool kE>
static cudaError_t launch_split(const SplitParams& p, int blocks, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(kSThreads);
  cfg.dynamicSmemBytes = kSSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_scan_split<kD, kT, kE>, p);
}

cudaError_t launch_scan_split(const SplitParams& p, int blocks, bool dump, bool even, cudaStream_t stream) {
  const cudaError_t ce = split_configure();
  if (ce != cudaSuccess) return ce;
  const int grid = blocks & ~1;
  cudaError_t e;
  if (dump)
    e = launch_split<true, false, false>(p, grid, stream);
  else if (p.top_k > 1)
    e = even ? launch_split<false, true, true>(p, grid, stream) : launch_split<false, true, false>(p, grid, stream);
  else
    e = even ? launch_split<false, false, true>(p, grid, stream) : launch_split<false, false, false>(p, grid, stream);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace epik2
