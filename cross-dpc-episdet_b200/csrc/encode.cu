// Genotype encoding and the per-SNP / per-pair count tables.
//
// encode : uint8 genotypes [n_samples][n_snps] (the reference's sample-major layout,
//          GPU/v4.cpp:94) -> per-class {g0, g1} bit planes, word-major.  Replaces the
//          host loops data_to_binary + binary_to_tiled (GPU/v4.cpp:112-196).  As there,
//          genotype 2 (and any value other than 0/1) sets neither plane, so g2 is the
//          complement of g0|g1 inside the class and padding bits stay zero.
// counts : single-SNP counts n_c(g) and pair counts n_c(g_x, g_y) for g in {0,1}, the
//          lower-order margins from which the search derives every cell that involves
//          genotype 2 (inclusion-exclusion; no reference counterpart -- the reference
//          counts all 27 cells directly, GPU/v4.cpp:331-385).
#include "epik2_internal.h"

namespace epik2 {

// One thread per (class word, SNP).  Threads of a block cover consecutive SNPs so the
// reads of one sample row are coalesced; the sample index comes from the class-sorted
// permutation (broadcast).
__global__ void k_encode(const uint8_t* __restrict__ geno, const int32_t* __restrict__ perm, uint2* __restrict__ planes,
                         int64_t n_snps, int64_t m_pad, int64_t w0, int64_t w1, int64_t n0, int64_t n1) {
  const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= m_pad) return;
  const int64_t wt = w0 + w1;
  for (int64_t w = blockIdx.y; w < wt; w += gridDim.y) {
    const bool cases = w >= w0;
    const int64_t base = 32 * (cases ? w - w0 : w);
    const int64_t n_class = cases ? n1 : n0;
    const int32_t* pc = perm + (cases ? n0 : 0);
    uint32_t g0 = 0, g1 = 0;
    if (m < n_snps) {
      const int64_t lim = n_class - base < 32 ? n_class - base : 32;
      for (int64_t b = 0; b < lim; b++) {
        const int64_t s = pc[base + b];
        const uint32_t g = geno[s * n_snps + m];
        g0 |= (uint32_t)(g == 0) << b;
        g1 |= (uint32_t)(g == 1) << b;
      }
    }
    planes[w * m_pad + m] = make_uint2(g0, g1);
  }
}

// The same encoding, 16 SNPs per thread, for matrices whose rows are whole 16-byte pieces
// (n_snps a multiple of 16): one 128-bit load per sample gives the thread all 16 genotypes.  Threads
// are numbered over (class word, group of 16 SNPs), groups fastest, so a warp reads up to 512
// consecutive bytes of a sample row per load and narrow matrices fill their warps too.  Eight samples
// are in flight at a time (100000 x 256 takes 26 us, 61 with one after the other).  Per
// 32-bit piece, __vcmpeq4 marks the bytes equal to 0 and to 1; bit b of a plane word is sample b of
// the class word, as in k_encode.  Groups past n_snps (up to m_pad) write zero planes.
__global__ void __launch_bounds__(128) k_encode16(const uint8_t* __restrict__ geno, const int32_t* __restrict__ perm,
                           uint2* __restrict__ planes, int64_t n_snps, int64_t m_pad, int64_t w0, int64_t w1,
                           int64_t n0, int64_t n1) {
  const int64_t groups = m_pad / 16, units = groups * (w0 + w1);
  for (int64_t unit = (int64_t)blockIdx.x * 128 + threadIdx.x; unit < units; unit += (int64_t)gridDim.x * 128) {
    const int64_t w = unit / groups, m0 = 16 * (unit - w * groups);
    const bool cases = w >= w0;
    const int64_t base = 32 * (cases ? w - w0 : w);
    const int64_t n_class = cases ? n1 : n0;
    const int32_t* pc = perm + (cases ? n0 : 0) + base;
    const int lim = (int)(n_class - base < 32 ? n_class - base : 32);
    uint32_t g0[16], g1[16];
#pragma unroll
    for (int q = 0; q < 16; q++) g0[q] = g1[q] = 0;
    if (m0 < n_snps) {
#pragma unroll 1
      for (int b0 = 0; b0 < 32; b0 += 8) {
        if (b0 >= lim) break;
        int64_t s[8];
        uint4 v[8];
#pragma unroll
        for (int b = 0; b < 8; b++) s[b] = __ldg(pc + (b0 + b < lim ? b0 + b : b0));
#pragma unroll
        for (int b = 0; b < 8; b++) v[b] = __ldg(reinterpret_cast<const uint4*>(geno + s[b] * n_snps + m0));
#pragma unroll
        for (int b = 0; b < 8; b++) {
          const uint32_t keep = b0 + b < lim ? 0xFFFFFFFFu : 0u;
          const uint32_t x[4] = {v[b].x, v[b].y, v[b].z, v[b].w};
#pragma unroll
          for (int h = 0; h < 4; h++) {
            const uint32_t z = __vcmpeq4(x[h], 0u) & keep, o = __vcmpeq4(x[h], 0x01010101u) & keep;
#pragma unroll
            for (int t = 0; t < 4; t++) {
              g0[4 * h + t] |= ((z >> (8 * t)) & 1u) << (b0 + b);
              g1[4 * h + t] |= ((o >> (8 * t)) & 1u) << (b0 + b);
            }
          }
        }
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(planes + w * m_pad + m0);
#pragma unroll
    for (int q = 0; q < 8; q++) dst[q] = make_uint4(g0[2 * q], g1[2 * q], g0[2 * q + 1], g1[2 * q + 1]);
  }
}

// singles[c][m][g] = popcount over class c's words of plane g of SNP m.  A block counts 32 SNPs
// (lanes, 256-byte rows) of one class, its 32 warps every 32nd word each: with one thread per SNP
// and class pair 100000 samples x 256 SNPs took 527 us, a chain of loads.
__global__ void __launch_bounds__(1024) k_singles(const uint2* __restrict__ planes, uint32_t* __restrict__ singles,
                                                  int64_t m_pad, int64_t w0, int64_t w1) {
  __shared__ uint2 s_cnt[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = (int)blockIdx.y;
  const int64_t m = 32 * (int64_t)blockIdx.x + lane;  // m_pad is a multiple of 32
  const int64_t we = c ? w0 + w1 : w0;
  uint32_t g0 = 0, g1 = 0;
#pragma unroll 4
  for (int64_t w = (c ? w0 : 0) + warp; w < we; w += 32) {
    const uint2 v = __ldg(planes + w * m_pad + m);
    g0 += __popc(v.x);
    g1 += __popc(v.y);
  }
  s_cnt[warp][lane] = make_uint2(g0, g1);
  __syncthreads();
  if (warp == 0) {
    uint2 t = make_uint2(0, 0);
#pragma unroll
    for (int x = 0; x < 32; x++) {
      t.x += s_cnt[x][lane].x;
      t.y += s_cnt[x][lane].y;
    }
    reinterpret_cast<uint2*>(singles)[c * m_pad + m] = t;
  }
}

// pairs[c][tri(x,y)] = (n(0,0), n(0,1), n(1,0), n(1,1)) of SNPs x < y in class c.
// Block (x, y-strip of 256); the x word is a broadcast load, y words are coalesced.
__global__ void k_pairs(const uint2* __restrict__ planes, uint4* __restrict__ pairs, int64_t m_pad, int64_t w0,
                        int64_t w1) {
  const int64_t x = blockIdx.x;
  const int64_t y = (int64_t)blockIdx.y * blockDim.x + threadIdx.x;
  if ((int64_t)blockIdx.y * blockDim.x + blockDim.x <= x + 1) return;  // whole strip at or below the diagonal
  if (y <= x || y >= m_pad) return;
  const int64_t tri = tri_size(m_pad);
  const int64_t off = tri_offset(m_pad, x, y);
  for (int c = 0; c < 2; c++) {
    const int64_t wb = c ? w0 : 0, we = c ? w0 + w1 : w0;
    uint32_t n00 = 0, n01 = 0, n10 = 0, n11 = 0;
    for (int64_t w = wb; w < we; w++) {
      const uint2 a = planes[w * m_pad + x];
      const uint2 b = planes[w * m_pad + y];
      n00 += __popc(a.x & b.x);
      n01 += __popc(a.x & b.y);
      n10 += __popc(a.y & b.x);
      n11 += __popc(a.y & b.y);
    }
    pairs[c * tri + off] = make_uint4(n00, n01, n10, n11);
  }
}

cudaError_t launch_encode(const DevDataset& d, cudaStream_t stream) {
  const int64_t wt = d.w0 + d.w1;
  if (wt == 0 || d.m_pad == 0) return cudaSuccess;
  // 16 SNPs per thread from 16384 threads on, where both take about 18 us (8192 x 1024); below that
  // there are too few threads to hide the loads (2048 x 128: 18 us against 8).
  const bool vec = d.m_pad / 16 * wt >= 16384 && d.n_snps % 16 == 0 && ((uintptr_t)d.geno % 16) == 0 && ((uintptr_t)d.planes % 16) == 0;
  if (vec) {  // 16 SNPs per thread
    const int64_t blocks = (d.m_pad / 16 * wt + 127) / 128;
    k_encode16<<<(unsigned)(blocks < (1 << 20) ? blocks : (1 << 20)), 128, 0, stream>>>(d.geno, d.perm, d.planes, d.n_snps, d.m_pad, d.w0, d.w1, d.n_controls,
                                         d.n_cases);
  } else {
    dim3 grid((unsigned)((d.m_pad + 255) / 256), (unsigned)(wt < 65535 ? wt : 65535));
    k_encode<<<grid, 256, 0, stream>>>(d.geno, d.perm, d.planes, d.n_snps, d.m_pad, d.w0, d.w1, d.n_controls,
                                      d.n_cases);
  }
  return cudaGetLastError();
}

cudaError_t launch_counts(const DevDataset& d, cudaStream_t stream, bool pairs) {
  if (d.m_pad == 0) return cudaSuccess;
  k_singles<<<dim3((unsigned)(d.m_pad / 32), 2), 1024, 0, stream>>>(d.planes, d.singles, d.m_pad, d.w0, d.w1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (d.m_pad < 2 || !pairs) return cudaSuccess;
  dim3 grid((unsigned)d.m_pad, (unsigned)((d.m_pad + 255) / 256));
  k_pairs<<<grid, 256, 0, stream>>>(d.planes, d.pairs, d.m_pad, d.w0, d.w1);
  return cudaGetLastError();
}

}  // namespace epik2
