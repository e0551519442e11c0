// Host-side data sources and the K2 log-factorial table.
//
// Compiled with -ffp-contract=off so that every double expression below rounds
// exactly as written (the table must match the reference CPU path bit for bit).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "epik2_internal.h"

namespace epik2 {

// ln n! as the reference CPU path computes it (CPU/v4_popc_avx512.cpp:213-241):
//   n < 748 : t[0] = t[1] = 0, t[n] = (float)((double)t[n-1] + log(n))      (my_factorial)
//   n >= 748: (float)((n + 0.5) * log(n) - (n - 1) * log(exp(1)) + TABLE_ERROR) in double
// The reference's GPU kernels evaluate the Stirling tail in float with the SYCL device
// log/exp (GPU/v4.cpp:52-61); that arithmetic is not reproducible here, so the search
// follows the CPU path, which the reference's CPU programs all share.
void build_k2_lut_range(int64_t n_begin, int64_t n_end, float* out) {
  const double table_error = -0.0810;  // TABLE_ERROR, GPU/v4.cpp:16
  float t[kTableMaxSize];
  t[0] = 0.0f;
  t[1] = 0.0f;
  for (int n = 2; n < kTableMaxSize; n++) t[n] = (float)((double)t[n - 1] + std::log((double)n));
  const double log_e = std::log(std::exp(1.0));
  for (int64_t n = n_begin; n < n_end; n++) {
    if (n < kTableMaxSize) {
      out[n - n_begin] = t[n];
    } else {
      double a = ((double)n + 0.5) * std::log((double)n);
      double b = (double)(n - 1) * log_e;
      out[n - n_begin] = (float)(a - b + table_error);
    }
  }
}

void build_k2_lut(int64_t n_max, float* lut) { build_k2_lut_range(0, n_max + 1, lut); }

// Screening bound of the split search.  With A = a + 1/2, N = a + b + 1 for a cell of a controls
// and b cases, p in (0, 1), q = 1 - p, D = A - p N and d = D / N:
//   ln (a+b+1)! - ln a! - ln b!  =  -A ln p - (N - A) ln q + ln(N)/2 - ln(2 pi)/2 - N KL(p + d || p) + S
// with S about 1/(12 N) + 1/(24 A) + 1/(24 (N - A)) (Stirling at half-integers; S N is least, 0.2258, at
// a = b = 0).  KL / d^2 is c2 = 1 / (2 p q) at d = 0 and known at both ends, d = q and d = -p; its
// inverse is concave on either side, so it lies above the chords:
//   N KL(p + d || p)  <=  c2 D^2 / (N - t1 D - t2 |D|).
// The cell's bound takes both at M = N + 7/16 instead of N, which costs nothing:
//   -A ln p - (N - A) ln q + ln(M)/2 - ln(2 pi)/2 - c2 D^2 / (M - t1 D - t2 |D|),
// log2 M from M's FP32 bits (linear between powers of two, never above).  What M adds, at most 7/(32 N)
// to the logarithm and a share 7/(16 M) of the quotient, is less than S, what the chord leaves and what
// the linear logarithm leaves together: the least slack, times N, is 0.019 over every p = kp/64 with all
// a, b < 5000, and positive on grids, edges, the ridge a = p N and around powers of two up to 65535 (M = N
// + 1/2 fails at (0, 1) for p near 1/4).  A table of rare alleles is mostly empty cells, each of which
// loses S = 0.2258 at M = N: 1000 samples, minor-allele frequencies 0.001 to 0.005: 1.5 below the score
// instead of 5.6 (512 SNPs x 2000 samples, 5 % cases, frequencies 0.005 to 0.02: 1.97 -> 0.60 ms with
// it and without a term t1^2 / 3.5 beside c2 that the logarithm of N - t1 D costs).  Summed over the 27
// cells this bounds the K2 score from below, for any p: kp/64 next to the share of controls, which
// makes 64 D an integer.  base = the terms that are the same for every triplet, less a margin for
// rounding: of the reference's FP32 table and sums (about 5 ulp of ln n!, 0.1 for the table below 748)
// and of the FP32 evaluation of the bound.
ScreenConsts screen_constants(int64_t n0, int64_t n1) {
  const double n = (double)(n0 + n1);
  int kp = (int)std::min(63.0, std::max(1.0, std::floor(64.0 * ((double)n0 + 13.5) / (n + 27.0) + 0.5)));
  // Nearly even classes take p = 1/2, where t1 = 0 and a cell costs an operation less (1024 x 8192: 3.94
  // ms, with the operation 4.21).  At a distance x of the controls' share from 1/2 the bound loses about
  // 2 n t2 x^3, which at most 1 keeps no larger than the 1 to 2 it is below the score anyway.
  const double x = ((double)n0 + 13.5) / (n + 27.0) - 0.5;
  if (1.115 * n * std::fabs(x * x * x) <= 1.0) kp = 32;
  const double p = kp / 64.0, q = 1.0 - p;
  const double c2 = 1.0 / (2.0 * p * q);
  const double up = (1.0 + c2 * q * q / std::log(p)) / q;    // 1 - up d meets c2 d^2 / KL at d = q
  const double down = (1.0 + c2 * p * p / std::log(q)) / p;  // 1 - down |d| at d = -p
  const double t1 = (up - down) / 2.0, t2 = (up + down) / 2.0;
  ScreenConsts s{};
  s.coef = (uint32_t)(uint8_t)(64 - kp) | ((uint32_t)(uint8_t)(-kp) << 8);
  s.bias = 32 - kp;
  s.theta1 = (float)(t1 / 64.0);
  s.theta2 = (float)(t2 * 1.000001 / 64.0);
  s.c = (float)(c2 * 1.000001 / (64.0 * 64.0));
  const double margin = 0.3 + 1e-6 * std::lgamma(n + 2.0);
  s.margin = (float)margin;
  s.base = (float)(-((double)n0 + 13.5) * std::log(p) - ((double)n1 + 13.5) * std::log(q) -
                   13.5 * std::log(2.0 * 3.14159265358979323846) - margin);
  return s;
}

float screen_bound(int64_t n0, int64_t n1, const uint32_t* table) {
  const ScreenConsts s = screen_constants(n0, n1);
  const int ka = (int8_t)(s.coef & 0xFF), kb = (int8_t)(s.coef >> 8);
  float acc = 0.0f;
  uint32_t bits = 0;
  for (int x = 0; x < 27; x++) {
    const int a = (int)table[x], b = (int)table[27 + x];
    const float D = (float)(ka * a + kb * b + s.bias), M = (float)(a + b + 1) + kScreenShift;
    uint32_t m;
    std::memcpy(&m, &M, 4);
    bits += m;
    const float P = std::fma(std::fabs(D), -s.theta2, M);
    acc = std::fma(D * (1.0f / (s.theta1 == 0.0f ? P : std::fma(D, -s.theta1, P))), D, acc);
  }
  return std::fma(kScreenLog, (float)(bits - 27u * 0x3F800000u), -s.c * acc) + s.base;
}

// The same ln n! evaluated entirely in double (precision form's FP64 rescore): the table
// part accumulated in double, the Stirling tail in double and not rounded to float.
void build_k2_lut64(int64_t n_max, double* lut) {
  const double table_error = -0.0810;
  const double log_e = std::log(std::exp(1.0));
  double acc = 0.0;
  for (int64_t n = 0; n <= n_max; n++) {
    if (n < kTableMaxSize) {
      if (n >= 2) acc += std::log((double)n);
      lut[n] = acc;
    } else {
      lut[n] = ((double)n + 0.5) * std::log((double)n) - (double)(n - 1) * log_e + table_error;
    }
  }
}

// The reference's synthetic input (GPU/v4.cpp:81-110): srand(100); rand()%3 per
// genotype in sample-major order; exactly n/2 cases by rejection sampling.  An index
// equal to n (rand()==RAND_MAX) is dropped, which is where the reference's write lands
// outside its phenotype vector.
void generate_reference(int64_t n, int64_t m, uint8_t* geno, uint8_t* pheno) {
  srand(100);
  for (int64_t i = 0; i < n; i++)
    for (int64_t j = 0; j < m; j++) geno[i * m + j] = (uint8_t)(rand() % 3);
  std::vector<uint8_t> b((size_t)n + 1, 0);
  for (int64_t i = 0; i < n / 2; i++) {
    int index = (int)(n * ((double)rand() / (RAND_MAX)));
    while (b[(size_t)index] == 1) index = (int)(n * ((double)rand() / (RAND_MAX)));
    b[(size_t)index] = 1;
  }
  for (int64_t i = 0; i < n; i++) pheno[i] = b[(size_t)i];
}

// Seeded Hardy-Weinberg matrix with planted triplets (benchmark workloads).
//   p_m = lo + (hi-lo)*u, then per sample, per SNP: g = 0 if u < q^2, 1 if u < q^2+2pq,
//   else 2 (q = 1-p).  u = (x >> 11) * 2^-53 from std::mt19937_64(seed).
//   Exactly n_cases cases: risk r_s = the largest effect among planted triplets whose
//   three SNPs all carry >= 1 minor allele, else r0 so that the risks sum to n_cases;
//   cases are the n_cases largest Efraimidis-Spirakis keys log(u')/w, w = r/(1-r),
//   u' = ((x >> 11) + 1) * 2^-53, ties to the lower sample index.
void generate_hwe(uint64_t seed, int64_t n, int64_t m, int64_t n_cases, double maf_lo, double maf_hi,
                  int n_planted, const int64_t* planted, const double* effects, uint8_t* geno, uint8_t* pheno) {
  std::mt19937_64 rng(seed);
  const double inv53 = 1.0 / 9007199254740992.0;
  auto u01 = [&]() { return (double)(rng() >> 11) * inv53; };
  std::vector<double> p((size_t)std::max<int64_t>(m, 1));
  for (int64_t j = 0; j < m; j++) p[(size_t)j] = maf_lo + (maf_hi - maf_lo) * u01();
  for (int64_t s = 0; s < n; s++) {
    uint8_t* row = geno + s * m;
    for (int64_t j = 0; j < m; j++) {
      double u = u01();
      double q = 1.0 - p[(size_t)j];
      double t0 = q * q;
      double t1 = t0 + 2.0 * p[(size_t)j] * q;
      row[j] = (uint8_t)(u < t0 ? 0 : (u < t1 ? 1 : 2));
    }
  }
  std::vector<double> risk((size_t)std::max<int64_t>(n, 1), -1.0);
  int64_t n_car = 0;
  double car_sum = 0.0;
  for (int64_t s = 0; s < n; s++) {
    double best = -1.0;
    for (int t = 0; t < n_planted; t++) {
      const int64_t* tr = planted + 3 * t;
      const uint8_t* row = geno + s * m;
      if (row[tr[0]] >= 1 && row[tr[1]] >= 1 && row[tr[2]] >= 1 && effects[t] > best) best = effects[t];
    }
    risk[(size_t)s] = best;
    if (best >= 0.0) {
      n_car++;
      car_sum += best;
    }
  }
  double r0 = (n > n_car) ? ((double)n_cases - car_sum) / (double)(n - n_car) : 0.5;
  r0 = std::min(std::max(r0, 1e-9), 1.0 - 1e-9);
  std::vector<std::pair<double, int64_t>> keys((size_t)n);
  for (int64_t s = 0; s < n; s++) {
    double rs = risk[(size_t)s] >= 0.0 ? risk[(size_t)s] : r0;
    double w = rs / (1.0 - rs);
    double u = ((double)(rng() >> 11) + 1.0) * inv53;
    keys[(size_t)s] = {std::log(u) / w, s};
  }
  std::sort(keys.begin(), keys.end(), [](const std::pair<double, int64_t>& a, const std::pair<double, int64_t>& b) {
    if (a.first != b.first) return a.first > b.first;
    return a.second < b.second;
  });
  for (int64_t s = 0; s < n; s++) pheno[s] = 0;
  for (int64_t s = 0; s < n_cases && s < n; s++) pheno[keys[(size_t)s].second] = 1;
}

}  // namespace epik2
