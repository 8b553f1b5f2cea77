// st_noadmix.cu -- the no-admixture Q update (NOADMIX=1): every individual
// comes from one population (src/Updates/UpdateQ.c:310-383 UpdateQNoAdmix).
//
// For individual i and population k the log likelihood of all its allele
// copies, ll_ik = sum_l sum_copy log P[l][k][allele], is accumulated in FP64
// from the stored log P.  (The reference keeps a running product rescaled
// below 1e-100; the two agree to rounding.)  Thread = individual, CTAs split
// the loci into chunks whose partial sums go to napart[chunk][i][k]; the
// pick kernel adds the chunks in order, forms exp(ll_ik - max_k ll_ik) and
// picks population k with the reference's PickAnOption rule (the first k
// with u * sum <= cumulative sum, src/mymath.c:80-100), u = rand()/2^31 from
// the Philox word at (i, 0) of stream kSNoAdmix.  Q_i becomes one-hot.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "st_device.cuh"
#include "st_kernels.h"

namespace st {
namespace {

constexpr int kNaBlock = 256;
constexpr int kNaPairs = 8;     // locus pairs per shared-memory stage (2-bit layout)

// 2-bit layout.  The pass was bound by its FP32-to-FP64 conversions (a quarter of
// the XU pipe's rate each: 2 K per genotype) and by one locus' loads at a time
// (519 us at N=2500, L=20,000, K=4).  The log probabilities of a pair of loci's 16
// genotype classes are formed once per CTA in shared memory, so a thread adds K
// doubles per two genotypes.  A class with a missing genotype holds the other
// locus' terms alone.
template <int KC>
__global__ void __launch_bounds__(kNaBlock)
noadmix_ll_b2g_kernel(const ChainDev* __restrict__ chp) {
  constexpr int kP = KC <= 16 ? kNaPairs : kNaPairs / 2;   // 16 KB of table at most
  __shared__ double2 tab[kP][KC / 2][16];   // class-minor: 8 classes span the banks
  __shared__ uint32_t sW[2 * kP][kNaBlock / 16];
  const ChainDev& ch = *chp;
  const int N = ch.N, L = ch.L, K = ch.K, A = ch.A, wpr = ch.wpr;
  const int i = blockIdx.x * kNaBlock + threadIdx.x;
  const bool active = i < N && !(ch.usepopinfo && ch.popflags[i]);   // flagged: migrant model
  double ll[KC];
#pragma unroll
  for (int k = 0; k < KC; k++) ll[k] = 0.0;
  const int l0 = blockIdx.y * ch.na_lchunk_len;
  const int l1 = min(L, l0 + ch.na_lchunk_len);
  const int wcol0 = (blockIdx.x * kNaBlock) >> 4, ncol = min(kNaBlock / 16, wpr - wcol0);
  const int sh = 2 * (threadIdx.x & 15), col = threadIdx.x >> 4;
  for (int lb = l0; lb < l1; lb += 2 * kP) {
    __syncthreads();
    for (int idx = threadIdx.x; idx < kP * 16 * KC; idx += kNaBlock) {
      const int e = idx & 1, c = (idx >> 1) & 15, k = 2 * ((idx >> 5) % (KC / 2)) + e;
      const int p = idx / (16 * KC);
      double v = 0.0;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int l = lb + 2 * p + h;
        const uint32_t g = (uint32_t)(c >> (2 * h)) & 3u;
        if (l < l1 && k < K && g != 3u) {
          const float* lp = ch.logP + ((size_t)l * K + k) * A;
          v += (double)lp[A > 1 ? g >> 1 : 0] + (double)lp[A > 1 ? (g | (g >> 1)) & 1u : 0];
        }
      }
      reinterpret_cast<double*>(tab)[idx] = v;
    }
    for (int idx = threadIdx.x; idx < 2 * kP * (kNaBlock / 16); idx += kNaBlock) {
      const int j = idx / (kNaBlock / 16), c = idx % (kNaBlock / 16);
      sW[j][c] = lb + j < l1 && c < ncol ? __ldg(ch.g2 + (size_t)(lb + j) * wpr + wcol0 + c)
                                         : 0xFFFFFFFFu;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < kP; p++) {
      const uint32_t c = ((sW[2 * p][col] >> sh) & 3u) | (((sW[2 * p + 1][col] >> sh) & 3u) << 2);
#pragma unroll
      for (int k = 0; k < KC; k += 2) {
        const double2 v = tab[p][k / 2][c];
        ll[k] += v.x;
        ll[k + 1] += v.y;
      }
    }
  }
  if (!active) return;
  double* out = ch.napart + ((size_t)blockIdx.y * N + i) * K;
#pragma unroll
  for (int k = 0; k < KC; k++)
    if (k < K) out[k] = ll[k];
}

// One byte per copy, any allele count.
template <int KC>
__global__ void __launch_bounds__(kNaBlock) noadmix_ll_u8_kernel(const ChainDev* __restrict__ chp) {
  const ChainDev& ch = *chp;
  const int N = ch.N, L = ch.L, K = ch.K, A = ch.A;
  const int i = blockIdx.x * kNaBlock + threadIdx.x;
  if (i >= N || (ch.usepopinfo && ch.popflags[i])) return;   // flagged: migrant model
  double ll[KC];
#pragma unroll
  for (int k = 0; k < KC; k++) ll[k] = 0.0;
  const int l0 = blockIdx.y * ch.na_lchunk_len;
  const int l1 = min(L, l0 + ch.na_lchunk_len);
  for (int l = l0; l < l1; l++) {
    const uint8_t b0 = __ldg(ch.g8 + ((size_t)l * N + i) * 2);
    const uint8_t b1 = __ldg(ch.g8 + ((size_t)l * N + i) * 2 + 1);
    const int a0 = b0 == kG8Missing ? -1 : b0, a1 = b1 == kG8Missing ? -1 : b1;
    const float* lp = ch.logP + (size_t)l * K * A;
#pragma unroll
    for (int k = 0; k < KC; k++) {
      if (k >= K) break;
      double v = 0.0;
      if (a0 >= 0) v += (double)__ldg(lp + k * A + a0);
      if (a1 >= 0) v += (double)__ldg(lp + k * A + a1);
      ll[k] += v;
    }
  }
  double* out = ch.napart + ((size_t)blockIdx.y * N + i) * K;
#pragma unroll
  for (int k = 0; k < KC; k++)
    if (k < K) out[k] = ll[k];
}

// G lanes per individual (power of two >= K), lane k = population k: the chunks'
// sums are loaded side by side instead of K x chunks loads behind one another in
// one thread (38 us at N=2500, 60 chunks, K=4).
__global__ void __launch_bounds__(kNaBlock) noadmix_pick_kernel(const ChainDev* __restrict__ chp,
                                                                int G) {
  const ChainDev& ch = *chp;
  const int N = ch.N, K = ch.K;
  const int i = (blockIdx.x * kNaBlock + threadIdx.x) / G, k = threadIdx.x % G;
  const bool active = i < N && !(ch.usepopinfo && ch.popflags[i < N ? i : 0]);
  const bool mine = active && k < K;
  // LOCPRIOR: the product starts at gamma of the individual's location
  // (src/Updates/UpdateQ.c:339-345)
  double s = mine && ch.locprior ? log(ch.locp[1 + (size_t)K * (ch.myloc[i] + 1) + k]) : 0.0;
  if (mine) {
    const double* part = ch.napart + (size_t)i * K + k;
    const size_t stride = (size_t)N * K;
#pragma unroll 8
    for (int c = 0; c < ch.na_lchunks; c++) s += part[c * stride];
  }
  // the largest over the populations, as a loop from population 0 that replaces on
  // greater (NaN never replaces; a NaN at population 0 stays)
  const int base = (threadIdx.x & 31) & ~(G - 1);
  double mx = __shfl_sync(0xffffffffu, s, base);
  for (int q = 1; q < K; q++) {
    const double o = __shfl_sync(0xffffffffu, s, base + q);
    if (o > mx) mx = o;
  }
  const double p = mine ? exp(s - mx) : 0.0;
  double sum = 0.0;
  for (int q = 0; q < K; q++) sum += __shfl_sync(0xffffffffu, p, base + q);
  const U4 w = philox_s((uint32_t)i, 0u, (uint32_t)*ch.rep, kSNoAdmix, ch.key);
  const double r = (double)(w.x >> 1) / 2147483648.0 * sum;
  double cum = 0.0;
  int pick = -1;   // the first population with r <= cum, the last one if none
  for (int q = 0; q < K; q++) {
    cum += __shfl_sync(0xffffffffu, p, base + q);
    if (pick < 0 && r <= cum) pick = q;
  }
  if (pick < 0) pick = K - 1;
  if (mine) {
    ch.Q[(size_t)i * K + k] = k == pick ? 1.0f : 0.0f;
    ch.logQ[(size_t)i * K + k] = k == pick ? 0.0f : -INFINITY;
  }
}

}  // namespace

void noadmix_plan(int N, int L, int* lchunks, int* lchunk_len) {
  const int tiles = (N + kNaBlock - 1) / kNaBlock;
  int ch = (148 * 4 + tiles - 1) / tiles;
  if (ch < 1) ch = 1;
  int len = (L + ch - 1) / ch;
  if (len < 64) len = 64;
  *lchunk_len = len;
  *lchunks = (L + len - 1) / len;
}

cudaError_t launch_noadmix(const ChainDev& h, const ChainDev* d_chain, cudaStream_t s) {
  const dim3 g((h.N + kNaBlock - 1) / kNaBlock, h.na_lchunks);
  if (h.layout == kLayoutB2G) {
    if (h.K <= 2) noadmix_ll_b2g_kernel<2><<<g, kNaBlock, 0, s>>>(d_chain);
    else if (h.K <= 4) noadmix_ll_b2g_kernel<4><<<g, kNaBlock, 0, s>>>(d_chain);
    else if (h.K <= 8) noadmix_ll_b2g_kernel<8><<<g, kNaBlock, 0, s>>>(d_chain);
    else if (h.K <= 16) noadmix_ll_b2g_kernel<16><<<g, kNaBlock, 0, s>>>(d_chain);
    else noadmix_ll_b2g_kernel<32><<<g, kNaBlock, 0, s>>>(d_chain);
  } else {
    if (h.K <= 8) noadmix_ll_u8_kernel<8><<<g, kNaBlock, 0, s>>>(d_chain);
    else if (h.K <= 16) noadmix_ll_u8_kernel<16><<<g, kNaBlock, 0, s>>>(d_chain);
    else noadmix_ll_u8_kernel<32><<<g, kNaBlock, 0, s>>>(d_chain);
  }
  int G = 1;
  while (G < h.K) G <<= 1;
  noadmix_pick_kernel<<<(unsigned)(((size_t)h.N * G + kNaBlock - 1) / kNaBlock), kNaBlock, 0, s>>>(
      d_chain, G);
  return cudaGetLastError();
}

}  // namespace st
