// st_zmetro.cuh -- the Metropolis pass on biallelic 2-bit data: per individual the log
// ratio sum_l log(T.P[a0] T.P[a1]) - log(Q.P[a0] Q.P[a1]) (CalcLike.c:281-345), as
// partials ldpart[group][i] in FP64.
//
// Lane = locus, a warp walks the chunk's individuals 16 per genotype word.  Q and T of
// a row lie side by side in shared memory, (Q_k, T_k) a packed pair that every lane
// reads at once, and multiply the lane's P[l][k][0] and P[l][k][1]: both alleles' sums
// (Q.P, T.P) come from 2 K packed multiply-adds, and a genotype selects two of them (4
// selects; selecting P per copy and population took 2 K, and Q and T were read as
// separate duplicated rows).  P stays in registers as duplicated pairs up to K class
// 12, where it fits; above, it is read from the lane's shared-memory column.
// A genotype whose products near FP32's lower end takes FP64 logarithms, looked for
// once per four genotypes.  The terms, their order of summation (transposed butterfly
// over the warp's loci, FP32 over the CTA's locus blocks, FP64 over warps) and so the
// ratios' bits depend on the locus blocks R of the tile alone.
#pragma once
#include "st_device.cuh"
#include "st_kernels.h"

namespace st {
namespace zmetro {

constexpr float kTiny = 1e-30f;

__host__ __device__ constexpr bool regp(int kt) { return kt <= 12; }
__host__ __device__ constexpr int width(int kt) { return kt <= 12 ? 8 : 2; }   // warps
__host__ __device__ constexpr int ctas(int kt) { return kt <= 5 ? 3 : kt <= 12 ? 2 : 8; }   // per SM

struct Layout { int qt, x, ld, total; };

__host__ __device__ inline Layout layout(int kt, int T) {
  Layout z;
  const int w = width(kt);
  int o = 0;
  z.qt = o; o += T * ((kt + 1) & ~1) * 8;
  z.x = o;  if (!regp(kt)) o += kt * 32 * w * 8;
  z.ld = o; o += T * w * 4;
  z.total = (o + 15) & ~15;
  return z;
}

template <int KT>
__global__ void __launch_bounds__(32 * width(KT), ctas(KT))
zmetro_kernel(ChainDev* __restrict__ chains, const int* __restrict__ prefix, int nchains, int flags) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int W = width(KT), NTH = 32 * W, KT2 = (KT + 1) & ~1;
  constexpr int NP = regp(KT) ? KT : 1;
  int c, tile;
  if (flags & kZfInterleave) {   // chains of one data set and tile, interleaved
    c = (int)blockIdx.x % nchains;
    tile = (int)blockIdx.x / nchains;
  } else {
    c = find_chain(prefix, nchains, blockIdx.x);
    tile = blockIdx.x - prefix[c];
  }
  ChainDev& ch = chains[c];
  const int T = ch.tileT, R = ch.tileR;
  const int ichunk = tile % ch.nchunks, grp = tile / ch.nchunks;
  const int N = ch.N, L = ch.L, A = ch.A, K = ch.K;
  const int i0 = ichunk * T;
  const int nT = min(N, i0 + T) - i0;
  const int nT16 = (nT + 15) & ~15;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Layout lay = layout(KT, T);
  float2* sQT = reinterpret_cast<float2*>(smem + lay.qt);
  float2* sX = reinterpret_cast<float2*>(smem + lay.x) + threadIdx.x;
  float* sLD = reinterpret_cast<float*>(smem + lay.ld);   // [W][nT16]
  for (int ii = threadIdx.x; ii < nT16; ii += NTH) {   // thread = row
    const float* q = ch.Q + (size_t)(i0 + ii) * K;
    const float* t = ch.TestQ + (size_t)(i0 + ii) * K;
#pragma unroll
    for (int k = 0; k < KT2; k++) {
      // a row beyond the chunk reads (1, 0, ...): sums away from zero, never stored
      const float pad = k == 0 ? 1.0f : 0.0f;
      sQT[ii * KT2 + k] = ii < nT ? (k < K ? make_float2(q[k], t[k]) : make_float2(0.0f, 0.0f))
                                  : make_float2(pad, pad);
    }
  }
  for (int idx = threadIdx.x; idx < nT16 * W; idx += NTH) sLD[idx] = 0.0f;
  __syncthreads();

  float* myLD = sLD + warp * nT16;
  for (int rb = 0; rb < R; rb++) {
    const int lbase = ((grp * R + rb) * W + warp) * 32;
    if (lbase >= L) break;  // warp-uniform
    const int l = lbase + lane;
    const bool valid = l < L;
    float2 p0[NP], p1[NP];   // (P, P) of both alleles
    {
      const float* P = ch.P + (size_t)(valid ? l : 0) * K * A;
#pragma unroll
      for (int k = 0; k < KT; k++) {
        // a lane beyond the last locus reads P = 1 and missing genotypes
        const float a = k < K ? (valid ? P[(size_t)k * A] : 1.0f) : 0.0f;
        const float b = k < K ? (valid ? (A > 1 ? P[(size_t)k * A + 1] : 0.0f) : 1.0f) : 0.0f;
        if constexpr (regp(KT)) {
          p0[k < NP ? k : 0] = make_float2(a, a);
          p1[k < NP ? k : 0] = make_float2(b, b);
        } else {
          sX[k * NTH] = make_float2(a, b);
        }
      }
    }
    const uint32_t* grow = ch.g2 + (size_t)(valid ? l : 0) * ch.wpr + (i0 >> 4);
    for (int wi = 0; wi < (nT16 >> 4); wi++) {
      const uint32_t word = valid ? __ldg(grow + wi) : 0xFFFFFFFFu;
      const uint32_t any = word | (word >> 1), mis = word & (word >> 1);
      float tr[16];
#pragma unroll
      for (int j0 = 0; j0 < 16; j0 += 4) {
        float2 S0[4], S1[4];   // per copy: (Q.P, T.P)
        float low = 1.0f;
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int j = j0 + e;
          const float4* row = reinterpret_cast<const float4*>(sQT + ((wi << 4) + j) * KT2);
          float2 C0 = make_float2(0.0f, 0.0f), C1 = C0;
#pragma unroll
          for (int k = 0; k < KT; k += 2) {
            const float4 v = row[k >> 1];
#pragma unroll
            for (int u = 0; u < 2; u++) {
              if (k + u < KT) {
                const float2 qt = u ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
                float2 x0, x1;
                if constexpr (regp(KT)) {
                  x0 = p0[k + u < NP ? k + u : 0];
                  x1 = p1[k + u < NP ? k + u : 0];
                } else {
                  const float2 x = sX[(k + u) * NTH];
                  x0 = make_float2(x.x, x.x);
                  x1 = make_float2(x.y, x.y);
                }
                C0 = k + u == 0 ? mul2_rn(qt, x0) : fma2_rn(qt, x0, C0);
                C1 = k + u == 0 ? mul2_rn(qt, x1) : fma2_rn(qt, x1, C1);
              }
            }
          }
          const bool h = (word >> (2 * j + 1)) & 1u, n = (any >> (2 * j)) & 1u;
          S0[e] = make_float2(h ? C1.x : C0.x, h ? C1.y : C0.y);
          S1[e] = make_float2(n ? C1.x : C0.x, n ? C1.y : C0.y);
          const float tp = S0[e].y * S1[e].y, tm = S0[e].x * S1[e].x;
          low = fminf(low, fminf(tp, tm));
          tr[j] = (mis >> (2 * j)) & 1u ? 0.0f : __logf(tp) - __logf(tm);
        }
        if (__any_sync(0xffffffffu, !(low > kTiny))) {
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int j = j0 + e;
            const float tp = S0[e].y * S1[e].y, tm = S0[e].x * S1[e].x;
            if (!((mis >> (2 * j)) & 1u) && !(tp > kTiny && tm > kTiny))
              tr[j] = (float)(log((double)S0[e].y) + log((double)S1[e].y) -
                              log((double)S0[e].x) - log((double)S1[e].x));
          }
        }
      }
      // the word's 16 row sums over the warp's 32 loci by a transposed butterfly: at
      // the exchange across lane bit b a lane keeps the half of its rows picked by its
      // own bit b and adds its partner's partial for the same rows; after lane bits
      // 4..1 lanes 2r, 2r+1 hold row r.  31 exchanges per word instead of 5 per row.
      float v8[8], v4[4], v2[2];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const bool hi = lane & 16;
        v8[i] = (hi ? tr[i + 8] : tr[i]) + __shfl_xor_sync(0xffffffffu, hi ? tr[i] : tr[i + 8], 16);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool hi = lane & 8;
        v4[i] = (hi ? v8[i + 4] : v8[i]) + __shfl_xor_sync(0xffffffffu, hi ? v8[i] : v8[i + 4], 8);
      }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const bool hi = lane & 4;
        v2[i] = (hi ? v4[i + 2] : v4[i]) + __shfl_xor_sync(0xffffffffu, hi ? v4[i] : v4[i + 2], 4);
      }
      const bool hi = lane & 2;
      float v = (hi ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, hi ? v2[0] : v2[1], 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      if (!(lane & 1)) myLD[(wi << 4) + (lane >> 1)] += v;   // this warp's rows only
    }
    __syncwarp();
  }
  __syncthreads();
  // the warps' partials in warp order: a fixed summation order
  double* dst = ch.ldpart + (size_t)grp * N + i0;
  for (int idx = threadIdx.x; idx < nT; idx += NTH) {
    double v = 0.0;
    for (int w = 0; w < W; w++) v += (double)sLD[w * nT16 + idx];
    dst[idx] = v;
  }
}

template <int KT>
cudaError_t launch_zmetro_k(const LaunchSet& ls, int flags, size_t smem) {
  auto fn = zmetro_kernel<KT>;
  if (const cudaError_t e = allow_dynamic_smem(fn, smem)) return e;
  fn<<<ls.total_ctas, 32 * width(KT), smem, ls.stream>>>(ls.chains, ls.prefix, ls.nchains, flags);
  return cudaGetLastError();
}

}  // namespace zmetro
}  // namespace st
