// st_zcount.cuh -- the sweep's counting Z pass on biallelic 2-bit data: draws
// every copy's population, adds the allele and ancestry counts, and reduces
// ln P(D) when the sweep collects.  Same draws, counts and ln P(D) terms as the
// general biallelic pass (st_zpass_fast.cuh), which serves the chains that store
// Z or count flagged individuals only.
//
// A draw is z = #{k : C_k < r} over the K - 1 thresholds C_k (cumulative mixture
// weights), and the C_k do not decrease, so a copy is told by the sign bits of
// C_k - r alone and z itself is never formed.  Every count follows from
//   cum_k = #{copies : C_k < r},   n_0 = copies - cum_0,  n_k = cum_{k-1} - cum_k,
// and cum_k is a sum of sign bits.  Four thresholds' sign bytes, replicated by
// PRMT, make one word of 0x00 / 0xFF bytes per copy; a sum of such words is
// 255 N (mod 2^32) for the word N of byte counts, so N = -sum * 0x01010101 as
// long as no byte's count exceeds 255.  The words are added in registers per
// locus (all copies, and allele 1's) and over the warp's 32 loci with
// redux.sync per individual.  A missing genotype draws no sign: its table class
// holds zeros, or its uniforms are masked to u = 0.
#pragma once
#include "st_device.cuh"
#include "st_kernels.h"
#include "st_zpass_fast.cuh"

namespace st {
namespace zcount {

using zfast::block_sum_d;
using zfast::finish_like;
using zfast::kLikeFastMin;

constexpr int kW = 8;              // warps per CTA
constexpr int kNT = 32 * kW;       // threads
constexpr int kFlushWords = 7;     // 7 x 16 genotypes x 2 copies = 224 <= 255
constexpr int kRedStride = 36;     // words per row of the reduction buffer (16-byte
                                   // aligned, rows 4 banks apart)

// Per K class: CTAs per SM, populations whose P pair stays in registers (two
// selects each instead of one 8-byte table load), table classes (4: a zero class
// for missing genotypes; 3: their uniforms are masked), unrolled parts of a word,
// and how a row's words are summed over the lanes (redux.sync, or through shared
// memory where one word per row leaves room).  From timing each class at N=2000,
// L=50,000 (SM cycles x 4 per 32 genotypes, ln P(D) on): K=5 102 (redux 105,
// 3 classes 102.5; 2 CTAs 113, 4 CTAs 108), K=8 143 (2 registers 147, two parts
// 150, 2 CTAs 152), K=10 179 (4 registers 180, 3 CTAs 181, two parts 183,
// shared-memory sums 186), K=20 382 (6 registers and 1 CTA 417, 14 registers
// 391, four parts 392, shared-memory sums 528); taken before K <= 5 predicated its
// likelihood product and added the loci's sign bytes a pair of rows at a time, which
// made K=5 1.3 % faster.  Where the table of every population fits three CTAs, registers
// only add selects; above K=8 they make room for two CTAs.
__host__ __device__ constexpr int zc_ctas(int kt) { return kt <= 8 ? 3 : kt <= 24 ? 2 : 1; }
__host__ __device__ constexpr int zc_nreg(int kt) {
  return kt <= 8 ? 0 : kt <= 12 ? 2 : kt <= 24 ? kt / 2 : 16;
}
__host__ __device__ constexpr int zc_nsm(int kt) { return kt - zc_nreg(kt); }
__host__ __device__ constexpr int zc_classes(int kt) { return kt <= 5 ? 4 : 3; }
__host__ __device__ constexpr int zc_halves(int kt) { return kt <= 12 ? 1 : 2; }
__host__ __device__ constexpr bool zc_redux(int kt) { return kt > 5; }
__host__ __device__ constexpr int zc_words(int kt) { return (kt + 2) / 4; }   // ceil((kt-1)/4)
__host__ __device__ constexpr int zc_kq(int kt) { return (kt + 3) & ~3; }
__host__ __device__ constexpr int zc_xslots(int kt) {   // 8-byte slots of one locus' table
  return zc_nsm(kt) * zc_classes(kt) + (zc_classes(kt) == 3 ? 1 : 0);
}

// words of one warp's row-sum buffer
__host__ __device__ constexpr int zc_red_words(int kt) {
  return zc_words(kt) * (16 / zc_halves(kt)) * (zc_redux(kt) ? 1 : kRedStride);
}

struct ZcLayout {
  int x, q, wide, red, m, pres, total;
};

__host__ __device__ inline ZcLayout zc_layout(int kt, int T) {
  ZcLayout z;
  int o = 0;
  z.x = o;    o += zc_xslots(kt) * kNT * 8;
  z.q = o;    o += T * zc_kq(kt) * 4;
  z.wide = o; o += zc_words(kt) * 4 * kNT * 4;
  z.red = o;  o += kW * zc_red_words(kt) * 4;
  z.m = o;    o += T * zc_words(kt) * 2 * 4;
  z.pres = o; o += T * 4;
  z.total = (o + 15) & ~15;
  return z;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// (w & m) | bits of -1.0f, opaque to the optimiser: it would narrow Philox' last
// 32 x 32 -> 64-bit products to the 23 bits kept, in more instructions.
__device__ __forceinline__ float and_or(uint32_t w, uint32_t m) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(w), "r"(m), "r"(0xBF800000u));
  return __uint_as_float(d);
}

// Sign bytes of d[0..n-1] (n = 1..4): byte j is 0xFF where d[j] is negative.
// With n < 4 the upper bytes repeat the last sign and are never read.
template <int N>
__device__ __forceinline__ uint32_t sign_bytes(const uint32_t* d) {
  if constexpr (N == 1) return prmt(d[0], d[0], 0xBBBBu);
  if constexpr (N == 2) return prmt(d[0], d[1], 0xFFFBu);
  if constexpr (N == 3) return prmt(prmt(d[0], d[1], 0xFBFBu), d[2], 0xFF10u);
  if constexpr (N == 4)
    return prmt(prmt(d[0], d[1], 0xFBFBu), prmt(d[2], d[3], 0xFBFBu), 0x5410u);
  return 0u;
}

// ln P(D) terms of one lane's 16 genotypes of a word in FP64 with the
// reference's per-copy clamp (CalcLike.c:75-133), from the same FP32 mixture
// sums as the draw.  Taken only for words that hold a term below kLikeFastMin.
template <int KT>
__device__ __noinline__ double word_like_exact(uint32_t word, const float* q, const float* P, int K,
                                               int A) {
  double s = 0.0;
  for (int gi = 0; gi < 16; gi++, q += zc_kq(KT)) {
    const uint32_t g = (word >> (2 * gi)) & 3u;
    if (g == 3u) continue;
    const int a0 = (int)(g >> 1), a1 = (int)((g | (g >> 1)) & 1u);
    float c0 = 0.0f, c1 = 0.0f;
    for (int k = 0; k < K; k++) {
      const float p0 = P[(size_t)k * A], p1 = A > 1 ? P[(size_t)k * A + 1] : 0.0f;
      const float x0 = a0 ? p1 : p0, x1 = a1 ? p1 : p0;
      c0 = k == 0 ? __fmul_rn(q[k], x0) : __fmaf_rn(q[k], x0, c0);
      c1 = k == 0 ? __fmul_rn(q[k], x1) : __fmaf_rn(q[k], x1, c1);
    }
    s += log(fmax((double)c0, 1e-50)) + log(fmax((double)c1, 1e-50));
  }
  return s;
}

// What a lane keeps of one of its loci through a chunk.
template <int KT>
struct Locus {
  static constexpr int NR = zc_nreg(KT) > 0 ? zc_nreg(KT) : 1;
  static constexpr int NWD = zc_words(KT) > 0 ? zc_words(KT) : 1;
  float p0[NR], p1[NR];          // P[l][k][0..1] of the populations kept in registers
  uint32_t all[NWD], one[NWD];   // sign sums: all copies, allele 1's copies
  int tot, tot1;                 // copies present, of allele 1
  const uint32_t* grow;          // genotype words of the chunk, or null beyond the last locus
  const float* Prow;
};

// DRAW: draws and counts (the sweep's pass); without it ln P(D) of the state only.
template <int KT, bool LIKE, bool DRAW>
__device__ __forceinline__ void zcount_words(int nwords, uint32_t pair0, const PhiloxRun& prun,
                                             const unsigned char* xtab, const float* sQ, int* sWide,
                                             uint32_t* sRed, int* sM, int* sPres, Locus<KT>& lo,
                                             double& like_acc, double magic, int K, int A) {
  constexpr int NT = DRAW ? KT - 1 : 0;
  constexpr int NW = DRAW ? zc_words(KT) : 0, NS = zc_nsm(KT), KQ = zc_kq(KT);
  constexpr int CSTR = kNT * 8, KSTR = CSTR * zc_classes(KT);
  constexpr bool kMask = zc_classes(KT) == 3;   // missing genotypes: u = 0 instead of zero P
  constexpr int kHalves = zc_halves(KT), kJN = 16 / kHalves;
  constexpr bool kRedux = zc_redux(KT);
  constexpr int kG = 32 / kJN;                  // lanes per row in the reduction
  const int lane = threadIdx.x & 31;
  const uint32_t t8 = threadIdx.x * 8;
  for (int w0 = 0; w0 < nwords; w0 += kFlushWords) {
    const int w1 = min(nwords, w0 + kFlushWords);
#pragma unroll
    for (int w = 0; w < NW; w++) lo.all[w] = lo.one[w] = 0u;
    for (int wi = w0; wi < w1; wi++) {
      const uint32_t word = lo.grow ? __ldg(lo.grow + wi) : 0xFFFFFFFFu;
      const uint32_t pw = prun.head ^ ((pair0 + (uint32_t)(wi << 3)) & 0xFFFFFFu);
      float wlike = 0.0f, wprod = 1.0f, wmin = 1.0f;
#pragma unroll 1
      for (int hb = 0; hb < kHalves; hb++) {
        const uint32_t hw = kHalves == 1 ? word : (word >> (2 * kJN * hb));
        const uint32_t hany = hw | (hw >> 1), hmiss = hw & (hw >> 1);
        const uint32_t phw = kHalves == 1 ? pw : (pw ^ (uint32_t)(hb * (kJN / 2)));
        const float* qrow = sQ + ((wi << 4) + hb * kJN) * KQ;
#pragma unroll
        for (int j = 0; j < kJN; j += 2) {
          U4 r4;
          uint32_t s_even[NW > 0 ? NW : 1];
          if (NT > 0) r4 = prun.block_r0(phw ^ (uint32_t)(j >> 1));
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int sh = 2 * (j + h);
            // class offset g * CSTR (2 KB) joined to the lane's column of the table
            const uint32_t off = (sh <= 11 ? ((hw << (11 - sh)) & 0x1800u)
                                           : ((hw >> (sh - 11)) & 0x1800u)) | t8;
            const unsigned char* xc = xtab + off;
            const bool any = (hany >> sh) & 1u, hi = (hw >> (sh + 1)) & 1u;
            const bool miss = (hmiss >> sh) & 1u;
            float2 C[KT];
#pragma unroll
            for (int k4 = 0; k4 < KQ; k4 += 4) {
              const float4 v = *reinterpret_cast<const float4*>(qrow + (j + h) * KQ + k4);
              const float qv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const int k = k4 + e;
                if (k < KT) {
                  float2 X;
                  if (k < NS) {
                    X = *reinterpret_cast<const float2*>(xc + k * KSTR);
                  } else {
                    const int r = k >= NS ? k - NS : 0;
                    X = make_float2(hi ? lo.p1[r] : lo.p0[r], any ? lo.p1[r] : lo.p0[r]);
                  }
                  const float2 qq = make_float2(qv[e], qv[e]);
                  C[k] = k == 0 ? mul2_rn(qq, X) : fma2_rn(qq, X, C[k > 0 ? k - 1 : 0]);
                }
              }
            }
            const float2 Tp = C[KT - 1];
            if constexpr (NT > 0) {
              // NR = RN(-u T), one fma of -(1 + u) (neg_one_plus_u23)
              const uint32_t um = kMask ? (miss ? 0u : 0x7FFFFFu) : 0x7FFFFFu;
              const float2 NM = make_float2(and_or(h ? r4.z : r4.x, um), and_or(h ? r4.w : r4.y, um));
              const float2 NR = fma2_rn(NM, Tp, Tp);
              uint32_t dx[NT], dy[NT];
#pragma unroll
              for (int k = 0; k < NT; k++) {
                const float2 D = add2_rn(C[k], NR);
                dx[k] = __float_as_uint(D.x);
                dy[k] = __float_as_uint(D.y);
              }
              uint32_t s[NW];
#pragma unroll
              for (int w = 0; w < NW; w++) {
                constexpr int kLast = NT % 4 == 0 ? 4 : NT % 4;
                uint32_t x, y;
                if (w < NW - 1) {
                  x = sign_bytes<4>(dx + 4 * w);
                  y = sign_bytes<4>(dy + 4 * w);
                } else {
                  x = sign_bytes<kLast>(dx + 4 * w);
                  y = sign_bytes<kLast>(dy + 4 * w);
                }
                s[w] = x + y;
                if (kRedux)
                  lo.all[w] += s[w];
                else if (h == 0)   // two genotypes' bytes in one three-operand addition
                  s_even[w] = s[w];
                else
                  lo.all[w] += s_even[w] + s[w];
                // 0/1 and 1/1: copy 1 carries allele 1; 1/1: copy 0 does too
                // (missing: x = y = 0).  As asm, the additions stay predicated
                // ones; otherwise they turn into masks of several operations.
                if (any) asm volatile("add.u32 %0, %0, %1;" : "+r"(lo.one[w]) : "r"(y));
                if (hi) asm volatile("add.u32 %0, %0, %1;" : "+r"(lo.one[w]) : "r"(x));
              }
              if constexpr (kRedux) {
#pragma unroll
                for (int w = 0; w < NW; w++) s[w] = __reduce_add_sync(0xffffffffu, s[w]);
                // every lane holds the sums and writes the same words
#pragma unroll
                for (int w = 0; w < NW; w++) sRed[(j + h) * NW + w] = s[w];
              } else {
#pragma unroll
                for (int w = 0; w < NW; w++) sRed[(w * kJN + j + h) * kRedStride + lane] = s[w];
              }
            }
            if (LIKE) {
              const float pr = Tp.x * Tp.y;
              if (((j + h) & 3) == 0)
                wprod = miss ? 1.0f : pr;
              else if (kRedux)
                wprod *= miss ? 1.0f : pr;
              else if (!miss)   // one predicated product; a select of 1 above K=5, where
                                // it measured the same or better
                asm volatile("mul.rn.f32 %0, %0, %1;" : "+f"(wprod) : "f"(pr));
              if (((j + h) & 3) == 3) {
                wmin = fminf(wmin, wprod);
                wlike += __logf(wprod);
              }
            }
          }
        }
        if constexpr (NT > 0) {
          // byte counts (<= 64) of the rows' sums over the warp's lanes, to 16-bit
          // fields of the CTA's rows
          __syncwarp();
          const int row0 = (wi << 4) + hb * kJN;
          if constexpr (kRedux) {
#pragma unroll
            for (int e = 0; e < (kJN * NW * 2 + 31) / 32; e++) {
              const int idx = lane + 32 * e, odd = idx & 1;   // (row, word, parity)
              if ((kJN * NW * 2) % 32 == 0 || idx < kJN * NW * 2) {
                const uint32_t n = sRed[idx >> 1] * 0xFEFEFEFFu;
                atomicAdd(&sM[row0 * NW * 2 + idx], (int)((odd ? n >> 8 : n) & 0x00FF00FFu));
              }
            }
          } else {
            const int row = lane / kG, part = lane % kG;
#pragma unroll
            for (int w = 0; w < NW; w++) {
              const uint4* src = reinterpret_cast<const uint4*>(
                  sRed + (w * kJN + row) * kRedStride + part * kJN);
              uint32_t v = 0;
#pragma unroll
              for (int e = 0; e < kJN / 4; e++) {
                const uint4 u = src[e];
                v += (u.x + u.y) + (u.z + u.w);
              }
#pragma unroll
              for (int o = 1; o < kG; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
              const uint32_t n = v * 0xFEFEFEFFu;
              if (part < 2)
                atomicAdd(&sM[((row0 + row) * NW + w) * 2 + part],
                          (int)((part ? n >> 8 : n) & 0x00FF00FFu));
            }
          }
          __syncwarp();
        }
      }
      if constexpr (DRAW) {
        // present loci of the word's 16 rows, and the locus' allele totals
        const uint32_t pres = ~(word & (word >> 1)) & 0x55555555u;
        const uint32_t h1 = (word >> 1) & ~word & 0x55555555u;                  // 1/1
        const uint32_t het = word & ~(word >> 1) & 0x55555555u;                 // 0/1
        lo.tot += __popc(pres);
        lo.tot1 += __popc(het | h1 | (h1 << 1));
        const uint32_t q0 = __reduce_add_sync(0xffffffffu, pres & 0x01010101u);
        const uint32_t q1 = __reduce_add_sync(0xffffffffu, (pres >> 2) & 0x01010101u);
        const uint32_t q2 = __reduce_add_sync(0xffffffffu, (pres >> 4) & 0x01010101u);
        const uint32_t q3 = __reduce_add_sync(0xffffffffu, (pres >> 6) & 0x01010101u);
        if (lane < 16) {   // row 4 b + j: byte b of q_j
          const uint32_t q = lane & 2 ? (lane & 1 ? q3 : q2) : (lane & 1 ? q1 : q0);
          atomicAdd(&sPres[(wi << 4) + lane], (int)((q >> (8 * (lane >> 2))) & 0xFFu));
        }
      }
      if (LIKE) {
        double wl = (double)wlike;
        if (__any_sync(0xffffffffu, !(wmin > kLikeFastMin))) {   // once per word, rare
          if (!(wmin > kLikeFastMin)) wl = word_like_exact<KT>(word, sQ + (wi << 4) * KQ, lo.Prow, K, A);
        }
        like_acc += __dsub_rn(__dadd_rn(wl, magic), magic);   // to the quantum
      }
    }
#pragma unroll
    for (int w = 0; w < NW; w++) {
      const uint32_t u = lo.all[w] * 0xFEFEFEFFu, v = lo.one[w] * 0xFEFEFEFFu;
      int* d = sWide + w * 4 * kNT;
      d[0] += (int)(u & 0x00FF00FFu);
      d[kNT] += (int)((u >> 8) & 0x00FF00FFu);
      d[2 * kNT] += (int)(v & 0x00FF00FFu);
      d[3 * kNT] += (int)((v >> 8) & 0x00FF00FFu);
    }
  }
}

template <int KT, bool DRAW, bool BEHIND>
__global__ void __launch_bounds__(kNT, zc_ctas(KT))
zcount_kernel(ChainDev* __restrict__ chains, const int* __restrict__ prefix, int nchains, int flags) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double sred[kW];
  constexpr int NW = zc_words(KT), NS = zc_nsm(KT), KQ = zc_kq(KT), CL = zc_classes(KT);
  int c, tile;
  if (flags & kZfInterleave) {   // chains of one data set and tile, interleaved
    c = (int)blockIdx.x % nchains;
    tile = (int)blockIdx.x / nchains;
  } else {
    c = find_chain(prefix, nchains, blockIdx.x);
    tile = blockIdx.x - prefix[c];
  }
  ChainDev& ch = chains[c];
  const int T = ch.ctT, R = ch.ctR;
  const int ichunk = tile % ch.ctchunks, grp = tile / ch.ctchunks;
  const int N = ch.N, L = ch.L, A = ch.A, K = ch.K;
  const int i0 = ichunk * T;
  const int nT = min(N, i0 + T) - i0;
  const int nT16 = (nT + 15) & ~15;  // whole words; padding genotypes are "missing"
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (BEHIND) after_previous_kernel();
  const int rep = *ch.rep;
  const bool collect = rep + 1 > ch.burnin;
  const bool want_like =
      !DRAW || (flags & kZfLikeAlways) || ((flags & kZfLikeIfCollect) && collect);

  const ZcLayout lay = zc_layout(KT, T);
  float2* sX = reinterpret_cast<float2*>(smem + lay.x);
  float* sQ = reinterpret_cast<float*>(smem + lay.q);
  int* sWide = reinterpret_cast<int*>(smem + lay.wide) + threadIdx.x;
  uint32_t* sRed = reinterpret_cast<uint32_t*>(smem + lay.red) +
                   warp * zc_red_words(KT);
  int* sM = reinterpret_cast<int*>(smem + lay.m);
  int* sPres = reinterpret_cast<int*>(smem + lay.pres);

  for (int ii = threadIdx.x; ii < nT16; ii += kNT) {   // thread = row
    const float* q = ch.Q + (size_t)(i0 + ii) * K;
#pragma unroll
    for (int k4 = 0; k4 < KQ; k4 += 4) {
      float4 v;
      v.x = ii < nT && k4 < K ? q[k4] : 0.0f;
      v.y = ii < nT && k4 + 1 < K ? q[k4 + 1] : 0.0f;
      v.z = ii < nT && k4 + 2 < K ? q[k4 + 2] : 0.0f;
      v.w = ii < nT && k4 + 3 < K ? q[k4 + 3] : 0.0f;
      *reinterpret_cast<float4*>(sQ + ii * KQ + k4) = v;
    }
  }
  if constexpr (DRAW) {
    for (int idx = threadIdx.x; idx < nT16 * NW * 2; idx += kNT) sM[idx] = 0;
    for (int idx = threadIdx.x; idx < nT16; idx += kNT) sPres[idx] = 0;
  }
  // the zero class of the lane's table; with three classes the slot behind the
  // last one, which a missing genotype reads (finite, its draw is masked)
  if (CL == 4) {
#pragma unroll
    for (int k = 0; k < NS; k++) sX[(k * CL + 3) * kNT + threadIdx.x] = make_float2(0.0f, 0.0f);
  } else {
    sX[NS * CL * kNT + threadIdx.x] = make_float2(0.0f, 0.0f);
  }
  __syncthreads();

  double like_acc = 0.0;
  const double magic = ch.ct_like_magic;
  const int n_sl = ch.n_sl, n_ska = ch.n_ska;
  for (int rb = 0; rb < R; rb++) {
    const int lbase = ((grp * R + rb) * kW + warp) * 32;
    if (lbase >= L) break;  // warp-uniform
    const int l = lbase + lane;
    const bool valid = l < L;
    Locus<KT> lo;
    lo.Prow = ch.P + (size_t)(valid ? l : 0) * K * A;
#pragma unroll
    for (int k = 0; k < KT; k++) {
      const float p0 = valid && k < K ? lo.Prow[(size_t)k * A] : 0.0f;
      const float p1 = valid && k < K && A > 1 ? lo.Prow[(size_t)k * A + 1] : 0.0f;
      if (k < NS) {
        float2* x = sX + k * CL * kNT + threadIdx.x;
        x[0] = make_float2(p0, p0);
        x[kNT] = make_float2(p0, p1);
        x[2 * kNT] = make_float2(p1, p1);
      } else {
        lo.p0[k >= NS ? k - NS : 0] = p0;
        lo.p1[k >= NS ? k - NS : 0] = p1;
      }
    }
    lo.grow = valid ? ch.g2 + (size_t)l * ch.wpr + (i0 >> 4) : nullptr;
    lo.tot = lo.tot1 = 0;
    const PhiloxRun prun((uint32_t)l, (uint32_t)rep, (uint32_t)kSZ, ch.key);
#pragma unroll
    for (int w = 0; w < (DRAW ? 4 * NW : 0); w++) sWide[w * kNT] = 0;
    __syncwarp();
    if (want_like)
      zcount_words<KT, true, DRAW>(nT16 >> 4, (uint32_t)(i0 >> 1), prun, smem, sQ, sWide, sRed, sM, sPres,
                             lo, like_acc, magic, K, A);
    else if constexpr (DRAW)
      zcount_words<KT, false, true>(nT16 >> 4, (uint32_t)(i0 >> 1), prun, smem, sQ, sWide, sRed, sM, sPres,
                              lo, like_acc, magic, K, A);
    if (DRAW && valid) {
      // copies with C_k < r, all and of allele 1: cum_{-1} is every copy
      int pa = 2 * lo.tot, p1 = lo.tot1;
      for (int k = 0; k < K; k++) {
        int ca = 0, c1 = 0;
        if (k < K - 1) {
          const int* d = sWide + ((k >> 2) * 4 + (k & 1)) * kNT;
          const int sft = (k & 2) * 8;
          ca = (d[0] >> sft) & 0xFFFF;
          c1 = (d[2 * kNT] >> sft) & 0xFFFF;
        }
        const int v1 = p1 - c1, v0 = pa - ca - v1;
        int32_t* dst = ch.npart + (size_t)l * n_sl + (size_t)k * A * n_ska;
        if (v0) atomicAdd(dst, v0);
        if (A > 1 && v1) atomicAdd(dst + n_ska, v1);
        pa = ca;
        p1 = c1;
      }
    }
    __syncwarp();
  }
  __syncthreads();
  if constexpr (DRAW) {
    // thread = row: n_k = cum_{k-1} - cum_k, cum_{-1} = copies present
    for (int ii = threadIdx.x; ii < nT; ii += kNT) {
      int* dst = ch.mpart + (size_t)(i0 + ii) * K;
      int prev = 2 * sPres[ii];
#pragma unroll
      for (int k = 0; k < KT; k++) {
        if (k < K) {
          int cum = 0;
          if (k < K - 1)
            cum = (int)(((uint32_t)sM[(ii * NW + (k >> 2)) * 2 + (k & 1)] >> ((k & 2) * 8)) & 0xFFFFu);
          if (prev != cum) atomicAdd(&dst[k], prev - cum);
          prev = cum;
        }
      }
    }
  }
  const int ntiles = ch.ctchunks * ch.ctgroups;
  if (want_like) {
    const double s = block_sum_d(like_acc, sred);
    if (threadIdx.x == 0) ch.likepart[tile] = s;
  }
  const bool advance = DRAW && (flags & kZfAdvance) != 0;
  if (want_like || advance) {
    if (last_cta_arrive(&ch.ctr[kCtrZ], (unsigned)ntiles)) {
      if (want_like) finish_like(ch, ntiles, collect && (flags & kZfCollect), sred);
      if (advance && threadIdx.x == 0) *ch.rep = rep + 1;
    }
  }
}

template <int KT>
cudaError_t launch_zcount_k(const LaunchSet& ls, int mode, int flags, size_t smem) {
  auto fn = mode == kZLike ? zcount_kernel<KT, false, false>
            : ls.behind    ? zcount_kernel<KT, true, true>
                           : zcount_kernel<KT, true, false>;
  if (const cudaError_t e = allow_dynamic_smem(fn, smem)) return e;
  if (mode == kZLike) {
    fn<<<ls.total_ctas, kNT, smem, ls.stream>>>(ls.chains, ls.prefix, ls.nchains, flags);
    return cudaGetLastError();
  }
  return launch_behind(ls, fn, fn, kNT, smem, ls.chains, ls.prefix, ls.nchains, flags);
}

}  // namespace zcount
}  // namespace st
