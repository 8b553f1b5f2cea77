// st_zpass_u8.cu -- the data pass on one-byte genotypes [L][N][2] (any allele count,
// half-missing genotypes): the sweep's Z draws with counts and ln P(D), ln P(D) of a
// state, and the Metropolis log ratios; Z is stored where the chain keeps it.  The
// initial Z, recounts, FP64 draws, injected uniforms and chains of few individuals
// (u8_plan) take the per-genotype kernel of st_zpass.cu; the draws here are the same
// bits as that kernel's in FP32.
//
// The layout puts individuals side by side, so that a warp reads the copies of 32 pairs
// at a locus as one piece ([N][2][L] took a sector per byte: 56 instead of 37 us).
// Thread = a pair of individuals (one Philox block serves both at a locus), CTA =
// 128 pairs x a chunk of loci whose P is staged in shared memory allele by allele,
// rows of an odd length: a copy reads its allele's row at fixed offsets, and lanes with
// different alleles meet different banks.  Missing copies are counted as 0 or into a
// spare slot, so that the loop has no branch but the rare logarithm (with branches and
// rows [k][a] it took 647 warp instructions per 32 pairs and locus, 58 us).  Ancestry
// counts are lane-private columns in shared memory, allele counts a histogram per CTA;
// both leave as one coalesced set of integer reductions per CTA.  A kernel that added
// every copy to both histograms with global atomics and took an FP64 logarithm per copy
// needed 188 us per sweep for 8 chains of N=1000, L=300, K=6, bound by those atomics'
// latency.
//
// Logarithms: a thread multiplies its copies' terms in FP64 and takes one logarithm
// whenever the product falls below 1e-100 (terms are at least 1e-50 after
// CalcLike's clamp, so no product underflows).
#include "st_device.cuh"
#include "st_kernels.h"
#include "st_zpass_fast.cuh"

namespace st {
namespace {

using zfast::block_sum_d;
using zfast::finish_like;

constexpr int kUT = 128;            // threads: pairs of individuals per CTA
constexpr int kUMaxLc = 16;         // loci per chunk at most
constexpr size_t kUSmem = 64 * 1024;

struct U8Layout { int p, n, m, total; };

__host__ __device__ constexpr int u8_row(int KT) { return KT | 1; }   // words of an allele's row

__host__ __device__ inline U8Layout u8_layout(int KT, int K, int A, int lc, int mode) {
  U8Layout u;
  int o = 0;
  u.p = o; o += lc * u8_row(KT) * A * (mode == kZMetro ? 8 : 4);
  u.n = o; if (mode == kZNormal) o += (lc * K * A + 1) * 4;   // and a spare slot
  u.m = o; if (mode == kZNormal) o += K * kUT * 4;
  u.total = (o + 15) & ~15;
  return u;
}

// A running product of factors and the logarithms already taken of it.
struct LogProduct {
  double p = 1.0, s = 0.0;
  __device__ __forceinline__ void mul(double x) {
    p *= x;
    if (!(p >= 1e-100)) flush();
  }
  __device__ __forceinline__ void flush() {
    s += log(p);
    p = 1.0;
  }
};

template <int KT, int MODE, bool BEHIND>
__global__ void __launch_bounds__(kUT, KT <= 8 ? 4 : 3)
u8_kernel(ChainDev* __restrict__ chains, const int* __restrict__ prefix, int nchains, int flags) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double sred[kUT / 32];
  const int c = find_chain(prefix, nchains, blockIdx.x);
  ChainDev& ch = chains[c];
  const int tile = blockIdx.x - prefix[c];
  const int N = ch.N, L = ch.L, K = ch.K, A = ch.A;
  const int pb = tile / ch.u8_chunks, l0 = (tile - pb * ch.u8_chunks) * ch.u8_lc;
  const int nl = min(ch.u8_lc, L - l0);
  if (BEHIND) after_previous_kernel();
  const int rep = *ch.rep;
  const bool collect = rep + 1 > ch.burnin;
  const bool want_like = MODE == kZLike ||
      (MODE == kZNormal && ((flags & kZfLikeAlways) || ((flags & kZfLikeIfCollect) && collect)));
  const U8Layout lay = u8_layout(KT, K, A, ch.u8_lc, MODE);
  int* sN = reinterpret_cast<int*>(smem + lay.n);
  int* sM = reinterpret_cast<int*>(smem + lay.m);

  // P of the chunk's loci, [l][A][KS], zero beyond K
  constexpr int KS = u8_row(KT);
  for (int la = threadIdx.x; la < nl * A; la += kUT) {
    const int l = la / A, a = la - l * A;
    const float* P = ch.P + (size_t)(l0 + l) * K * A + a;
#pragma unroll
    for (int k = 0; k < KT; k++) {
      const float v = k < K ? P[(size_t)k * A] : 0.0f;
      if (MODE == kZMetro) reinterpret_cast<double*>(smem + lay.p)[la * KS + k] = (double)v;
      else reinterpret_cast<float*>(smem + lay.p)[la * KS + k] = v;
    }
  }
  if (MODE == kZNormal) {
    for (int idx = threadIdx.x; idx < nl * K * A; idx += kUT) sN[idx] = 0;
    for (int k = 0; k < K; k++) sM[k * kUT + threadIdx.x] = 0;
  }
  __syncthreads();

  const int pair = pb * kUT + threadIdx.x;
  const int i0 = 2 * pair;
  const int nh = min(2, N - i0);   // individuals of this thread (<= 0: none)
  double like_acc = 0.0;
  if constexpr (MODE == kZMetro) {
    const double* sP = reinterpret_cast<const double*>(smem + lay.p);
    for (int h = 0; h < nh; h++) {
      const int i = i0 + h;
      double q[KT], t[KT];
#pragma unroll
      for (int k = 0; k < KT; k++) {
        q[k] = k < K ? (double)ch.Q[(size_t)i * K + k] : 0.0;
        t[k] = k < K ? (double)ch.TestQ[(size_t)i * K + k] : 0.0;
      }
      const uint16_t* g = reinterpret_cast<const uint16_t*>(ch.g8) + (size_t)l0 * N + i;
      LogProduct tp, tm;
      for (int l = 0; l < nl; l++) {
        const uint32_t ab = __ldg(g + (size_t)l * N);
#pragma unroll
        for (int line = 0; line < 2; line++) {
          const int a = (int)((ab >> (8 * line)) & 0xFFu);
          if (a == kG8Missing) continue;
          const double* P = sP + (l * A + a) * KS;
          double st = 0.0, sm = 0.0;
#pragma unroll
          for (int k = 0; k < KT; k++) {
            const double p = P[k];
            st += t[k] * p;
            sm += q[k] * p;
          }
          tp.mul(st);
          tm.mul(sm);
        }
      }
      tp.flush();
      tm.flush();
      const double ld = tp.s - tm.s;
      if (ld != 0.0) atomicAdd(&ch.ldpart[i], ld);
    }
    return;
  } else {
    const float* sP = reinterpret_cast<const float*>(smem + lay.p);
    const uint32_t key = ch.key;
    float q[2][KT];
    bool ncnt[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
#pragma unroll
      for (int k = 0; k < KT; k++)
        q[h][k] = h < nh && k < K ? ch.Q[(size_t)(i0 + h) * K + k] : 0.0f;
      ncnt[h] = h < nh && (!ch.pfrompopflagonly || ch.popflags[i0 + h] == 1);
    }
    const bool store_z = MODE == kZNormal && (flags & kZfStoreZ) && ch.Z;
    const int spare = nl * K * A, KA = K * A;
    // the signs of the K - 1 thresholds: those of the class' padding count only where
    // a weight is negative (a caller may set any Q and P), and z then stays below K
    const uint32_t zkeep = KT <= 8 ? 0xFFFFFFFFu   // classes of one K
                                   : 0xFFFFFFFFu << (KT - K);
    int* myM = sM + threadIdx.x;
    LogProduct lp;
    // the pair's copies at a locus: two 16-bit loads side by side; individuals beyond
    // the last are missing
    const uint16_t* g = reinterpret_cast<const uint16_t*>(ch.g8) + (size_t)l0 * N + (nh > 0 ? i0 : 0);
    uint32_t nx[2];
    auto fetch = [&](int l) {
      nx[0] = nh > 0 ? __ldg(g + (size_t)l * N) : 0xFFFFu;
      nx[1] = nh > 1 ? __ldg(g + (size_t)l * N + 1) : 0xFFFFu;
    };
    fetch(0);
    for (int l = 0; l < nl; l++) {
      const uint32_t a[4] = {nx[0] & 0xFFu, nx[0] >> 8, nx[1] & 0xFFu, nx[1] >> 8};
      if (l + 1 < nl) fetch(l + 1);
      U4 w{0, 0, 0, 0};
      if (MODE == kZNormal)
        w = philox_s((uint32_t)(l0 + l), (uint32_t)pair, (uint32_t)rep, (uint32_t)kSZ, key);
      const float* Pl = sP + l * A * KS;
      double prod = 1.0;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const bool m0 = a[2 * h] == kG8Missing, m1 = a[2 * h + 1] == kG8Missing;
        const int a0 = m0 ? 0 : (int)a[2 * h], a1 = m1 ? 0 : (int)a[2 * h + 1];
        const float* P0 = Pl + a0 * KS;
        const float* P1 = Pl + a1 * KS;
        float2 C[KT];
#pragma unroll
        for (int k = 0; k < KT; k++) {
          const float2 X = make_float2(P0[k], P1[k]);
          const float2 qq = make_float2(q[h][k], q[h][k]);
          C[k] = k == 0 ? mul2_rn(qq, X) : fma2_rn(qq, X, C[k > 0 ? k - 1 : 0]);
        }
        const float2 T = C[KT - 1];
        if (want_like) {
          // CalcLike's clamp at 1e-50 lies below the least FP32 number, so only a
          // zero meets it
          const double x = m0 ? 1.0 : T.x > 0.0f ? (double)T.x : 1e-50;
          const double y = m1 ? 1.0 : T.y > 0.0f ? (double)T.y : 1e-50;
          prod *= x * y;
        }
        if (MODE == kZNormal) {
          // z = #{k : C_k < RN(u T)}: the signs of C_k - r (st_zpass_fast.cuh)
          const float2 NM = make_float2(neg_one_plus_u23(h ? w.z : w.x),
                                        neg_one_plus_u23(h ? w.w : w.y));
          const float2 NR = fma2_rn(NM, T, T);
          uint32_t t0 = 0u, t1 = 0u;
#pragma unroll
          for (int k = 0; k < KT - 1; k++) {
            const float2 D = add2_rn(C[k], NR);
            t0 = __funnelshift_l(__float_as_uint(D.x), t0, 1);
            t1 = __funnelshift_l(__float_as_uint(D.y), t1, 1);
          }
          const int z0 = __popc(t0 & zkeep), z1 = __popc(t1 & zkeep), one = h ? 65536 : 1;
          atomicAdd(&myM[z0 * kUT], m0 ? 0 : one);
          atomicAdd(&myM[z1 * kUT], m1 ? 0 : one);
          atomicAdd(&sN[!m0 && ncnt[h] ? l * KA + z0 * A + a0 : spare], 1);
          atomicAdd(&sN[!m1 && ncnt[h] ? l * KA + z1 * A + a1 : spare], 1);
          if (store_z && h < nh) {
            uint8_t* Z = ch.Z + (size_t)(i0 + h) * 2 * L + l0 + l;
            Z[0] = m0 ? kZMissing : (uint8_t)z0;
            Z[L] = m1 ? kZMissing : (uint8_t)z1;
          }
        }
      }
      if (want_like) lp.mul(prod);   // four factors of at least 1e-50 at a time
    }
    if (want_like) {
      lp.flush();
      like_acc = lp.s;
    }
    if (BEHIND && (flags & kZfEarly)) next_kernel_may_launch();
    if (MODE == kZNormal) {
      __syncthreads();
      for (int idx = threadIdx.x; idx < nl * K * A; idx += kUT) {   // locus fastest
        const int ka = idx / nl, l = idx - ka * nl;
        const int v = sN[l * K * A + ka];
        if (v) atomicAdd(&ch.npart[(size_t)ka * L + l0 + l], v);
      }
      // ancestry counts, coalesced: element e = (row, k) in steps of kUT
      const int r0 = pb * 2 * kUT, ne = min(2 * kUT, N - r0) * K;
      int* dst = ch.mpart + (size_t)r0 * K;
      const int dr = kUT / K, dk = kUT - dr * K;
      int row = threadIdx.x / K, k = threadIdx.x - row * K;
      for (int e = threadIdx.x; e < ne; e += kUT) {
        const int v = (sM[k * kUT + (row >> 1)] >> (16 * (row & 1))) & 0xFFFF;
        if (v) atomicAdd(&dst[e], v);
        row += dr;
        k += dk;
        if (k >= K) {
          k -= K;
          row++;
        }
      }
    }
  }
  const int ntiles = ch.u8_chunks * ((N + 2 * kUT - 1) / (2 * kUT));
  if (want_like) {
    const double s = block_sum_d(like_acc, sred);
    if (threadIdx.x == 0) ch.likepart[tile] = s;
  }
  const bool advance = MODE == kZNormal && (flags & kZfAdvance) != 0;
  if (want_like || advance) {
    if (last_cta_arrive(&ch.ctr[kCtrZ], (unsigned)ntiles)) {
      if (want_like) finish_like(ch, ntiles, collect && (flags & kZfCollect), sred);
      if (advance && threadIdx.x == 0) *ch.rep = rep + 1;
    }
  }
}

template <int KT>
cudaError_t launch_kt(const LaunchSet& ls, int mode, int flags, size_t smem) {
  auto go = [&](auto fn, auto fnb) {
    if (const cudaError_t e = allow_dynamic_smem(ls.behind ? fnb : fn, smem)) return e;
    return launch_behind(ls, fn, fnb, kUT, smem, ls.chains, ls.prefix, ls.nchains, flags);
  };
  switch (mode) {
    case kZNormal: return go(u8_kernel<KT, kZNormal, false>, u8_kernel<KT, kZNormal, true>);
    case kZLike: return go(u8_kernel<KT, kZLike, false>, u8_kernel<KT, kZLike, true>);
    case kZMetro: return go(u8_kernel<KT, kZMetro, false>, u8_kernel<KT, kZMetro, true>);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

int u8_kclass(int K) {
  for (int k : {1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 16, 24, 32})
    if (k >= K) return k;
  return 0;
}

int ctas_u8(const ChainDev& c) { return c.u8_chunks * ((c.N + 2 * kUT - 1) / (2 * kUT)); }

size_t u8_smem(const ChainDev& c, int mode) {
  return (size_t)u8_layout(u8_kclass(c.K), c.K, c.A, c.u8_lc, mode).total;
}

// Loci per chunk: about one CTA per SM from one chain (a small chain gets one locus
// per CTA, a large one up to 16 so that a CTA's staging and reductions are shared by
// more copies: 8 chains of N=1000, L=300, K=6 take 37 us with 9 loci, 43 with 5; one
// such chain 17.8 against 16.9), within the shared memory and the room for the
// partials.  It depends on the chain's shape alone, so ln P(D) is the same in a batch.
// 0: the per-genotype kernel, which also serves chains of few individuals: the P of a
// chunk is then staged for few copies, more of them with more alleles and populations
// (ten sweeps, us, per-genotype against tiled: 16 x 40,000, K=3, 2 alleles 921 / 1142,
// 32 x 40,000 1411 / 1188; K=10, 6 alleles 16 x 5000 616 / 720, 48 x 5000 770 / 734;
// K=20, 30 alleles 100 x 5000 3574 / 3968, 2 x 5000 2967 / 3880).  Chunks of one locus
// fill the chip less than once either way, and stage less.
int u8_plan(int N, int L, int K, int A, long cap) {
  const long blocks = (N + 2 * kUT - 1) / (2 * kUT);
  long lc = (L * blocks + 148 - 1) / 148;
  if (lc > kUMaxLc) lc = kUMaxLc;
  if (lc > 1 && 4 * (long)(N - 18) < (long)K * A) return 0;
  const int KT = u8_kclass(K);
  while (lc > 1 && (u8_layout(KT, K, A, (int)lc, kZNormal).total > (int)kUSmem ||
                    u8_layout(KT, K, A, (int)lc, kZMetro).total > (int)kUSmem))
    lc--;
  while (lc <= kUMaxLc && blocks * ((L + lc - 1) / lc) > cap) lc++;
  if (lc > kUMaxLc || u8_layout(KT, K, A, (int)lc, kZNormal).total > (int)kMaxDynamicSmem ||
      u8_layout(KT, K, A, (int)lc, kZMetro).total > (int)kMaxDynamicSmem)
    return 0;
  return (int)lc;
}

// The launch's chains share the K class KT; smem: their largest u8_smem.
cudaError_t launch_u8(const LaunchSet& ls, int KT, int mode, int flags, size_t smem) {
  switch (KT) {
#define ST_KCASE(k) case k: return launch_kt<k>(ls, mode, flags, smem);
    ST_KCASE(1) ST_KCASE(2) ST_KCASE(3) ST_KCASE(4) ST_KCASE(5) ST_KCASE(6) ST_KCASE(7) ST_KCASE(8)
    ST_KCASE(10) ST_KCASE(12) ST_KCASE(16) ST_KCASE(24) ST_KCASE(32)
#undef ST_KCASE
  }
  return cudaErrorInvalidValue;
}

}  // namespace st
