// st_zpass.cu -- the data pass of a sweep: one read of the genotypes that
// draws every allele copy's population of origin Z (Updates/UpdateZ.c:13-56,
// mymath.c:105-129), histograms the draws into the allele counts n[l][k][a]
// (Updates/UpdateP.c:60-99 GetNumFromPops) and ancestry counts m[i][k]
// (Updates/UpdateQ.c:17-35 GetNumLociPop) for the next sweep's P and Q
// updates, and, when asked, reduces ln P(D|Q,P) (CalcLike.c:75-133,387-426).
// The Metropolis Q move's likelihood ratio (CalcLike.c:281-345) and the initial random
// Z (Init.c:125-169) are passes over the same data.
//
// This file holds the dispatchers, the tile rules, the per-genotype kernel of one-byte
// data (FP64 arithmetic, injected uniforms, initial Z, counts of a given Z, chains of few
// individuals) and the packing of that data.  The paths by data and chain:
//   2 bits per genotype   draws and counts, ln P(D)    st_zcount.cuh
//                         Metropolis ratio             st_zmetro.cuh
//                         Init, recount; Z stored,     st_zpass_fast.cuh
//                         PFROMPOPFLAGONLY
//   one byte per copy     draws, ln P(D), Metropolis   st_zpass_u8.cu
//                         the rest                     zpass_u8_kernel, below
#include <algorithm>
#include <cmath>
#include <cstdio>
#include "st_device.cuh"
#include "st_kernels.h"

namespace st {

namespace {

// Deterministic block sum of one double per thread (fixed tree order).
__device__ __forceinline__ double block_sum_d(double v, double* sred) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sred[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    for (int w = 0; w < nw; w++) s += sred[w];
  }
  return s;  // valid in thread 0
}

// Last CTA of a chain: sum the per-CTA ln-likelihood partials in a fixed
// order (each thread a compensated sum of a strided subset, then the block's
// tree) and fold them into the chain's stats.
static __device__ void finish_like(ChainDev& ch, int ntiles, bool collect, double* sred) {
  CompSum v;
  for (int j = threadIdx.x; j < ntiles; j += blockDim.x) v.add(ch.likepart[j]);
  double s = block_sum_d(v.value(), sred);
  if (threadIdx.x == 0) {
    ch.stats[kStLike] = s;
    if (collect) {
      ch.stats[kStSumLikes] += s;
      ch.stats[kStSumSq] += s * s;
      ch.stats[kStNLike] += 1.0;
    }
  }
}

}  // namespace

namespace zfast {
template <int KT, int W>
cudaError_t launch_b2g_kw(const LaunchSet& ls, int mode, int flags, size_t smem);
size_t zlayout_total(int KT, int K, int T, int nw32, int mode);
}  // namespace zfast

int ctas_zpass_b2g(const ChainDev& c) { return c.nchunks * c.ngroups; }

size_t zpass_b2g_smem(int KT, int K, int T, int W, int mode) {
  return zfast::zlayout_total(KT, K, T, 32 * W, mode);
}

int zpass_b2g_width(int KT) { return KT <= 12 ? 8 : 2; }

// smem must be sized for the largest tile among the chains of the launch; the
// CTA width is fixed per K class (zpass_b2g_width).
cudaError_t launch_zpass_b2g(const LaunchSet& ls, int KT, int W, int mode, int flags,
                             size_t smem) {
  if (W != zpass_b2g_width(KT)) return cudaErrorInvalidConfiguration;
  switch (KT) {
#define ST_KCASE(k, w) case k: return zfast::launch_b2g_kw<k, w>(ls, mode, flags, smem);
    ST_KCASE(1, 8) ST_KCASE(2, 8) ST_KCASE(3, 8) ST_KCASE(4, 8) ST_KCASE(5, 8) ST_KCASE(6, 8)
    ST_KCASE(7, 8) ST_KCASE(8, 8) ST_KCASE(9, 8) ST_KCASE(10, 8) ST_KCASE(11, 8) ST_KCASE(12, 8)
    ST_KCASE(16, 2) ST_KCASE(20, 2) ST_KCASE(24, 2) ST_KCASE(32, 2)
#undef ST_KCASE
  }
  return cudaErrorInvalidValue;
}

namespace zcount {
template <int KT>
cudaError_t launch_zcount_k(const LaunchSet& ls, int mode, int flags, size_t smem);
size_t zc_layout_total(int kt, int T);
int zc_ctas_of(int kt);
}  // namespace zcount

size_t zcount_smem(int KT, int T) { return zcount::zc_layout_total(KT, T); }
bool zcount_fits(int KT, int T) {
  return T >= kZcountMinT && T <= kZcountMaxT && T % 16 == 0 && zcount_smem(KT, T) <= kMaxDynamicSmem;
}
long zcount_ctas(int N, int L, CountTile t) {
  const long blocks = (L + 255) / 256;   // 8 warps of 32 loci
  return (blocks + t.R - 1) / t.R * ((N + t.T - 1) / t.T);
}

// Individuals per chunk: the count of equal chunks with the least estimated time.  A
// CTA costs its rows plus about 24 rows of fixed work per locus block (measured at
// K=5: 128 rows 4 % above 256, 336 rows 1 % below); CTAs that share an SM share its
// pipes, with fewer of them using it less fully (K=5: 2 instead of 3 CTAs 12 %
// slower, 1 about 35 %).  A grid within one wave takes as long as its fullest SM; a
// longer one, its mean plus half a wave of tail.  Several locus blocks per CTA save
// next to nothing (0.3 % at K=5): R only keeps the CTAs within their partials.
CountTile zcount_tile(int N, int L, int KT, int tile_t, int tile_r, int chains, long cap) {
  const int np = (N + 15) & ~15;
  auto with_r = [&](int T) {
    CountTile t{T, tile_r > 0 ? (tile_r < kZcountMaxR ? tile_r : kZcountMaxR) : 1};
    while (t.R < kZcountMaxR && zcount_ctas(N, L, t) > cap) t.R++;
    return t;
  };
  CountTile best{0, 1};
  if (tile_t > 0) {
    int T = (tile_t + 15) & ~15;
    T = T > np ? np : T;
    T = T > kZcountMaxT ? kZcountMaxT : T < kZcountMinT ? kZcountMinT : T;
    while (T > kZcountMinT && !zcount_fits(KT, T)) T -= 16;
    const CountTile t = with_r(T);
    return zcount_ctas(N, L, t) <= cap ? t : best;
  }
  double best_t = 1e300;
  // (each tile once: the count that gives the largest, then the next smaller one's)
  for (int n = (N - 1) / kZcountMaxT + 1, next; n <= (np + kZcountMinT - 1) / kZcountMinT; n = next) {
    int T = ((N + n - 1) / n + 15) & ~15;
    if (T < kZcountMinT) T = kZcountMinT;
    next = T > kZcountMinT ? std::max(n + 1, (N - 1) / (T - 16) + 1) : n + 1;
    if (!zcount_fits(KT, T)) continue;
    const CountTile c = with_r(T);
    const long ctas1 = zcount_ctas(N, L, c);
    if (ctas1 > cap) continue;
    int occ = (int)((227 * 1024) / (zcount_smem(KT, T) + 1024 + 64));
    if (occ > zcount::zc_ctas_of(KT)) occ = zcount::zc_ctas_of(KT);
    const long ctas = ctas1 * chains, per_sm = (ctas + 147) / 148;
    const int live = per_sm < occ ? (int)per_sm : occ;
    const double eff = live >= 3 ? 1.0 : live == 2 ? 1.12 : 1.35;
    const double n_sm = per_sm <= occ ? (double)per_sm : (double)ctas / 148.0 + 0.5 * occ;
    const double t = n_sm * eff * c.R * (T + 24);
    if (t < best_t) {
      best_t = t;
      best = c;
    }
    if (T <= kZcountMinT) break;
  }
  return best;
}

// ln P(D) is the sum of one FP32 value per genotype word (16 genotypes of a locus).
// Rounded to a common quantum 2^-(47 - log2 words), the values add exactly in FP64
// while they average below 32, so the sum does not depend on the tile: a batch and a
// chain alone, at their own tiles, get the same bits.  The quantum is far below the
// words' own FP32 rounding (2^-24 at 2^23 words of about 10 +- 2^-21).  Adding and
// subtracting 1.5 x 2^52 quanta rounds to it.
double zcount_like_magic(int N, int L) {
  const double words = (double)L * ((N + 15) / 16);
  int lg = 0;
  while (lg < 46 && (double)(1ull << lg) < words) lg++;
  return ldexp(1.5, 52 - (47 - lg));
}

cudaError_t launch_zcount(const LaunchSet& ls, int KT, int mode, int flags, size_t smem) {
  switch (KT) {
#define ST_KCASE(k) case k: return zcount::launch_zcount_k<k>(ls, mode, flags, smem);
    ST_KCASE(1) ST_KCASE(2) ST_KCASE(3) ST_KCASE(4) ST_KCASE(5) ST_KCASE(6) ST_KCASE(7) ST_KCASE(8)
    ST_KCASE(9) ST_KCASE(10) ST_KCASE(11) ST_KCASE(12) ST_KCASE(16) ST_KCASE(20) ST_KCASE(24)
    ST_KCASE(32)
#undef ST_KCASE
  }
  return cudaErrorInvalidValue;
}

namespace zmetro {
template <int KT>
cudaError_t launch_zmetro_k(const LaunchSet& ls, int flags, size_t smem);
size_t layout_total(int kt, int T);
}  // namespace zmetro

size_t zmetro_smem(int KT, int T) { return zmetro::layout_total(KT, T); }

cudaError_t launch_zmetro(const LaunchSet& ls, int KT, int flags, size_t smem) {
  switch (KT) {
#define ST_KCASE(k) case k: return zmetro::launch_zmetro_k<k>(ls, flags, smem);
    ST_KCASE(1) ST_KCASE(2) ST_KCASE(3) ST_KCASE(4) ST_KCASE(5) ST_KCASE(6) ST_KCASE(7) ST_KCASE(8)
    ST_KCASE(9) ST_KCASE(10) ST_KCASE(11) ST_KCASE(12) ST_KCASE(16) ST_KCASE(20) ST_KCASE(24)
    ST_KCASE(32)
#undef ST_KCASE
  }
  return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Generic path: one thread per (individual, locus), any allele count, runtime
// K, FP32 or FP64 arithmetic, Philox or injected uniforms.  Counts go to slice
// 0 of the partial arrays with global atomics (zeroed by the host before), summed
// over the CTA before that: thousands of copies share an individual's or, with many
// individuals, a locus' few counts.
// ---------------------------------------------------------------------------
constexpr int kU8Threads = 256;   // 2^8
constexpr int kU8Bins = 2048;   // allele counts of a CTA's loci kept in shared memory

template <typename TF>
__device__ __forceinline__ int pick_generic(const float* q, const float* Pl, int K, int A,
                                            int a, TF u, TF& total, int& errb);

template <>
__device__ __forceinline__ int pick_generic<float>(const float* q, const float* Pl, int K, int A,
                                                   int a, float u, float& total, int& errb) {
  float C[kMaxPops];
  C[0] = q[0] * Pl[a];
  for (int k = 1; k < K; k++) C[k] = __fmaf_rn(q[k], Pl[(size_t)k * A + a], C[k - 1]);
  total = C[K - 1];
  const float r = u * total;
  int z = 0;
  for (int k = 0; k < K - 1; k++) z += (C[k] < r);
  return z;
}

template <>
__device__ __forceinline__ int pick_generic<double>(const float* q, const float* Pl, int K, int A,
                                                    int a, double u, double& total, int& errb) {
  double Wt[kMaxPops];
  double sum = 0.0;
  for (int k = 0; k < K; k++) {
    Wt[k] = __dmul_rn((double)q[k], (double)Pl[(size_t)k * A + a]);
    sum = __dadd_rn(sum, Wt[k]);
  }
  total = sum;
  const double r = __dadd_rn(0.0, __dmul_rn(u, __dadd_rn(sum, -0.0)));
  double so = 0.0;
  int k = 0;
  for (; k < K; k++) {
    so = __dadd_rn(so, Wt[k]);
    if (r <= so) break;
  }
  if (k == K) { k = K - 1; errb |= kErrFallThrough; }
  return k;
}

template <typename TF>
__global__ void __launch_bounds__(256)
zpass_u8_kernel(ChainDev* __restrict__ chains, const int* __restrict__ prefix, int nchains,
                int mode, int flags) {
  __shared__ double sred[8];
  __shared__ int sM[32 * kMaxPops], sN[kU8Bins];
  const int c = find_chain(prefix, nchains, blockIdx.x);
  ChainDev& ch = chains[c];
  const int tile = blockIdx.x - prefix[c];
  const int N = ch.N, L = ch.L, K = ch.K, A = ch.A;
  const int inds = 1 << ch.gen_shift, loci = kU8Threads >> ch.gen_shift;
  const int it = tile / ch.gen_ltiles;
  const int i0 = it * inds, l0 = (tile - it * ch.gen_ltiles) * loci;
  const int ii = (int)threadIdx.x & (inds - 1), li = (int)threadIdx.x >> ch.gen_shift;
  const int i = i0 + ii, l = l0 + li;
  const bool active = i < N && l < L;
  const bool counts = mode == kZNormal || mode == kZInit || mode == kZRecount;
  const bool binned = loci * K * A <= kU8Bins;
  if (counts) {
    for (int e = threadIdx.x; e < inds * K; e += kU8Threads) sM[e] = 0;
    if (binned)
      for (int e = threadIdx.x; e < loci * K * A; e += kU8Threads) sN[e] = 0;
    __syncthreads();
  }
  const int rep = *ch.rep;
  const bool collect = rep + 1 > ch.burnin;
  const bool want_like = (mode == kZLike) ||
      (mode == kZNormal && ((flags & kZfLikeAlways) || ((flags & kZfLikeIfCollect) && collect)));
  const bool injected = (flags & kZfInjected) && ch.injected;
  int errb = 0;
  double like_acc = 0.0;

  if (active) {
    const uint8_t* g = ch.g8 + ((size_t)l * N + i) * 2;
    const uint8_t gv[2] = {g[0], g[1]};
    const float* q = ch.Q + (size_t)i * K;
    const float* Pl = ch.P + (size_t)l * K * A;
    U4 r4 = {0, 0, 0, 0};
    if (!injected && (mode == kZNormal || mode == kZInit))
      r4 = philox_s((uint32_t)l, (uint32_t)(i >> 1), mode == kZInit ? 0u : (uint32_t)rep,
                    mode == kZInit ? (uint32_t)kSInitZ : (uint32_t)kSZ, ch.key);
    const uint32_t wsel[2] = {(i & 1) ? r4.z : r4.x, (i & 1) ? r4.w : r4.y};
    int taken = 0;
    double ld = 0.0;
    for (int line = 0; line < 2; line++) {
      const int a = gv[line];
      const bool miss = a == kG8Missing;
      int z = 0;
      if (mode == kZNormal || mode == kZLike) {
        if (miss) { if (ch.Z && (flags & kZfStoreZ)) ch.Z[((size_t)i * 2 + line) * L + l] = kZMissing; continue; }
        TF total;
        TF u;
        if (injected) u = (TF)ch.injected[(size_t)i * L * 2 + (size_t)l * 2 + taken];
        else u = (TF)u23(wsel[line]);
        taken++;
        z = pick_generic<TF>(q, Pl, K, A, a, u, total, errb);
        if (want_like) like_acc += log(fmax((double)total, 1e-50));
      } else if (mode == kZInit) {
        if (miss) { if (ch.Z && (flags & kZfStoreZ)) ch.Z[((size_t)i * 2 + line) * L + l] = kZMissing; continue; }
        z = (int)(((uint64_t)(wsel[line] >> 1) * (uint64_t)K) >> 31);
        // USEPOPINFO: start at the given population (src/Init.c:74-117)
        if (ch.initpop && ch.initpop[i] >= 0) z = ch.initpop[i];
      } else if (mode == kZRecount) {
        if (miss) continue;
        z = ch.Z[((size_t)i * 2 + line) * L + l];
        if (z >= K) { errb |= kErrBounds; continue; }
      } else if (mode == kZMetro) {
        if (miss) continue;
        double tp = 0.0, tm = 0.0;
        for (int k = 0; k < K; k++) {
          const double p = (double)Pl[(size_t)k * A + a];
          tp += (double)ch.TestQ[(size_t)i * K + k] * p;
          tm += (double)q[k] * p;
        }
        ld += log(tp) - log(tm);
        continue;
      }
      if (mode == kZNormal || mode == kZInit || mode == kZRecount) {
        if (mode != kZRecount && ch.Z && (flags & kZfStoreZ))
          ch.Z[((size_t)i * 2 + line) * L + l] = (uint8_t)z;
        if (mode == kZLike) continue;
        atomicAdd(&sM[ii * K + z], 1);
        if (!ch.pfrompopflagonly || ch.popflags[i] == 1) {
          if (binned) atomicAdd(&sN[(z * A + a) * loci + li], 1);
          else atomicAdd(&ch.npart[((size_t)z * A + a) * L + l], 1);
        }
      }
    }
    if (mode == kZMetro) atomicAdd(&ch.ldpart[i], ld);
  }
  if (errb) set_err(ch.err, errb);
  if (counts) {
    __syncthreads();
    for (int e = threadIdx.x; e < inds * K; e += kU8Threads)
      if (sM[e]) atomicAdd(&ch.mpart[(size_t)i0 * K + e], sM[e]);
    if (binned)
      for (int e = threadIdx.x; e < loci * K * A; e += kU8Threads)
        if (sN[e])
          atomicAdd(&ch.npart[(size_t)(e >> (8 - ch.gen_shift)) * L + l0 + (e & (loci - 1))], sN[e]);
  }
  const int ntiles = (N + inds - 1) / inds * ch.gen_ltiles;
  if (want_like) {
    double s = block_sum_d(like_acc, sred);
    if (threadIdx.x == 0) ch.likepart[tile] = s;
  }
  const bool advance = (flags & kZfAdvance) != 0;
  if (want_like || advance) {
    if (last_cta_arrive(&ch.ctr[kCtrZ], (unsigned)ntiles)) {
      if (want_like) finish_like(ch, ntiles, collect && (flags & kZfCollect), sred);
      if (advance && threadIdx.x == 0) *ch.rep = rep + 1;
    }
  }
}

// Individuals of a CTA: a power of two up to 32, neighbouring lanes, as the genotypes
// [L][N][2] lie, for at most an eighth of idle lanes; its loci are kU8Threads over that.
void set_zpass_u8_tile(ChainDev* c) {
  int s = 5;
  while (s > 0 && (((c->N - 1) >> s) + 1) << s > c->N + c->N / 8) s--;
  const int loci = kU8Threads >> s;
  c->gen_shift = s;
  c->gen_ltiles = (c->L - 1) / loci + 1;
}

int ctas_zpass_u8(const ChainDev& c) { return (((c.N - 1) >> c.gen_shift) + 1) * c.gen_ltiles; }

cudaError_t launch_zpass_u8(const LaunchSet& ls, int mode, int flags) {
  dim3 grid(ls.total_ctas), block(kU8Threads);
  if (flags & kZfF64)
    zpass_u8_kernel<double><<<grid, block, 0, ls.stream>>>(ls.chains, ls.prefix, ls.nchains, mode, flags);
  else
    zpass_u8_kernel<float><<<grid, block, 0, ls.stream>>>(ls.chains, ls.prefix, ls.nchains, mode, flags);
  return cudaGetLastError();
}

// int32 reference genotypes (-9 missing) of `rows` copies (row = 2 i + line, from row0)
// at `cols` loci (from col0), [rows][cols], to one byte per copy (0xFF missing) in
// [L][N][2].  A CTA turns a tile in shared memory: loads run along the loci, stores
// along the copies.
constexpr int kPackTile = 64;

__global__ void __launch_bounds__(256)
pack_u8_kernel(const int32_t* __restrict__ geno, uint8_t* __restrict__ g8, size_t row0, int rows,
               int col0, int cols, size_t nrows) {
  __shared__ uint8_t tile[kPackTile][kPackTile + 4];   // [locus][row]; odd in words
  const int r0 = blockIdx.y * kPackTile, c0 = blockIdx.x * kPackTile;
  const int x = threadIdx.x % kPackTile, y = threadIdx.x / kPackTile;
  for (int r = y; r < kPackTile; r += 256 / kPackTile)
    if (r0 + r < rows && c0 + x < cols) {
      const int v = geno[(size_t)(r0 + r) * cols + c0 + x];
      tile[x][r] = (v < 0 || v > 254) ? kG8Missing : (uint8_t)v;
    }
  __syncthreads();
  for (int c = y; c < kPackTile; c += 256 / kPackTile)
    if (r0 + x < rows && c0 + c < cols)
      g8[(size_t)(col0 + c0 + c) * nrows + row0 + r0 + x] = tile[c][x];
}

cudaError_t launch_pack_u8(const int32_t* geno, uint8_t* g8, size_t row0, int rows, int col0,
                           int cols, int N, cudaStream_t s) {
  const dim3 grid((cols + kPackTile - 1) / kPackTile, (rows + kPackTile - 1) / kPackTile);
  pack_u8_kernel<<<grid, 256, 0, s>>>(geno, g8, row0, rows, col0, cols, (size_t)N * 2);
  return cudaGetLastError();
}

// Clears the allele and ancestry histograms (n [K][A][L], m [N][K]) of every
// chain of a batch before the counting Z pass: one launch, blockIdx.y = chain.
__global__ void clear_counts_kernel(const ChainDev* __restrict__ chains) {
  const ChainDev& ch = chains[blockIdx.y];
  const size_t nn = (size_t)ch.K * ch.A * ch.L, nm = (size_t)ch.N * ch.K;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < nn + nm; j += stride) {
    if (j < nn) ch.npart[j] = 0;
    else ch.mpart[j - nn] = 0;
  }
}

cudaError_t launch_clear_counts(const ChainDev* d_table, int nchains, cudaStream_t s) {
  clear_counts_kernel<<<dim3(64, nchains), 256, 0, s>>>(d_table);
  return cudaGetLastError();
}

}  // namespace st
