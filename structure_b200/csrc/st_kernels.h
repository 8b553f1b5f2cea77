// st_kernels.h -- host-side launchers of the sweep kernels.
#pragma once
#include <cuda_runtime.h>
#include "st_types.h"

namespace st {

// Chains covered by one launch: a device table of ChainDev and, per launch
// kind, the exclusive prefix of CTA counts (device array, nchains entries).
struct LaunchSet {
  ChainDev* chains;      // device pointer
  const int* prefix;     // device pointer
  int nchains;
  int total_ctas;
  cudaStream_t stream;
  bool behind = false;   // the launch may start while the kernel before it drains
};

// Dynamic shared memory that the planners of the data passes give a CTA at most.
constexpr size_t kMaxDynamicSmem = 200 * 1024;

// Lets `fn` be launched with `smem` bytes of dynamic shared memory.  The limit is the
// function's, for every context and thread on the device, so it is always set to the
// same ceiling: set to a launch's own size, another thread could lower it between
// this thread's setting and its launch.
template <typename F>
inline cudaError_t allow_dynamic_smem(F* fn, size_t smem) {
  if (smem <= 40 * 1024) return cudaSuccess;   // the default is 48 KB with the static part
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynamicSmem);
}

// Launches `fn`, or with ls.behind its instantiation `fnb`, which may start while the
// kernel before it on the stream drains (programmatic dependent launch).  fnb calls
// st_device.cuh's after_previous_kernel before it touches anything that a sweep's kernels
// write.  What it reads before that (parameters, chain descriptors) must have been
// written by a copy or by a kernel that an ordinary launch has followed since.
// The kernels do not signal before they end, so only the launch itself overlaps: blocks
// that are there early take the SMs that are free first, up to four on one, and a locus
// kernel of one to four blocks per SM then runs on some of the SMs while others idle.
// Ten sweeps of a lone chain, us, ordinary launches / a signal behind each main loop /
// none: 16 x 50,000 SNPs, K=10, F model 1524 / 1920 / 1447; 100 x 30,000, K=6 919 / 1017 /
// 854; 733 x 9973, K=3 870 / 813 / 773; 2 x 3000, K=3 325 / 282 / 278; 2500 x 20,000, K=6
// 2557 / 2485 / 2490.  Two signal early: the one-byte pass (kZfEarly) where the locus
// kernel behind it is of at most 16 blocks, too short for its place to matter (100
// microsatellites of 20 individuals, K=3: 264 against 275; 20 of 200, K=2: 265 against
// 280; but 1000 of 100, K=6, F model 602 against 503); and the locus kernel ahead of an F
// stage or called by itself, with the short individual kernel behind it (1000 x 10,001,
// K=4, an update at a time 77.0 against 78.8 us a step; 16 x 500, K=3 without F 284
// against 271).
// A lone chain's sweeps ask for it.
template <typename... P, typename... A>
inline cudaError_t launch_behind(const LaunchSet& ls, void (*fn)(P...), void (*fnb)(P...),
                                 unsigned block, size_t smem, A... args) {
  if (!ls.behind) {
    fn<<<ls.total_ctas, block, smem, ls.stream>>>(static_cast<P>(args)...);
    return cudaGetLastError();
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ls.total_ctas);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ls.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fnb, static_cast<P>(args)...);
}

// Z-pass modes.
enum ZMode : int { kZNormal = 0, kZInit = 1, kZRecount = 2, kZMetro = 3, kZLike = 4 };
// Z-pass flags.
enum : int {
  kZfLikeIfCollect = 0x1,  // compute ln P(D) when the sweep collects
  kZfLikeAlways = 0x2,     // compute ln P(D) regardless
  kZfStoreZ = 0x4,         // write Z bytes
  kZfCollect = 0x8,        // fold ln P(D) into sumlikes/sumsqlikes when collecting
  kZfAdvance = 0x10,       // bump the device sweep counter at the end
  kZfF64 = 0x20,           // generic path: FP64 arithmetic (reference bit-parity)
  kZfInjected = 0x40,      // generic path: uniforms from the injected array
  kZfCleared = 0x100,      // the count histograms are zero already
  kZfEarly = 0x200,        // the next kernel on the stream may launch before this one ends
  kZfInterleave = 0x80     // fast path: the launch's chains share one data set and
                           // tile, and block b runs tile b / nchains of chain
                           // b % nchains, so the chains' CTAs over the same loci run
                           // together and read the genotype words once from DRAM
};

// Locus-kernel stages.
// kLocClear: the P stage zeroes every allele count once it has read those it needs, and
// kIndClear (with the last launch of a sweep's Q update) the ancestry counts, so that
// the sweep's Z pass needs no memsets (kZfCleared).
enum : int { kLocP = 0x1, kLocEps = 0x2, kLocFst = 0x4, kLocCollect = 0x8, kLocClear = 0x10 };
// Individual-kernel modes and stages.
enum : int { kIndGibbs = 0, kIndPropose = 1, kIndAccept = 2, kIndNone = 3 };
enum : int { kIndAlpha = 0x1, kIndCollect = 0x2, kIndClear = 0x4 };

size_t zpass_b2g_smem(int KT, int K, int T, int W, int mode);
// CTAs of the general Z pass at its default tile for a chain of this shape
// (st_api.cu choose_tile).
long default_zpass_ctas(int N, int L, int K);
int zpass_b2g_width(int KT);   // CTA width (warps) of the fast path for a K class
cudaError_t launch_zpass_b2g(const LaunchSet& ls, int KT, int W, int mode, int flags,
                             size_t smem);
// The sweep's counting Z pass (biallelic data, no stored Z, every individual's
// alleles counted).  A tile is T individuals x R blocks of 256 loci per CTA.
struct CountTile { int T, R; };
constexpr int kZcountMinT = 32, kZcountMaxT = 512;
constexpr int kZcountMaxR = 127;   // 16-bit row counts: 512 copies per block
size_t zcount_smem(int KT, int T);
bool zcount_fits(int KT, int T);
long zcount_ctas(int N, int L, CountTile t);
// The tile for `chains` chains of this shape in one launch, with at most `cap` CTAs a
// chain (room for their ln P(D) partials); tile_t, tile_r: the caller's choice, or 0.
// T = 0: no tile fits.
CountTile zcount_tile(int N, int L, int KT, int tile_t, int tile_r, int chains, long cap);
double zcount_like_magic(int N, int L);
// mode: kZNormal, or kZLike (ln P(D) of the state, no draws)
cudaError_t launch_zcount(const LaunchSet& ls, int KT, int mode, int flags, size_t smem);
// The Metropolis pass on the general pass' tile (T, R) and CTAs.
size_t zmetro_smem(int KT, int T);
cudaError_t launch_zmetro(const LaunchSet& ls, int KT, int flags, size_t smem);
cudaError_t launch_zpass_u8(const LaunchSet& ls, int mode, int flags);
// One-byte layout, FP32 draws (st_zpass_u8.cu): modes kZNormal, kZLike and kZMetro.
// u8_plan chooses the loci per chunk with at most `cap` CTAs; 0: the per-genotype kernel.
int u8_plan(int N, int L, int K, int A, long cap);
int ctas_u8(const ChainDev& c);
size_t u8_smem(const ChainDev& c, int mode);
cudaError_t launch_u8(const LaunchSet& ls, int KT, int mode, int flags, size_t smem);
int u8_kclass(int K);
cudaError_t launch_locus(const LaunchSet& ls, int stages, int block);
cudaError_t launch_ind(const LaunchSet& ls, int mode, int stages, int block);
cudaError_t launch_collect(const LaunchSet& ls, int block);
cudaError_t launch_lambda(const LaunchSet& ls, int block);
// NOADMIX: per-individual population log likelihoods and the one-hot pick
void noadmix_plan(int N, int L, int* lchunks, int* lchunk_len);
cudaError_t launch_noadmix(const ChainDev& h, const ChainDev* d_chain, cudaStream_t s);
// USEPOPINFO: migrant-model Q of individuals with prior population information
void popinfo_plan(int N, int L, int* lchunks, int* lchunk_len);
cudaError_t launch_popinfo(const ChainDev& h, const ChainDev* d_chain, cudaStream_t s);

// LOCPRIOR (st_locprior.cu): UpdateLocPrior (r, and nu / gamma without
// admixture; also adds the LocPrior sums when collecting) and
// UpdateAlphaLocPrior (global and location alphas, with their sums).
cudaError_t launch_locprior(const ChainDev& h, const ChainDev* d_chain, cudaStream_t s);
cudaError_t launch_alpha_locprior(const ChainDev& h, const ChainDev* d_chain, cudaStream_t s);
// Injected-array parity modes (st_injected.cu): UpdateP and the proposal and
// accept steps of UpdateQMetro with the reference's own samplers.
cudaError_t launch_inj_p(const ChainDev& h, ChainDev* d_chain, const double* uni, cudaStream_t s);
cudaError_t launch_inj_metro_propose(const ChainDev& h, ChainDev* d_chain, const double* uni,
                                     int* taken, cudaStream_t s);
cudaError_t launch_inj_metro_accept(const ChainDev& h, ChainDev* d_chain, const double* uni,
                                    const int* taken, cudaStream_t s);
cudaError_t launch_pack_u8(const int32_t* geno, uint8_t* g8, size_t row0, int rows, int col0,
                           int cols, int N, cudaStream_t s);
cudaError_t launch_clear_counts(const ChainDev* d_table, int nchains, cudaStream_t s);
cudaError_t launch_init_chain(const ChainDev& h, ChainDev* d_chain, int* d_prefix,
                              const double* eps0, int arows, float q0, float lq0, double f0,
                              double alpha0, double lambda0, cudaStream_t s);

// CTA counts per chain for each launch kind (host-side mirror of the tiling).
int ctas_zpass_b2g(const ChainDev& c);
// CTAs of the per-genotype kernel, at the tile that set_zpass_u8_tile chose.
void set_zpass_u8_tile(ChainDev* c);
int ctas_zpass_u8(const ChainDev& c);
int ctas_locus(const ChainDev& c, int block);
int locus_lanes(int L, int K, int A, long others);
int ctas_ind(const ChainDev& c, int block);
int ctas_collect(const ChainDev& c, int block);
int ctas_lambda(const ChainDev& c, int block);

// Gradient of ln P(D|Q,P) (Z marginalised) w.r.t. softmax logits, biallelic
// 2-bit data.  T = float or double in every T buffer.
constexpr int kGradMaxK = 16;
struct GradArgs {
  int N, L, K, wpr;
  const uint32_t* g2;
  const void* qlog;       // T [N][K]
  const void* plog;       // T [L][K][2]
  void* Q;                // T [N][K]    softmax workspace
  void* P;                // T [L][K][2] softmax workspace
  void* gqpart;           // T [lchunks][N][K]
  double* llpart;         // [lchunks][N]
  void* gppart;           // T [ichunks][L][K][2]
  void* dq;               // T [N][K]
  void* dp;               // T [L][K][2]
  double* ll_ind;         // [N] or null
  double* loglik;         // scalar or null
  double* blockpart;      // [nblocks_q]
  int lchunks, lchunk_len, ichunks, ichunk_len, nblocks_q;
  cudaStream_t stream;
};
int grad_kclass(int K);                        // 0 if K is out of range
void grad_plan(int N, int L, int K, bool fp64, GradArgs* a);   // chunk sizes and counts
cudaError_t launch_loglik_grad(const GradArgs& a, bool fp64);
cudaError_t launch_grad_q(const GradArgs& a);   // ll_i and dll/dlogit(Q) only, FP32
// One Langevin move on every Q_i of a chain: cur.Q = chain Q, prop.Q = mQp.
cudaError_t launch_mala_step(const GradArgs& cur, const GradArgs& prop, const ChainDev* d_chain);

}  // namespace st
