// Tensor contraction D = beta*D + alpha * sum_contracted L*R for sm_100a.
//
// Reference semantics: tensor_block_contract (tensor_algebra_cpu.F90:3675-4358)
// and gpu_tensor_block_contract_dlf (tensor_algebra_gpu_nvidia.cu:5847-7183):
// digital pattern, conjugation bits (the D bit flips the L and R bits), real
// kinds use real(alpha), beta = 1 when accumulative else D is overwritten.
//
// Design (no transpose + GEMM + transpose): every operand stays in its own
// layout.  The contraction is viewed as C[m,n] = sum_k A[m,k] B[k,n] where
//   m runs over L's uncontracted indices (L order), n over R's uncontracted
//   indices (R order) and k over the contracted pairs,
// and three small offset tables (m -> L and D offsets, n -> R and D offsets,
// k -> L and R offsets) built on the device turn every tile load into a
// gather and the epilogue into a scatter in D's own layout.  Tile loads are
// mapped so that the operand's stride-1 index runs across the lanes.
//  * R8: warp-level DMMA (mma.sync m8n8k4 f64) on a multistage cp.async
//    pipeline, FP64 end to end.
//  * C8: four DMMA products per complex product; R4 / C4: register-blocked packed
//    FP32 FMA; all on the same tables and pipeline.
//  * Degenerate patterns: full contraction (dot, deterministic two-pass),
//    scalar x tensor (the permute-add kernel with a device-side scale) and
//    scalar x scalar.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.h"
#include "device_once.h"

namespace tb {
int permute_scaled_by_device_scalar(int kind, int rank, const int *dims, const int *o2n,
                                    const void *src, void *dst, double alpha_re, double alpha_im,
                                    const void *scalar_dev, int scalar_conj, int tensor_conj,
                                    int accumulate, void *stream);
int permute_dot_launch(int kind, int rank, const int *dims, const int *o2n, const void *src, const void *dst,
                       int conj_src, int conj_dst, double2 *part, int64_t max_parts, int *nparts, cudaStream_t st);
namespace {

constexpr int kMaxGR = 24;  // max indices per group (m, n or k)

struct TableParams {
  int nm, nn, nk, nh;
  int64_t M, N, K, H;
  int64_t mext[kMaxGR], mstrL[kMaxGR], mstrD[kMaxGR];
  int64_t next[kMaxGR], nstrR[kMaxGR], nstrD[kMaxGR];
  int64_t kext[kMaxGR], kstrL[kMaxGR], kstrR[kMaxGR];
  // hyper-indices (in D, L and R): one independent GEMM per combination
  int64_t hext[kMaxGR], hstrL[kMaxGR], hstrR[kMaxGR], hstrD[kMaxGR];
  int64_t *mL, *mD, *nR, *nD, *kL, *kR;  // L and R offsets in bytes, D offsets in elements
  int64_t *hL, *hR, *hD;  // used when nh > 0 (all in elements)
  int es;                 // bytes per element of L and R
  int *cnt;               // arrival counters to zero (split contracted range)
  int64_t ncnt;
};

// Offsets of index i of a group: coordinates by 32-bit division (a group's
// range is below 2^31), first index fastest.
template <typename E>
__device__ __forceinline__ void group_offsets(uint32_t r, int n, const E *ext, const int64_t *sa, const int64_t *sb,
                                              int64_t &x, int64_t &y) {
  x = y = 0;
  for (int d = 0; d < n; ++d) {
    const uint32_t e = (uint32_t)ext[d], q = r / e;
    const int64_t c = (int64_t)(r - q * e);
    r = q;
    x += c * sa[d];
    y += c * sb[d];
  }
}

__global__ void build_tables_kernel(const TableParams T) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < T.ncnt; i += (int64_t)gridDim.x * blockDim.x)
    T.cnt[i] = 0;
  const int64_t mnk = T.M + T.N + T.K;
  const int64_t total = mnk + (T.nh > 0 ? T.H : 0);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int64_t x, y;
    if (i >= mnk) {
      const uint32_t r = (uint32_t)(i - mnk);
      group_offsets(r, T.nh, T.hext, T.hstrL, T.hstrR, x, y);
      T.hL[r] = x;
      T.hR[r] = y;
      group_offsets(r, T.nh, T.hext, T.hstrD, T.hstrD, x, y);
      T.hD[r] = x;
    } else if (i < T.M) {
      group_offsets((uint32_t)i, T.nm, T.mext, T.mstrL, T.mstrD, x, y);
      T.mL[i] = x * T.es;
      T.mD[i] = y;
    } else if (i < T.M + T.N) {
      group_offsets((uint32_t)(i - T.M), T.nn, T.next, T.nstrR, T.nstrD, x, y);
      T.nR[i - T.M] = x * T.es;
      T.nD[i - T.M] = y;
    } else {
      const int64_t k = i - T.M - T.N;
      group_offsets((uint32_t)k, T.nk, T.kext, T.kstrL, T.kstrR, x, y);
      T.kL[k] = x * T.es;
      T.kR[k] = y * T.es;
    }
  }
}

struct GemmArgs {
  int M, N, K;
  int tiles_m;
  int tiles_mn;                      // tiles of one GEMM (hyper-index launches)
  int H;                             // hyper combinations (1 without hyper-indices)
  const int64_t *hL, *hR, *hD;       // per hyper combination offsets, or null
  const int64_t *mL, *mD, *nR, *nD, *kL, *kR;
  double alpha_re, alpha_im;
  int beta;       // 1: D += ..., 0: D = ...
  int a_along_m;  // A tile loads: lanes along m (else along k)
  int b_along_n;  // B tile loads: lanes along n (else along k)
  int conj_l, conj_r;
  // Split contracted range (nsplit > 1): CTA (tile, s) sums k in
  // [s kchunk, (s+1) kchunk) and the partial tiles meet in `part`; without room
  // for them (part null) the CTA of a tile walks the splits itself (SeqSum).
  int nsplit, kchunk, gsz;
  int ncnt;   // arrival counters of this contraction (zeroed by the table kernel)
  void *part;
  int *cnt;
};

// One CTA's work: output tile (tm, tn) of one GEMM, the K range of its split,
// and the tile's number among all tiles of the launch (partial sums).
struct TileWork {
  int tm, tn, split, lin;
};

// Single-contraction launches: block b runs tile b mod tiles_mn of the GEMM for
// hyper combination (b / tiles_mn) mod H, whose operands start at the table
// offsets; the splits of the contracted range are the slowest index, so the
// CTAs in flight share their operands' k range in L2.
template <typename T>
__device__ __forceinline__ TileWork block_work(const GemmArgs &a, const T *&L, const T *&R, T *&D) {
  const int per = a.tiles_mn * (a.H > 1 ? a.H : 1);
  TileWork w;
  w.split = a.nsplit > 1 ? (int)blockIdx.x / per : 0;
  w.lin = (int)blockIdx.x - w.split * per;
  int local = w.lin;
  if (a.hL != nullptr) {
    const int h = local / a.tiles_mn;
    local -= h * a.tiles_mn;
    L += a.hL[h];
    R += a.hR[h];
    D += a.hD[h];
  }
  w.tm = local % a.tiles_m;
  w.tn = local / a.tiles_m;
  return w;
}

// Fragment arithmetic of the partial sums.
__device__ __forceinline__ void vadd(double2 &a, const double2 &b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void vadd(float4 &a, const float4 &b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }

// Meeting point of the CTAs that share an output tile (nsplit > 1).  Each CTA
// stores its partial fragments (16 bytes per slot, coalesced, at the thread's
// position `pos` in the tile; `mask` drops fragments beyond the tile's extents)
// and counts itself in; the last
// CTA of a group of gsz splits adds that group's partials in split order, and
// the last group adds the group sums in group order, so no CTA ever waits and
// the sum order does not depend on arrival.  Two levels keep the serial part
// at about 2 sqrt(nsplit) tile reads: one CTA adding 444 partial 64 x 64 tiles
// alone would read 14.5 MB.  Returns true in the CTA that holds the final sum.
// Counters go back to zero, so a recorded launch can be replayed.
template <int NF, int NT, typename V>
__device__ __forceinline__ bool split_combine(V (&acc)[NF], uint32_t mask, int pos, const GemmArgs &a, int lin,
                                              int split) {
  __shared__ int last;
  const int tid = threadIdx.x;
  V *base = (V *)a.part + (int64_t)lin * a.nsplit * (NF * NT) + pos;
  const int ng = (a.nsplit + a.gsz - 1) / a.gsz, g = split / a.gsz, s0 = g * a.gsz;
  const int gm = min(a.gsz, a.nsplit - s0);
  int *cnt = a.cnt + (int64_t)lin * (ng + 1);
  auto publish = [&](int s, int *c, int want) {
    V *to = base + (int64_t)s * (NF * NT);
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if ((mask >> f) & 1u) __stcg(to + f * NT, acc[f]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(c, 1) == want - 1 ? 1 : 0;
    __syncthreads();
    if (last && tid == 0) *c = 0;
    __threadfence();
    return last != 0;
  };
  auto gather = [&](int s, int n, int step) {
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if ((mask >> f) & 1u) acc[f] = __ldcg(base + (int64_t)s * (NF * NT) + f * NT);
    for (int j = 1; j < n; ++j) {
      const V *from = base + (int64_t)(s + j * step) * (NF * NT);
#pragma unroll
      for (int f = 0; f < NF; ++f)
        if ((mask >> f) & 1u) vadd(acc[f], __ldcg(from + f * NT));
    }
  };
  if (!publish(split, cnt + g, gm)) return false;
  gather(s0, gm, 1);
  if (ng == 1) return true;
  if (!publish(s0, cnt + ng, ng)) return false;
  gather(0, ng, a.gsz);
  return true;
}

// The sum of split_combine where there is no room for partial tiles: one CTA
// walks the splits in order and keeps the running group sum and the total, so
// a short scratch costs time and changes no bit.
template <int NF, typename V>
struct SeqSum {
  V group[NF], total[NF];
  __device__ __forceinline__ void add(const V (&acc)[NF], const GemmArgs &a, int s) {
    const int i = s % a.gsz;
    const bool closes = i == a.gsz - 1 || s == a.nsplit - 1;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      if (i == 0) group[f] = acc[f];
      else vadd(group[f], acc[f]);
      if (closes) {
        if (s < a.gsz) total[f] = group[f];
        else vadd(total[f], group[f]);
      }
    }
  }
};

// ---------------------------------------------------------------- R8: DMMA
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma_8x8x4(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

constexpr int kKRing = 4;  // slots of the shared k-offset ring

template <int BM, int BN>
struct DmmaCfg {
  // warp tile: 32x32, or 16x16 in 32x32 CTA tiles (four warps per CTA either way)
  static constexpr int WM = BM <= 32 ? 16 : 32, WN = BN <= 32 ? 16 : 32;
  static constexpr int WARPS_M = BM / WM, WARPS_N = BN / WN;
  static constexpr int THREADS = WARPS_M * WARPS_N * 32;
  static constexpr int BK = 16, STAGES = 3;
  static constexpr int AP = BM + 4, BP = BN + 4;    // pitches: conflict-free fragment loads
  static constexpr size_t SMEM = (size_t)STAGES * BK * (AP + BP) * sizeof(double) +
                                 (size_t)(2 * BM + 2 * BN + 2 * kKRing * BK) * sizeof(int64_t);
};

// k-offset tables of the k-tiles in flight live in a shared ring (slot t % 4
// holds tile t's BK entries of kL and kR, k counted from the split's first).
// Tiles 0..ST are fetched before the main loop; iteration t copies tile
// t+ST+1's entries asynchronously with its own load group, two iterations
// before the loads that use them, so neither an address nor an iteration waits
// for a table read (fetched through registers one iteration ahead, the reads'
// latency bounded every k step of thin tiles).
template <int BK, int ST>
__device__ __forceinline__ void kring_init(const int64_t *kL, const int64_t *kR, int K, int64_t *kLs, int64_t *kRs,
                                           int tid, int nt) {
  static_assert(ST + 1 <= kKRing, "prefetched tiles fit the ring");
  for (int i = tid; i < (ST + 1) * BK; i += nt) {
    kLs[i] = i < K ? kL[i] : 0;
    kRs[i] = i < K ? kR[i] : 0;
  }
}
// The copies of one warp: lane l < BK the kL entries of a tile, the others kR's.
template <int BK, int ST>
struct KRing {
  static_assert(2 * BK == 32, "one warp copies both tables of a tile");
  const int64_t *from;
  uint32_t to;
  __device__ __forceinline__ void init(const int64_t *kL, const int64_t *kR, int64_t *kLs, int64_t *kRs) {
    const int j = threadIdx.x % BK;
    from = (threadIdx.x % 32 < BK ? kL : kR) + j;
    to = (uint32_t)__cvta_generic_to_shared((threadIdx.x % 32 < BK ? kLs : kRs) + j);
  }
  __device__ __forceinline__ void step(int kt, int K) const {
    if (threadIdx.x < 32) {
      const int t = kt + ST + 1, k = t * BK;
      const int n = k + (int)(threadIdx.x % BK) < K ? 8 : 0;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(to + (t % kKRing) * (BK * 8)),
                   "l"(from + (n ? k : 0)), "r"(n));
    }
  }
};

// Column swizzle of the FP64 tiles: row k stores column c at c ^ ((k >> 2) & 3).
// With rows 8 banks apart (pitch BM + 4 doubles) a fragment load's four k-rows
// fill all 32 banks, and tile loads whose lanes run along k (the operand's
// stride-1 index is contracted) hit 16 different bank pairs per half-warp.
__device__ __forceinline__ int kswz(int k) { return (k >> 2) & 3; }

// Valid 8-row fragments of warp `w` of `W` along one tile dimension with `rem`
// rows left: fragment i of the warp covers rows (i W + w) 8.  Interleaving the
// warps' fragments spreads a ragged tile's valid ones over all warps.
__device__ __forceinline__ int frag_count(int rem, int w, int W, int F) {
  return max(0, min(F, (rem - w * 8 + 8 * W - 1) / (8 * W)));
}

// Shared-memory reads by 32-bit address, and the copy of one ES-byte element.
__device__ __forceinline__ int64_t lds64(uint32_t a) {
  int64_t v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}
template <int ES, bool TAIL>
__device__ __forceinline__ void cp_elem(uint32_t s, const char *g, bool v) {
  if constexpr (TAIL) {
    const int n = v ? ES : 0;
    if constexpr (ES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(g), "r"(n));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(s), "l"(g), "n"(ES), "r"(n));
  } else {
    if constexpr (ES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(g));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(g), "n"(ES));
  }
}

// One operand's k-tile loads: X free-index rows (`rem` of them inside the
// tensor) by BK k-rows, element (x, k) at G + fs[x] + ks[k] bytes and at column
// x (XOR kswz(k) if SWZ) of shared row k.  `along`: a thread keeps one free
// index and steps through k, its lanes along the free index; else it keeps one
// k and steps through the free index.  Everything that does not change with the
// k-tile is kept here, so an element costs an offset read, an add and the copy
// (with the index arithmetic in the loop, about 25 instructions per element
// bounded thin tiles and took issue slots from the tensor pipe in full ones).
template <int X, int BK, int NT, int PITCH, int ES, bool SWZ>
struct Side {
  static constexpr int N = X * BK / NT;    // elements per thread and k-tile
  static constexpr int W = 4;              // offsets read before the copies that use them: the reads
                                           // overlap instead of costing a shared-memory latency each
  static constexpr int SF = NT / X;        // k step of a thread along its free index
  static constexpr int SK = NT / BK;       // free-index step of a thread along its k
  static_assert(NT % X == 0 && NT % BK == 0 && X * BK % NT == 0, "whole elements per thread");
  static_assert(!SWZ || (SF <= 4 && 4 % SF == 0 && SK % 4 == 0), "the swizzle is constant per element slot");
  const char *g;   // along: the row's base, else the operand
  uint32_t s;      // shared address of the thread's first element in stage 0
  uint32_t u;      // along: column (swizzled per element); else shared address of its first row offset
  int k0, lim;     // first k-row; along: rows left (> 0: loads), else rows it may load
  bool along;

  __device__ __forceinline__ void init(const void *G, const int64_t *fs_, const void *stage0, bool along_, int rem) {
    const int tid = threadIdx.x;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(stage0);
    along = along_;
    if (along) {
      const int x0 = tid % X;
      k0 = tid / X;
      g = (const char *)G + fs_[x0];
      s = base + (uint32_t)(k0 * PITCH + (SWZ ? 0 : x0)) * ES;
      lim = rem - x0;
      u = (uint32_t)x0;
    } else {
      static_assert(N % W == 0, "whole groups of offset reads");
      const int x0 = tid / BK;
      k0 = tid % BK;
      g = (const char *)G;
      s = base + (uint32_t)(k0 * PITCH + (SWZ ? x0 ^ kswz(k0) : x0)) * ES;
      lim = rem - x0;
      u = (uint32_t)__cvta_generic_to_shared(fs_ + x0);
    }
  }
  // Loads of one k-tile: `so` bytes to its stage, k offsets at shared address
  // ks, k-rows from klim on zero-filled (TAIL).
  template <bool TAIL>
  __device__ __forceinline__ void load(uint32_t so, uint32_t ks, int klim) const {
    if (along) {
      if (lim <= 0) return;
#pragma unroll
      for (int i0 = 0; i0 < N; i0 += W) {
        int64_t o[W];
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] = lds64(ks + (k0 + (i0 + i) * SF) * 8);  // zero past the range
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const bool v = !TAIL || k0 + (i0 + i) * SF < klim;
          const uint32_t c = SWZ ? (u ^ kswz((i0 + i) * SF)) * ES : 0u;
          cp_elem<ES, TAIL>(s + so + c + (uint32_t)((i0 + i) * SF * PITCH * ES), g + o[i], v);
        }
      }
    } else {
      const bool v = !TAIL || k0 < klim;
      const char *gk = g + lds64(ks + k0 * 8);
#pragma unroll
      for (int i0 = 0; i0 < N; i0 += W) {
        int64_t o[W];
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] = lds64(u + (i0 + i) * SK * 8);
#pragma unroll
        for (int i = 0; i < W; ++i)
          if ((i0 + i) * SK < lim) cp_elem<ES, TAIL>(s + so + (uint32_t)((i0 + i) * SK * ES), gk + o[i], v);
      }
    }
  }
  __device__ __forceinline__ void load_tile(uint32_t so, uint32_t ks, int klim) const {
    if (klim >= BK) load<false>(so, ks, klim);
    else if (klim > 0) load<true>(so, ks, klim);
  }
};

// One BM x BN tile of a gather-GEMM (shared by the single-contraction kernel and
// the batched one) over the k range of its split.  The loads of the tile
// ST - 1 ahead are issued between the tensor-pipe steps (A's after the first,
// B's after the third): issued in one block after the barrier they left the
// pipe idle in every warp at once.  Rows and columns beyond the tensor are neither loaded (their stale
// shared values only reach outputs that are not stored) nor multiplied.
template <int BM, int BN, bool SEQ>
__device__ __forceinline__ void dmma_tile(const double *__restrict__ L, const double *__restrict__ R,
                                          double *D, const GemmArgs &a, const TileWork &w,
                                          unsigned char *smem) {
  using C = DmmaCfg<BM, BN>;
  constexpr int BK = C::BK, ST = C::STAGES, AP = C::AP, BP = C::BP, NT = C::THREADS;
  double *As = reinterpret_cast<double *>(smem);
  double *Bs = As + ST * BK * AP;
  int64_t *mLs = reinterpret_cast<int64_t *>(Bs + ST * BK * BP);
  int64_t *mDs = mLs + BM;
  int64_t *nRs = mDs + BM;
  int64_t *nDs = nRs + BN;
  int64_t *kLs = nDs + BN;
  int64_t *kRs = kLs + kKRing * BK;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = w.tm * BM, n0 = w.tn * BN;
  const int mrem = a.M - m0, nrem = a.N - n0;
  for (int i = tid; i < BM; i += NT) {
    const int m = m0 + i;
    mLs[i] = m < a.M ? a.mL[m] : 0;
    mDs[i] = m < a.M ? a.mD[m] : 0;
  }
  for (int i = tid; i < BN; i += NT) {
    const int n = n0 + i;
    nRs[i] = n < a.N ? a.nR[n] : 0;
    nDs[i] = n < a.N ? a.nD[n] : 0;
  }
  using Int0 = std::integral_constant<int, 0>;
  using Int1 = std::integral_constant<int, 1>;
  using Int2 = std::integral_constant<int, 2>;
  using Int3 = std::integral_constant<int, 3>;
  constexpr int FM = C::WM / 8, FN = C::WN / 8;
  double2 acc[FM * FN];
  // Ragged tiles give the low warp positions more fragments; the positions turn
  // with the CTA's number.  CTAs of one launch that share an SM are mostly a
  // multiple of 148 = 4 x 37 apart and turn alike, so little comes of it: 40 x 40
  // outputs 167.4 -> 165.7 us, batch of 768 4324 -> 4302.  (Turning by the number
  // over 148 as well, 162 -> 177 us, was not kept.)
  const int wr = (warp + w.lin + w.split) % (C::WARPS_M * C::WARPS_N);
  const int wm = wr % C::WARPS_M, wn = wr / C::WARPS_M;
  const int fr = lane >> 2, fc = lane & 3;
  const int fm = frag_count(mrem, wm, C::WARPS_M, FM), fn = frag_count(nrem, wn, C::WARPS_N, FN);
  SeqSum<FM * FN, double2> seq;
  for (int split = SEQ ? 0 : w.split;; ++split) {
    const int k0 = a.nsplit > 1 ? split * a.kchunk : 0;
    const int K = a.nsplit > 1 ? min(a.kchunk, a.K - k0) : a.K;
    const int64_t *kLg = a.kL + k0, *kRg = a.kR + k0;
#pragma unroll
    for (int f = 0; f < FM * FN; ++f) acc[f] = make_double2(0.0, 0.0);
    kring_init<BK, ST>(kLg, kRg, K, kLs, kRs, tid, NT);
    __syncthreads();

    const int numK = (K + BK - 1) / BK;
    Side<BM, BK, NT, AP, 8, true> sa;
    Side<BN, BK, NT, BP, 8, true> sb;
    sa.init(L, mLs, As, a.a_along_m, mrem);
    sb.init(R, nRs, Bs, a.b_along_n, nrem);
    constexpr uint32_t SAB = BK * AP * 8, SBB = BK * BP * 8;  // bytes per stage
    KRing<BK, ST> ring;
    ring.init(kLg, kRg, kLs, kRs);
    const uint32_t ksa = (uint32_t)__cvta_generic_to_shared(kLs), ksb = (uint32_t)__cvta_generic_to_shared(kRs);
    auto load_a = [&](int kt, int s) { sa.load_tile(s * SAB, ksa + (kt % kKRing) * (BK * 8), K - kt * BK); };
    auto load_b = [&](int kt, int s) { sb.load_tile(s * SBB, ksb + (kt % kKRing) * (BK * 8), K - kt * BK); };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
      load_a(s, s);
      load_b(s, s);
      cp_async_commit();
    }
    auto main_loop = [&](auto full_c) {
      constexpr bool FULL = decltype(full_c)::value;
      int st = 0, ps = ST - 1;  // stage of tile kt, stage filled during iteration kt
      for (int kt = 0; kt < numK; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        const double *as = As + (st * BK + fc) * AP + wm * 8;
        const double *bs = Bs + (st * BK + fc) * BP + wn * 8;
        auto step = [&](auto ksc) {
          constexpr int ks = decltype(ksc)::value;
          double af[FM], bf[FN];
          const double *ap = as + (fr ^ ks), *bp = bs + (fr ^ ks);  // kswz(4 ks + fc) = ks
#pragma unroll
          for (int i = 0; i < FM; ++i) af[i] = ap[ks * 4 * AP + i * C::WARPS_M * 8];
#pragma unroll
          for (int j = 0; j < FN; ++j) bf[j] = bp[ks * 4 * BP + j * C::WARPS_N * 8];
#pragma unroll
          for (int i = 0; i < FM; ++i) {
            if (!FULL && i >= fm) break;
#pragma unroll
            for (int j = 0; j < FN; ++j)
              if (FULL || j < fn) dmma_8x8x4(acc[i * FN + j].x, acc[i * FN + j].y, af[i], bf[j]);
          }
          if constexpr (ks == 0) load_a(kt + ST - 1, ps);
          if constexpr (ks == 2) load_b(kt + ST - 1, ps);
        };
        step(Int0{});
        step(Int1{});
        step(Int2{});
        step(Int3{});
        ring.step(kt, K);
        cp_async_commit();
        ps = st;
        st = st + 1 == ST ? 0 : st + 1;
      }
    };
    if (fm == FM && fn == FN) main_loop(std::true_type{});
    else main_loop(std::false_type{});
    cp_async_wait<0>();
    if constexpr (!SEQ) break;
    seq.add(acc, a, split);
    if (split + 1 == a.nsplit) break;
    __syncthreads();  // the next split refills the stages and the offset ring
  }

  if constexpr (SEQ) {
#pragma unroll
    for (int f = 0; f < FM * FN; ++f) acc[f] = seq.total[f];
  }
  if (!SEQ && a.nsplit > 1) {
    uint32_t mask = 0;
#pragma unroll
    for (int f = 0; f < FM * FN; ++f)
      if (f / FN < fm && f % FN < fn) mask |= 1u << f;
    if (!split_combine<FM * FN, NT>(acc, mask, wr * 32 + lane, a, w.lin, w.split)) return;
  }
  // Epilogue: the D values of a fragment row are all loaded before any is
  // stored (the compiler cannot move a load above a store that may alias it).
  const double alpha = a.alpha_re;
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    const int ml = (i * C::WARPS_M + wm) * 8 + fr;
    if (ml >= mrem) continue;
    double *p[FN * 2];
    double d[FN * 2];
#pragma unroll
    for (int j = 0; j < FN * 2; ++j) {
      const int nl = ((j / 2) * C::WARPS_N + wn) * 8 + fc * 2 + (j & 1);
      p[j] = nl < nrem ? D + mDs[ml] + nDs[nl] : nullptr;
      d[j] = (a.beta && p[j]) ? *p[j] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < FN * 2; ++j) {
      const double v = (j & 1) ? acc[i * FN + j / 2].y : acc[i * FN + j / 2].x;
      if (p[j]) *p[j] = a.beta ? fma(alpha, v, d[j]) : alpha * v;
    }
  }
}

// Trip count (0 or 1) of a block that skips the four DMMAs of a fragment beyond
// a ragged tile.  Written as a loop whose count the compiler cannot see: a plain
// `if` becomes predication, and a predicated-off DMMA still takes its turn on
// the tensor pipe (batch of 768: 5105 -> 4907 us).  The real tile, with one DMMA
// per fragment, keeps the `if`: there the branches cost more (167 -> 187 us for
// a 40 x 40 output).
__device__ __forceinline__ int one_if(bool c) {
  int n = c ? 1 : 0;
  asm volatile("" : "+r"(n));
  return n;
}

// Complex-double tile on the FP64 tensor pipe: complex elements stay
// interleaved in shared memory (one 16-byte cp.async per element, one 128-bit
// load per fragment element), and
// C_re += A_re B_re + A_im (-B_im), C_im += A_re B_im + A_im B_re run as four
// DMMA products.  Row pitches of BM + 2 elements put the four k-rows of a
// fragment load in different bank groups.
// Warp tiles are 32 x 16 (16 x 16 in 32x32 CTA tiles): two accumulator sets
// (real, imaginary) per fragment.
template <int BM, int BN>
struct ZmmaCfg {
  static constexpr int WM = BM <= 32 ? 16 : 32, WN = 16;
  static constexpr int WARPS_M = BM / WM, WARPS_N = BN / WN;
  static constexpr int THREADS = WARPS_M * WARPS_N * 32;
  static constexpr int BK = 16, STAGES = BM <= 32 ? 2 : 3;  // two stages keep five small CTAs per SM
  static constexpr int AP = BM + 2, BP = BN + 2;           // in complex elements
  static constexpr size_t SMEM = (size_t)STAGES * BK * (AP + BP) * sizeof(double2) +
                                 (size_t)(2 * BM + 2 * BN + 2 * kKRing * BK) * sizeof(int64_t);
};

template <int BM, int BN, bool SEQ>
__device__ __forceinline__ void zmma_tile(const double2 *__restrict__ L, const double2 *__restrict__ R,
                                          double2 *D, const GemmArgs &a, const TileWork &w,
                                          unsigned char *smem) {
  using C = ZmmaCfg<BM, BN>;
  constexpr int BK = C::BK, ST = C::STAGES, AP = C::AP, BP = C::BP, NT = C::THREADS;
  double2 *As = reinterpret_cast<double2 *>(smem);
  double2 *Bs = As + ST * BK * AP;
  int64_t *mLs = reinterpret_cast<int64_t *>(Bs + ST * BK * BP);
  int64_t *mDs = mLs + BM;
  int64_t *nRs = mDs + BM;
  int64_t *nDs = nRs + BN;
  int64_t *kLs = nDs + BN;
  int64_t *kRs = kLs + kKRing * BK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = w.tm * BM, n0 = w.tn * BN;
  const int mrem = a.M - m0, nrem = a.N - n0;
  for (int i = tid; i < BM; i += NT) {
    const int m = m0 + i;
    mLs[i] = m < a.M ? a.mL[m] : 0;
    mDs[i] = m < a.M ? a.mD[m] : 0;
  }
  for (int i = tid; i < BN; i += NT) {
    const int n = n0 + i;
    nRs[i] = n < a.N ? a.nR[n] : 0;
    nDs[i] = n < a.N ? a.nD[n] : 0;
  }
  using Int0 = std::integral_constant<int, 0>;
  using Int1 = std::integral_constant<int, 1>;
  using Int2 = std::integral_constant<int, 2>;
  using Int3 = std::integral_constant<int, 3>;
  constexpr int FM = C::WM / 8, FN = C::WN / 8;
  double2 acc[2 * FM * FN];  // fragment f: real parts at 2 f, imaginary parts at 2 f + 1
  // Warp positions turn with the CTA's number, as in the real tile.
  const int wr = (warp + w.lin + w.split) % (C::WARPS_M * C::WARPS_N);
  const int wm = wr % C::WARPS_M, wn = wr / C::WARPS_M;
  const int fr = lane >> 2, fc = lane & 3;
  const int fm = frag_count(mrem, wm, C::WARPS_M, FM), fn = frag_count(nrem, wn, C::WARPS_N, FN);
  // conjugation flips the sign bit of the imaginary part
  const int ml = a.conj_l ? (int)0x80000000 : 0, mr = a.conj_r ? (int)0x80000000 : 0;
  auto flip = [](double x, int m) { return __hiloint2double(__double2hiint(x) ^ m, __double2loint(x)); };
  SeqSum<2 * FM * FN, double2> seq;
  for (int split = SEQ ? 0 : w.split;; ++split) {
    const int k0 = a.nsplit > 1 ? split * a.kchunk : 0;
    const int K = a.nsplit > 1 ? min(a.kchunk, a.K - k0) : a.K;
    const int64_t *kLg = a.kL + k0, *kRg = a.kR + k0;
#pragma unroll
    for (int f = 0; f < 2 * FM * FN; ++f) acc[f] = make_double2(0.0, 0.0);
    kring_init<BK, ST>(kLg, kRg, K, kLs, kRs, tid, NT);
    __syncthreads();
    const int numK = (K + BK - 1) / BK;
    Side<BM, BK, NT, AP, 16, false> sa;
    Side<BN, BK, NT, BP, 16, false> sb;
    sa.init(L, mLs, As, a.a_along_m, mrem);
    sb.init(R, nRs, Bs, a.b_along_n, nrem);
    constexpr uint32_t SAB = BK * AP * 16, SBB = BK * BP * 16;  // bytes per stage
    KRing<BK, ST> ring;
    ring.init(kLg, kRg, kLs, kRs);
    const uint32_t ksa = (uint32_t)__cvta_generic_to_shared(kLs), ksb = (uint32_t)__cvta_generic_to_shared(kRs);
    auto load_a = [&](int kt, int s) { sa.load_tile(s * SAB, ksa + (kt % kKRing) * (BK * 8), K - kt * BK); };
    auto load_b = [&](int kt, int s) { sb.load_tile(s * SBB, ksb + (kt % kKRing) * (BK * 8), K - kt * BK); };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
      load_a(s, s);
      load_b(s, s);
      cp_async_commit();
    }
    auto main_loop = [&](auto full_c) {
      constexpr bool FULL = decltype(full_c)::value;
      int st = 0, ps = ST - 1;
      for (int kt = 0; kt < numK; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        const double2 *as = As + (st * BK + fc) * AP + wm * 8 + fr;
        const double2 *bs = Bs + (st * BK + fc) * BP + wn * 8 + fr;
        auto step = [&](auto ksc) {
          constexpr int ks = decltype(ksc)::value;
          double ar[FM], ai[FM], br[FN], bi[FN], nbi[FN];
#pragma unroll
          for (int i = 0; i < FM; ++i) {
            const double2 v = as[ks * 4 * AP + i * C::WARPS_M * 8];
            ar[i] = v.x;
            ai[i] = flip(v.y, ml);
          }
#pragma unroll
          for (int j = 0; j < FN; ++j) {
            const double2 v = bs[ks * 4 * BP + j * C::WARPS_N * 8];
            br[j] = v.x;
            bi[j] = flip(v.y, mr);
            nbi[j] = -bi[j];
          }
#pragma unroll
          for (int i = 0; i < FM; ++i) {
#pragma unroll
            for (int j = 0; j < FN; ++j) {
              double2 &cr = acc[2 * (i * FN + j)], &ci = acc[2 * (i * FN + j) + 1];
#pragma unroll 1
              for (int x = FULL ? 1 : one_if(i < fm && j < fn); x > 0; --x) {
                dmma_8x8x4(cr.x, cr.y, ar[i], br[j]);
                dmma_8x8x4(cr.x, cr.y, ai[i], nbi[j]);
                dmma_8x8x4(ci.x, ci.y, ar[i], bi[j]);
                dmma_8x8x4(ci.x, ci.y, ai[i], br[j]);
              }
            }
          }
          if constexpr (ks == 0) load_a(kt + ST - 1, ps);
          if constexpr (ks == 2) load_b(kt + ST - 1, ps);
        };
        step(Int0{});
        step(Int1{});
        step(Int2{});
        step(Int3{});
        ring.step(kt, K);
        cp_async_commit();
        ps = st;
        st = st + 1 == ST ? 0 : st + 1;
      }
    };
    if (fm == FM && fn == FN) main_loop(std::true_type{});
    else main_loop(std::false_type{});
    cp_async_wait<0>();
    if constexpr (!SEQ) break;
    seq.add(acc, a, split);
    if (split + 1 == a.nsplit) break;
    __syncthreads();
  }
  if constexpr (SEQ) {
#pragma unroll
    for (int f = 0; f < 2 * FM * FN; ++f) acc[f] = seq.total[f];
  }
  if (!SEQ && a.nsplit > 1) {
    uint32_t mask = 0;
#pragma unroll
    for (int f = 0; f < FM * FN; ++f)
      if (f / FN < fm && f % FN < fn) mask |= 3u << (2 * f);
    if (!split_combine<2 * FM * FN, NT>(acc, mask, wr * 32 + lane, a, w.lin, w.split)) return;
  }
  const double alr = a.alpha_re, ali = a.alpha_im;
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    const int ml = (i * C::WARPS_M + wm) * 8 + fr;
    if (ml >= mrem) continue;
    double2 *p[FN * 2];
    double2 d[FN * 2];
#pragma unroll
    for (int j = 0; j < FN * 2; ++j) {
      const int nl = ((j / 2) * C::WARPS_N + wn) * 8 + fc * 2 + (j & 1);
      p[j] = nl < nrem ? D + mDs[ml] + nDs[nl] : nullptr;
      d[j] = (a.beta && p[j]) ? *p[j] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < FN * 2; ++j) {
      const double2 fr2 = acc[2 * (i * FN + j / 2)], fi2 = acc[2 * (i * FN + j / 2) + 1];
      const double cr = (j & 1) ? fr2.y : fr2.x, ci = (j & 1) ? fi2.y : fi2.x;
      const double vr = cr * alr - ci * ali;
      const double vi = cr * ali + ci * alr;
      if (p[j]) *p[j] = a.beta ? make_double2(d[j].x + vr, d[j].y + vi) : make_double2(vr, vi);
    }
  }
}

// Resident CTAs per SM asked of the compiler.
template <int BM, int BN> struct GemmOcc { static constexpr int D = 1, Z = 1; };
template <> struct GemmOcc<64, 64> { static constexpr int D = 4, Z = 2; };
template <> struct GemmOcc<32, 32> { static constexpr int D = 6, Z = 5; };

template <int BM, int BN, bool SEQ>
__global__ void __launch_bounds__(ZmmaCfg<BM, BN>::THREADS, SEQ ? 1 : GemmOcc<BM, BN>::Z)
    zgemm_gather_kernel(const double2 *__restrict__ L, const double2 *__restrict__ R, double2 *D,
                        const GemmArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const double2 *Lp = L, *Rp = R;
  double2 *Dp = D;
  const TileWork w = block_work(a, Lp, Rp, Dp);
  zmma_tile<BM, BN, SEQ>(Lp, Rp, Dp, a, w, smem);
}

template <int BM, int BN, bool SEQ>
__global__ void __launch_bounds__(DmmaCfg<BM, BN>::THREADS, SEQ ? 1 : GemmOcc<BM, BN>::D)
    dgemm_gather_kernel(const double *__restrict__ L, const double *__restrict__ R, double *D,
                        const GemmArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const double *Lp = L, *Rp = R;
  double *Dp = D;
  const TileWork w = block_work(a, Lp, Rp, Dp);
  dmma_tile<BM, BN, SEQ>(Lp, Rp, Dp, a, w, smem);
}

// ------------------------------------------------- R4 / C4: packed FP32 FMA
// Bound by the FP32 pipe (74 TFLOP/s nominal).  The packed form
// fma.rn.f32x2 does two FMAs per instruction, so a k step of a thread's
// sub-tile leaves issue slots for its shared-memory reads and for the tile
// loads, which are the asynchronous gathers of the FP64 kernels (Side).  Each
// accumulator is one chain of FMAs in k order, whatever the tile.
__device__ __forceinline__ void ffma2(uint64_t &c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// A thread's sub-tile: MC x NC blocks of VE x VE elements (VE elements per
// 16-byte shared read); block (c, d) covers rows c TMN VE + tm VE + 0..VE-1.
template <typename T, int BM, int BN>
struct FmmaCfg {
  static constexpr int VE = 16 / (int)sizeof(T);
  static constexpr int MC = (sizeof(T) == 4 ? 2 : 4) / (BM <= 32 ? 2 : 1), NC = sizeof(T) == 4 && BN <= 32 ? 1 : 2;
  static constexpr int TMN = BM / (MC * VE), TNN = BN / (NC * VE);  // threads along m and n
  static constexpr int THREADS = TMN * TNN;
  static constexpr int BK = 16, STAGES = 3;
  static constexpr int AP = BM + VE, BP = BN + VE;
  static constexpr size_t SMEM = (size_t)STAGES * BK * (AP + BP) * sizeof(T) +
                                 (size_t)(2 * BM + 2 * BN + 2 * kKRing * BK) * sizeof(int64_t);
};

template <typename T, int BM, int BN, bool SEQ>
__device__ __forceinline__ void fmma_tile(const T *__restrict__ L, const T *__restrict__ R, T *D, const GemmArgs &a,
                                          const TileWork &w, unsigned char *smem) {
  using C = FmmaCfg<T, BM, BN>;
  constexpr int BK = C::BK, ST = C::STAGES, AP = C::AP, BP = C::BP, NT = C::THREADS, VE = C::VE;
  constexpr int TM = C::MC * VE, TN = C::NC * VE, ES = (int)sizeof(T);
  constexpr bool CPLX = sizeof(T) == 8;
  T *As = reinterpret_cast<T *>(smem);
  T *Bs = As + ST * BK * AP;
  int64_t *mLs = reinterpret_cast<int64_t *>(Bs + ST * BK * BP);
  int64_t *mDs = mLs + BM;
  int64_t *nRs = mDs + BM;
  int64_t *nDs = nRs + BN;
  int64_t *kLs = nDs + BN;
  int64_t *kRs = kLs + kKRing * BK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = w.tm * BM, n0 = w.tn * BN;
  const int mrem = a.M - m0, nrem = a.N - n0;
  for (int i = tid; i < BM; i += NT) {
    const int m = m0 + i;
    mLs[i] = m < a.M ? a.mL[m] : 0;
    mDs[i] = m < a.M ? a.mD[m] : 0;
  }
  for (int i = tid; i < BN; i += NT) {
    const int n = n0 + i;
    nRs[i] = n < a.N ? a.nR[n] : 0;
    nDs[i] = n < a.N ? a.nD[n] : 0;
  }
  const int tm = (lane & 3) + 4 * (warp % (C::TMN / 4)), tn = (lane >> 2) + 8 * (warp / (C::TMN / 4));
  // Accumulator pairs.  Complex: acc[i][j] is element (i, j), (re, im).  Real:
  // a pair of rows meets a pair of columns as they come from shared memory, and
  // the pair of columns swapped: for rows i, i+1 and columns j, j+1 (all even i,
  // j) acc[i][j/2] = (c(i,j), c(i+1,j+1)) and acc[i+1][j/2] = (c(i,j+1), c(i+1,j)).
  // That costs one swap per column pair where pairs of equal row values would
  // cost two moves per row.
  constexpr int NP = CPLX ? TN : TN / 2;
  uint64_t acc[TM][NP];
  const uint32_t cl = a.conj_l ? 0x80000000u : 0u, cr = a.conj_r ? 0x80000000u : 0u;
  constexpr int NF = TM * NP / 2;  // 16-byte units: two accumulator pairs of a row
  auto to_units = [&](float4(&u)[NF]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int i = f / (NP / 2), j = f % (NP / 2);
      const float2 x = unpack2(acc[i][2 * j]), y = unpack2(acc[i][2 * j + 1]);
      u[f] = make_float4(x.x, x.y, y.x, y.y);
    }
  };
  auto from_units = [&](const float4(&u)[NF]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const int i = f / (NP / 2), j = f % (NP / 2);
      acc[i][2 * j] = pack2(u[f].x, u[f].y);
      acc[i][2 * j + 1] = pack2(u[f].z, u[f].w);
    }
  };
  SeqSum<NF, float4> seq;
  for (int split = SEQ ? 0 : w.split;; ++split) {
    const int k0 = a.nsplit > 1 ? split * a.kchunk : 0;
    const int K = a.nsplit > 1 ? min(a.kchunk, a.K - k0) : a.K;
    const int64_t *kLg = a.kL + k0, *kRg = a.kR + k0;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < NP; ++j) acc[i][j] = 0;
    kring_init<BK, ST>(kLg, kRg, K, kLs, kRs, tid, NT);
    __syncthreads();
    const int numK = (K + BK - 1) / BK;
    Side<BM, BK, NT, AP, ES, false> sa;
    Side<BN, BK, NT, BP, ES, false> sb;
    sa.init(L, mLs, As, a.a_along_m, mrem);
    sb.init(R, nRs, Bs, a.b_along_n, nrem);
    constexpr uint32_t SAB = BK * AP * ES, SBB = BK * BP * ES;
    KRing<BK, ST> ring;
    ring.init(kLg, kRg, kLs, kRs);
    const uint32_t ksa = (uint32_t)__cvta_generic_to_shared(kLs), ksb = (uint32_t)__cvta_generic_to_shared(kRs);
    auto load_a = [&](int kt, int s) { sa.load_tile(s * SAB, ksa + (kt % kKRing) * (BK * 8), K - kt * BK); };
    auto load_b = [&](int kt, int s) { sb.load_tile(s * SBB, ksb + (kt % kKRing) * (BK * 8), K - kt * BK); };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
      load_a(s, s);
      load_b(s, s);
      cp_async_commit();
    }
    int st = 0, ps = ST - 1;
    for (int kt = 0; kt < numK; ++kt) {
      cp_async_wait<ST - 2>();
      __syncthreads();
      const T *as = As + st * BK * AP + tm * VE;
      const T *bs = Bs + st * BK * BP + tn * VE;
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        uint64_t av[C::MC * 2], bv[C::NC * 2];
#pragma unroll
        for (int c = 0; c < C::MC; ++c) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(as + k * AP + c * (C::TMN * VE));
          av[2 * c] = v.x;
          av[2 * c + 1] = v.y;
        }
#pragma unroll
        for (int c = 0; c < C::NC; ++c) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(bs + k * BP + c * (C::TNN * VE));
          bv[2 * c] = v.x;
          bv[2 * c + 1] = v.y;
        }
        if constexpr (CPLX) {
          // (re, im) += x.re (y.re, y.im), then += x.im (-y.im, y.re)
          uint64_t by[TN], bx[TN];
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const float2 y = unpack2(bv[j]);
            const float yi = __uint_as_float(__float_as_uint(y.y) ^ cr);
            by[j] = pack2(y.x, yi);
            bx[j] = pack2(-yi, y.x);
          }
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            const float2 x = unpack2(av[i]);
            const float xi = __uint_as_float(__float_as_uint(x.y) ^ cl);
            const uint64_t xr2 = pack2(x.x, x.x), xi2 = pack2(xi, xi);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              ffma2(acc[i][j], xr2, by[j]);
              ffma2(acc[i][j], xi2, bx[j]);
            }
          }
        } else {
          uint64_t bs2[NP];
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            const float2 y = unpack2(bv[j]);
            bs2[j] = pack2(y.y, y.x);
          }
#pragma unroll
          for (int i = 0; i < TM; i += 2)
#pragma unroll
            for (int j = 0; j < NP; ++j) {
              ffma2(acc[i][j], av[i / 2], bv[j]);
              ffma2(acc[i + 1][j], av[i / 2], bs2[j]);
            }
        }
        if (k == 1) load_a(kt + ST - 1, ps);
        if (k == BK / 2 + 1) load_b(kt + ST - 1, ps);
      }
      ring.step(kt, K);
      cp_async_commit();
      ps = st;
      st = st + 1 == ST ? 0 : st + 1;
    }
    cp_async_wait<0>();

    if constexpr (!CPLX) {  // back to rows: acc[i][j/2] = (c(i,j), c(i,j+1))
#pragma unroll
      for (int i = 0; i < TM; i += 2)
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          const float2 d = unpack2(acc[i][j]), x = unpack2(acc[i + 1][j]);
          acc[i][j] = pack2(d.x, x.x);
          acc[i + 1][j] = pack2(x.y, d.y);
        }
    }
    if constexpr (!SEQ) break;
    float4 u[NF];
    to_units(u);
    seq.add(u, a, split);
    if (split + 1 == a.nsplit) break;
    __syncthreads();
  }
  if constexpr (SEQ) from_units(seq.total);
  auto row_of = [&](int i) { return (i / VE) * (C::TMN * VE) + tm * VE + i % VE; };
  auto col_of = [&](int j) { return (j / VE) * (C::TNN * VE) + tn * VE + j % VE; };
  if (!SEQ && a.nsplit > 1) {
    float4 part[NF];
    uint32_t mask = 0;
    to_units(part);
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if (row_of(f / (NP / 2)) < mrem && col_of(f % (NP / 2) * (TN * 2 / NP)) < nrem) mask |= 1u << f;
    if (!split_combine<NF, NT>(part, mask, tid, a, w.lin, w.split)) return;
    from_units(part);
  }
  // Epilogue through the stage buffers, so that the lanes of a warp meet D along
  // its neighbours: straight from the sub-tiles a store filled half of each sector
  // it touched, which showed where D is most of the traffic (R4, us: outer product
  // 3000 x 1001 20.2 -> 16.5, 3000 x 3000 at K = 16 42 -> 31, 131000 x 64 at K = 30
  // 49 -> 35; 3249 x 576 x 3249 307 -> 304).
  constexpr int CP = BM + VE;                                       // column pitch
  constexpr int CW = BN * CP <= ST * BK * (AP + BP) ? BN : BN / 2;  // columns per part
  static_assert(CW * CP <= ST * BK * (AP + BP) && C::TNN * VE <= CW && NT % BM == 0 && NT % CW == 0, "parts fit the stages");
  T *Cs = As;
  const float alr = (float)a.alpha_re, ali = (float)a.alpha_im;
  const bool along_n = nrem > 1 && (mrem <= 1 || nDs[1] - nDs[0] < mDs[1] - mDs[0]);
  auto emit = [&](T c, T d) {
    if constexpr (CPLX) {
      const float vr = c.x * alr - c.y * ali, vi = c.x * ali + c.y * alr;
      return a.beta ? make_float2(d.x + vr, d.y + vi) : make_float2(vr, vi);
    } else {
      const float v = c * alr;
      return a.beta ? d + v : v;
    }
  };
#pragma unroll
  for (int c0 = 0; c0 < BN; c0 += CW) {
    __syncthreads();  // every warp is done with the stages, or with the part before
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      if ((j / VE) * (C::TNN * VE) / CW != c0 / CW) continue;
#pragma unroll
      for (int i = 0; i < TM; i += VE) {
        T *to = Cs + (col_of(j) - c0) * CP + row_of(i);
        if constexpr (CPLX) {
          *reinterpret_cast<ulonglong2 *>(to) = make_ulonglong2(acc[i][j], acc[i + 1][j]);
        } else {
          float4 v;
          float *e = &v.x;
#pragma unroll
          for (int q = 0; q < VE; ++q) {
            const float2 c = unpack2(acc[i + q][j / 2]);
            e[q] = (j & 1) ? c.y : c.x;
          }
          *reinterpret_cast<float4 *>(to) = v;
        }
      }
    }
    __syncthreads();
    const int cols = min(CW, nrem - c0);
    constexpr int U = 8;
    if (!along_n) {
      const int row = tid % BM;
      if (row < mrem) {
        T *dm = D + mDs[row];
        for (int c = tid / BM; c < cols; c += U * (NT / BM)) {
          T d[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int n = c + u * (NT / BM);
            d[u] = a.beta && n < cols ? dm[nDs[c0 + n]] : T();
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int n = c + u * (NT / BM);
            if (n < cols) dm[nDs[c0 + n]] = emit(Cs[n * CP + row], d[u]);
          }
        }
      }
    } else {
      const int n = tid % CW;
      if (n < cols) {
        T *dn = D + nDs[c0 + n];
        const int rows = min(BM, mrem);
        for (int r = tid / CW; r < rows; r += U * (NT / CW)) {
          T d[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int m = r + u * (NT / CW);
            d[u] = a.beta && m < rows ? dn[mDs[m]] : T();
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int m = r + u * (NT / CW);
            if (m < rows) dn[mDs[m]] = emit(Cs[n * CP + m], d[u]);
          }
        }
      }
    }
  }
}

// Resident CTAs per SM asked of the compiler.
template <typename T, int BM> struct FmmaOcc { static constexpr int N = 4; };
template <> struct FmmaOcc<float, 64> { static constexpr int N = 6; };  // 7: 5 % slower (spills)
template <> struct FmmaOcc<float, 128> { static constexpr int N = 2; };
template <> struct FmmaOcc<float, 32> { static constexpr int N = 16; };
template <> struct FmmaOcc<float2, 32> { static constexpr int N = 8; };

template <typename T, int BM, int BN, bool SEQ>
__global__ void __launch_bounds__(FmmaCfg<T, BM, BN>::THREADS, SEQ ? 1 : FmmaOcc<T, BM>::N)
    fgemm_gather_kernel(const T *__restrict__ L, const T *__restrict__ R, T *D, const GemmArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const T *Lp = L, *Rp = R;
  T *Dp = D;
  const TileWork w = block_work(a, Lp, Rp, Dp);
  fmma_tile<T, BM, BN, SEQ>(Lp, Rp, Dp, a, w, smem);
}

// ------------------------------------------------------ full contraction
constexpr int kDotThreads = 256;

__device__ __forceinline__ double2 warp_sum2(double2 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_down_sync(0xffffffffu, v.x, o);
    v.y += __shfl_down_sync(0xffffffffu, v.y, o);
  }
  return v;
}
__device__ double2 block_sum2(double2 v) {
  __shared__ double2 ws[kDotThreads / 32];
  v = warp_sum2(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) ws[warp] = v;
  __syncthreads();
  double2 r = make_double2(0.0, 0.0);
  if (warp == 0) {
    r = (lane < kDotThreads / 32) ? ws[lane] : make_double2(0.0, 0.0);
    r = warp_sum2(r);
  }
  return r;
}

template <typename T> __device__ __forceinline__ double2 as_c(const T &x, bool cj);
template <> __device__ __forceinline__ double2 as_c<float>(const float &x, bool) { return make_double2(x, 0.0); }
template <> __device__ __forceinline__ double2 as_c<double>(const double &x, bool) { return make_double2(x, 0.0); }
template <> __device__ __forceinline__ double2 as_c<float2>(const float2 &x, bool cj) { return make_double2(x.x, cj ? -x.y : x.y); }
template <> __device__ __forceinline__ double2 as_c<double2>(const double2 &x, bool cj) { return make_double2(x.x, cj ? -x.y : x.y); }

template <typename T> __device__ __forceinline__ void store_c(T *p, double2 v);
template <> __device__ __forceinline__ void store_c<float>(float *p, double2 v) { *p = (float)v.x; }
template <> __device__ __forceinline__ void store_c<double>(double *p, double2 v) { *p = v.x; }
template <> __device__ __forceinline__ void store_c<float2>(float2 *p, double2 v) { *p = make_float2((float)v.x, (float)v.y); }
template <> __device__ __forceinline__ void store_c<double2>(double2 *p, double2 v) { *p = v; }

template <typename T>
__global__ void __launch_bounds__(kDotThreads)
    dot_partial_kernel(const T *__restrict__ L, const T *__restrict__ R, const int64_t *kL,
                       const int64_t *kR, int64_t K, int64_t chunk, int cl, int cr, double2 *part) {
  const int64_t beg = (int64_t)blockIdx.x * chunk, end = min(K, beg + chunk);
  double2 acc = make_double2(0.0, 0.0);
  for (int64_t k = beg + threadIdx.x; k < end; k += kDotThreads) {
    const double2 x = as_c<T>(*(const T *)((const char *)L + kL[k]), cl);
    const double2 y = as_c<T>(*(const T *)((const char *)R + kR[k]), cr);
    acc.x += x.x * y.x - x.y * y.y;
    acc.y += x.x * y.y + x.y * y.x;
  }
  const double2 s = block_sum2(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

template <typename T>
__global__ void __launch_bounds__(kDotThreads)
    dot_final_kernel(const double2 *part, int n, T *D, double ar, double ai, int beta) {
  double2 acc = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < n; i += kDotThreads) { acc.x += part[i].x; acc.y += part[i].y; }
  const double2 s = block_sum2(acc);
  if (threadIdx.x == 0) {
    double2 v = make_double2(s.x * ar - s.y * ai, s.x * ai + s.y * ar);
    if (beta) {
      const double2 d = as_c<T>(*D, false);
      v.x += d.x;
      v.y += d.y;
    }
    store_c<T>(D, v);
  }
}

// scalar x scalar: d = (beta ? d : 0) + (l*r)*alpha in complex(8) arithmetic.
template <typename T>
__global__ void scalar_mul_kernel(const T *L, const T *R, T *D, double ar, double ai, int cl,
                                  int cr, int beta) {
  const double2 l = as_c<T>(*L, cl), r = as_c<T>(*R, cr);
  const double2 p = make_double2(l.x * r.x - l.y * r.y, l.x * r.y + l.y * r.x);
  double2 v = make_double2(p.x * ar - p.y * ai, p.x * ai + p.y * ar);
  if (beta) {
    const double2 d = as_c<T>(*D, false);
    v.x = d.x + v.x;
    v.y = d.y + v.y;
  }
  store_c<T>(D, v);
}

int dot_blocks(int64_t K) {
  int64_t b = (K + 16383) / 16384;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 1024));
}

struct Analysis {
  TableParams T;
  bool a_along_m = true, b_along_n = true;
  int hyper = 0;
};

int64_t align_up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

// Splits the pattern into m / n / k index groups with their strides.
int analyze(const int *cptrn, int drank, const int *ddims, int lrank, const int *ldims, int rrank,
            const int *rdims, Analysis &an) {
  TableParams &T = an.T;
  std::memset(&T, 0, sizeof(T));
  int64_t dstr[kMaxRank], lstr[kMaxRank], rstr[kMaxRank];
  int64_t s = 1;
  for (int i = 0; i < drank; ++i) { dstr[i] = s; s *= ddims[i]; }
  s = 1;
  for (int i = 0; i < lrank; ++i) { lstr[i] = s; s *= ldims[i]; }
  s = 1;
  for (int i = 0; i < rrank; ++i) { rstr[i] = s; s *= rdims[i]; }
  // Validation in the manner of the GPU path (reference :5934-5966).
  int dseen[kMaxRank] = {0}, lseen[kMaxRank] = {0}, rseen[kMaxRank] = {0};
  for (int i = 0; i < lrank; ++i) {
    const int j = cptrn[i];
    if (j > 0) {
      if (j > drank || ddims[j - 1] != ldims[i]) return TALSH_INVALID_ARGS;
      dseen[j - 1]++;
    } else if (j < 0) {
      if (-j > rrank || rdims[-j - 1] != ldims[i] || cptrn[lrank - j - 1] != -(i + 1)) return TALSH_INVALID_ARGS;
      if (rseen[-j - 1]++) return TALSH_INVALID_ARGS;
    } else {
      return TALSH_INVALID_ARGS;
    }
  }
  for (int i = 0; i < rrank; ++i) {
    const int j = cptrn[lrank + i];
    if (j > 0) {
      if (j > drank || ddims[j - 1] != rdims[i]) return TALSH_INVALID_ARGS;
      dseen[j - 1]++;
    } else if (j < 0) {
      if (-j > lrank || ldims[-j - 1] != rdims[i] || cptrn[-j - 1] != -(i + 1)) return TALSH_INVALID_ARGS;
      if (lseen[-j - 1]++) return TALSH_INVALID_ARGS;
    } else {
      return TALSH_INVALID_ARGS;
    }
  }
  for (int i = 0; i < drank; ++i) {
    if (dseen[i] == 2) an.hyper++;
    else if (dseen[i] != 1) return TALSH_INVALID_ARGS;
  }
  // h: indices in D, L and R, in L order (reference nhu groups,
  // tensor_algebra_cpu.F90:5829-5839).
  T.H = 1;
  for (int i = 0; i < lrank; ++i) {
    const int j = cptrn[i];
    if (j <= 0 || dseen[j - 1] != 2 || ldims[i] == 1) continue;
    int r = 0;
    while (r < rrank && cptrn[lrank + r] != j) ++r;
    if (r == rrank) return TALSH_INVALID_ARGS;
    if (T.nh >= kMaxGR) return TALSH_LIMIT_EXCEEDED;
    T.hext[T.nh] = ldims[i]; T.hstrL[T.nh] = lstr[i]; T.hstrR[T.nh] = rstr[r]; T.hstrD[T.nh] = dstr[j - 1];
    T.H *= ldims[i]; T.nh++;
  }
  int64_t lvol = 1, rvol = 1;
  for (int i = 0; i < lrank; ++i) lvol *= ldims[i];
  for (int i = 0; i < rrank; ++i) rvol *= rdims[i];
  // m: L uncontracted in L order; n: R uncontracted in R order.
  T.M = T.N = T.K = 1;
  for (int i = 0; i < lrank; ++i) {
    if (cptrn[i] > 0 && dseen[cptrn[i] - 1] == 1 && ldims[i] > 1) {
      if (T.nm >= kMaxGR) return TALSH_LIMIT_EXCEEDED;
      T.mext[T.nm] = ldims[i]; T.mstrL[T.nm] = lstr[i]; T.mstrD[T.nm] = dstr[cptrn[i] - 1];
      T.M *= ldims[i]; T.nm++;
    }
  }
  for (int i = 0; i < rrank; ++i) {
    if (cptrn[lrank + i] > 0 && dseen[cptrn[lrank + i] - 1] == 1 && rdims[i] > 1) {
      if (T.nn >= kMaxGR) return TALSH_LIMIT_EXCEEDED;
      T.next[T.nn] = rdims[i]; T.nstrR[T.nn] = rstr[i]; T.nstrD[T.nn] = dstr[cptrn[lrank + i] - 1];
      T.N *= rdims[i]; T.nn++;
    }
  }
  // k: follow R's order when R's leading index is contracted and L's is not
  // (or R is the larger operand), otherwise L's order.
  const bool l_lead_k = lrank > 0 && cptrn[0] < 0;
  const bool r_lead_k = rrank > 0 && cptrn[lrank] < 0;
  const bool k_in_r_order = r_lead_k && (!l_lead_k || rvol > lvol);
  if (k_in_r_order) {
    for (int i = 0; i < rrank; ++i) {
      const int j = cptrn[lrank + i];
      if (j < 0 && rdims[i] > 1) {
        if (T.nk >= kMaxGR) return TALSH_LIMIT_EXCEEDED;
        T.kext[T.nk] = rdims[i]; T.kstrR[T.nk] = rstr[i]; T.kstrL[T.nk] = lstr[-j - 1];
        T.K *= rdims[i]; T.nk++;
      }
    }
  } else {
    for (int i = 0; i < lrank; ++i) {
      const int j = cptrn[i];
      if (j < 0 && ldims[i] > 1) {
        if (T.nk >= kMaxGR) return TALSH_LIMIT_EXCEEDED;
        T.kext[T.nk] = ldims[i]; T.kstrL[T.nk] = lstr[i]; T.kstrR[T.nk] = rstr[-j - 1];
        T.K *= ldims[i]; T.nk++;
      }
    }
  }
  // Lane mapping for the tile loads: along the operand's stride-1 group.
  an.a_along_m = T.nm > 0 && (T.nk == 0 || T.mstrL[0] <= T.kstrL[0]);
  an.b_along_n = T.nn > 0 && (T.nk == 0 || T.nstrR[0] <= T.kstrR[0]);
  return TALSH_SUCCESS;
}

// Elements of one 64-row (or 64-column) tile that lie next to each other in a
// tensor: its stride-1 dimension as far as the tile covers it, and the next one
// where it is covered whole.  A group's dimension is covered as far as 64 rows
// reach past the dimensions before it; contracted dimensions are walked whole.
struct GroupView {
  int n;
  const int64_t *ext, *str;
  bool whole;
};
int64_t tile_run(const GroupView &a, const GroupView &b) {
  int64_t run = 1;
  for (;;) {
    int64_t covered = 0, extent = 0;
    for (const GroupView *g : {&a, &b}) {
      int64_t before = 1;
      for (int d = 0; d < g->n && before <= 64; ++d) {
        if (g->str[d] == run) {
          extent = g->ext[d];
          covered = g->whole ? extent : std::min(extent, 64 / before);
        }
        if (!g->whole) before *= g->ext[d];
      }
    }
    if (covered < 2) return run;
    run *= covered;
    if (covered < extent) return run;
  }
}

// Order of the free indices for the GEMM tiles.  `analyze` lists them in their
// operand's order, which makes that operand's loads contiguous when its
// stride-1 index is free, but may scatter D, whose sectors then cross the L2
// once per element, read and written.  Where the stride-1 index is contracted
// anyway, or K < 384 and D's fastest index belongs to the group but does not
// lead it, the group takes D's order if that moves fewer sectors: L is read
// ceil(N / 64) times, R ceil(M / 64) times, D read and written once, at es / 32
// sectors per element and about one more per run.  One sector of D weighs as
// much as `w` of an operand, fitted to where the two orders met on
// D(e,m,i) += L(m,k,e,c) R(c,k,i), 131328 x i outputs (us, operand's / D's order):
//   R8  i = 1:  44 / 65 at K = 20, 186 / 650 at 300;   8: 84 / 69, 217 / 660
//      24: 207 / 241 at 100;   64: 344 / 249 at 100, 453 / 660 at 300
//   R4  i = 8: 98 / 124 at 100;  64: 317 / 237 at 200, 355 / 355 at 300
//   C8  i = 8: 152 / 154 at 100, 290 / 353 at 300;  64: 848 / 692 at 300
//   C4  i = 8: 120 / 124 at 20;  64: 411 / 398 at 100, 573 / 699 at 200
// (K < 384 alone chose D's order in all of these).  Outputs wide both ways gain
// most: D(a,b,c,d) += L(e,b,a,d) R(c,e), 101 x 69 x 105 x 58, K = 51 in R4: 997
// -> 307 us; D(a,b,c,d,e,f) += L(d,e,g,a) R(g,f,b,c), 4608 x 4896 in R8: 728 ->
// 230 us at K = 64, 993 -> 776 at 300.  The order moves elements between tiles
// only: every element's sum is unchanged.
void order_by_output(Analysis &an, int es, bool cplx) {
  TableParams &T = an.T;
  auto smallest = [](const int64_t *str, int n) {
    int64_t s = INT64_MAX;
    for (int i = 0; i < n; ++i) s = std::min(s, str[i]);
    return s;
  };
  const int64_t dm = smallest(T.mstrD, T.nm), dn = smallest(T.nstrD, T.nn);
  const bool short_k = T.K < 384;
  const bool may_m = !an.a_along_m || (short_k && dm < dn && T.nm > 0 && T.mstrD[0] != dm);
  const bool may_n = !an.b_along_n || (short_k && dn < dm && T.nn > 0 && T.nstrD[0] != dn);
  if (!may_m && !may_n) return;
  struct Group {
    int64_t ext[kMaxGR], op[kMaxGR], d[kMaxGR];
  };
  auto take = [](Group &g, int n, const int64_t *ext, const int64_t *op, const int64_t *d, bool sorted) {
    for (int i = 0; i < n; ++i) {
      int j = i;
      for (; sorted && j > 0 && d[i] < g.d[j - 1]; --j) {
        g.ext[j] = g.ext[j - 1];
        g.op[j] = g.op[j - 1];
        g.d[j] = g.d[j - 1];
      }
      g.ext[j] = ext[i];
      g.op[j] = op[i];
      g.d[j] = d[i];
    }
  };
  const double w = cplx ? (es == 16 ? 12.0 : 2.0) : (es == 8 ? 3.0 : 5.0);
  const double M = (double)T.M, N = (double)T.N, K = (double)T.K;
  auto sectors = [&](int64_t run) { return es / 32.0 + (1.0 - es / 32.0) / (double)run; };
  double least = 0.0;
  Group m, n;
  for (int c = 0; c < 4; ++c) {  // bit 0: m in D's order, bit 1: n
    if (((c & 1) && !may_m) || ((c & 2) && !may_n)) continue;
    Group gm, gn;
    take(gm, T.nm, T.mext, T.mstrL, T.mstrD, c & 1);
    take(gn, T.nn, T.next, T.nstrR, T.nstrD, c & 2);
    // where both move as much, D's order is the faster one under a contracted stride-1 index
    const double even = ((c & 1) && !an.a_along_m ? 0.98 : 1.0) * ((c & 2) && !an.b_along_n ? 0.98 : 1.0);
    const double cost =
        even *
        (M * K * std::ceil(N / 64) * sectors(tile_run({T.nm, gm.ext, gm.op, false}, {T.nk, T.kext, T.kstrL, true})) +
        N * K * std::ceil(M / 64) * sectors(tile_run({T.nn, gn.ext, gn.op, false}, {T.nk, T.kext, T.kstrR, true})) +
        w * M * N * sectors(tile_run({T.nm, gm.ext, gm.d, false}, {T.nn, gn.ext, gn.d, false})));
    if (c == 0 || cost < least) {
      least = cost;
      m = gm;
      n = gn;
    }
  }
  std::copy(m.ext, m.ext + T.nm, T.mext); std::copy(m.op, m.op + T.nm, T.mstrL); std::copy(m.d, m.d + T.nm, T.mstrD);
  std::copy(n.ext, n.ext + T.nn, T.next); std::copy(n.op, n.op + T.nn, T.nstrR); std::copy(n.d, n.d + T.nn, T.nstrD);
}

int sm_count_dev() { return current_sm_count(); }

size_t table_bytes(const TableParams &T) {
  return (size_t)align_up(8 * (2 * T.M + 2 * T.N + 2 * T.K + (T.nh > 0 ? 3 * T.H : 0)), 256);
}

// Split of the contracted range.  A contraction with few output tiles and a
// long contracted range leaves most SMs idle (a 40 x 40 output with K = 501760
// ran on one CTA: 44 ms); its K is cut so that as many CTAs per SM have work as
// fit at once (R8 four: 217 / 193 / 185 us there with two / three / four; C8
// two), each at least 256 long (16 pipeline steps; 512 makes short ranges up to
// 15 % slower).  The cut depends on the
// shape alone, so the same contraction sums in the same order alone and in any
// batch, whatever tile runs it and whatever scratch it has.
struct KSplit {
  int nsplit = 1, kchunk = 0, gsz = 1;
};
constexpr int kSplitMinK = 256;
KSplit k_split(int kind, int64_t M, int64_t N, int64_t K, int64_t H) {
  KSplit s;
  // Shapes past 2^31 reach this only through the scratch queries (the launch
  // refuses them): K first, then each factor of the tile count, so that neither
  // the chunk nor the product leaves its type.
  if (K > 0x7fffffffLL) return s;
  const int64_t most = K / kSplitMinK, many = 8 * 148;
  if (most < 2 || (M + 63) / 64 >= many || (N + 63) / 64 >= many || H >= many) return s;
  const int64_t tiles = ((M + 63) / 64) * ((N + 63) / 64) * std::max<int64_t>(H, 1);
  if (tiles >= many) return s;
  int64_t want = std::min((kind == C8 ? 2 : kind == R4 ? 6 : 4) * 148 / tiles, most);
  if (tiles >= 148) {
    // Every SM has a tile, but not the same number of them: cut K when that
    // evens them out.  Cost of n cuts: items of the fullest SM times an item's
    // length, plus about 48 k for its start and end and 32 k for its partial sums.
    double best = 0.0;
    want = 1;
    for (int64_t n = 1; n <= std::min<int64_t>(most, 6); ++n) {
      const double cost = (double)((tiles * n + 147) / 148) * ((double)K / n + (n > 1 ? 80 : 48));
      if (n == 1 || cost < 0.99 * best) { best = cost; want = n; }
    }
  }
  if (want < 2) return s;
  s.kchunk = (int)(((K + want - 1) / want + 15) / 16 * 16);
  s.nsplit = (int)((K + s.kchunk - 1) / s.kchunk);
  s.gsz = s.nsplit;
  if (s.nsplit > 8)
    for (s.gsz = 1; s.gsz * s.gsz < s.nsplit; ++s.gsz) {}
  return s;
}
int64_t split_counters(const KSplit &s, int64_t tiles) {
  return s.nsplit > 1 ? tiles * ((s.nsplit + s.gsz - 1) / s.gsz + 1) : 0;
}
// Bytes of the partial tiles (edge x edge) and of the arrival counters.
int64_t split_bytes(const KSplit &s, int kind, int64_t M, int64_t N, int64_t H, int edge) {
  if (s.nsplit <= 1) return 0;
  const int64_t tiles = ((M + edge - 1) / edge) * ((N + edge - 1) / edge) * std::max<int64_t>(H, 1);
  return tiles * s.nsplit * edge * edge * kind_size(kind) + align_up(4 * split_counters(s, tiles), 256);
}

// CTA tile edge of a single contraction.  R8, C8: 64, or 32 when even the split
// 64 x 64 tiles do not give every SM one.  (128 x 128 R8 tiles, one CTA of 16
// warps per SM, were 1.5 % slower than four 64 x 64 CTAs on 3072 x 3072 x 3072:
// independent CTAs fill each other's barrier gaps.)  C4: 32, whose two warps
// leave eight CTAs per SM to hide a k step's latency behind (64 / 32, us: 18
// tiles of 64, K = 169: 55 / 25, 45 before the packed kernel; 105 tiles, K =
// 459: 125 / 76; 131000 x 1, K = 20: 98 / 53; 3000 x 3000 x 3000: 5847 / 5799).
// R4: 32 (4 x 4 sub-tiles) when one side is no wider, or when 64 x 64 tiles are
// fewer than three for two SMs (64 / 32, us: 131000 x 1, K = 20: 25 / 21; 300 x
// 300, K = 30: 14.6 / 10.5, 13.0 before the packed kernel; 512 x 512, K = 400: 39
// / 25; 900 x 900 x 900, 225 tiles: 74 / 70 and, loads along k, 76 / 86), else 128
// when two of those per SM exist and are mostly filled, else 64.  Results do not
// depend on it.
int gemm_edge(int kind, int64_t M, int64_t N, int64_t H, const KSplit &s) {
  auto tiles = [&](int64_t e) { return ((M + e - 1) / e) * ((N + e - 1) / e) * std::max<int64_t>(H, 1); };
  const int64_t sms = sm_count_dev();
  if (kind == R4 && (std::min(M, N) <= 32 || 2 * tiles(64) * s.nsplit < 3 * sms)) return 32;
  if (kind == R4) return tiles(128) >= 2 * sms && tiles(64) >= 3 * tiles(128) ? 128 : 64;
  if (kind == C4) return 32;
  return tiles(64) * s.nsplit >= sms ? 64 : 32;
}

// A split contracted range without room for partial tiles.
bool sequential(const GemmArgs &ga) { return ga.nsplit > 1 && ga.part == nullptr; }

// Grid of a gather-GEMM launch: tiles of one GEMM times hyper combinations
// times the splits that run in CTAs of their own.
int gemm_grid(GemmArgs &ga, int bm, int bn, int64_t *blocks) {
  ga.tiles_m = (ga.M + bm - 1) / bm;
  const int64_t per = (int64_t)ga.tiles_m * ((ga.N + bn - 1) / bn);
  const int64_t all = per * std::max(ga.H, 1) * (sequential(ga) ? 1 : std::max(ga.nsplit, 1));
  if (per > 0x7fffffffLL || all > 0x7fffffffLL) return TALSH_LIMIT_EXCEEDED;
  ga.tiles_mn = (int)per;
  *blocks = all;
  return TALSH_SUCCESS;
}

template <int BM, int BN, bool SEQ>
int launch_dmma_as(const double *L, const double *R, double *D, GemmArgs ga, cudaStream_t st) {
  using C = DmmaCfg<BM, BN>;
  static std::atomic<uint64_t> attr_set{0};
  once_per_device(attr_set, [] {
    cudaFuncSetAttribute(dgemm_gather_kernel<BM, BN, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)C::SMEM);
  });
  int64_t tiles = 0;
  if (gemm_grid(ga, BM, BN, &tiles)) return TALSH_LIMIT_EXCEEDED;
  dgemm_gather_kernel<BM, BN, SEQ><<<(unsigned)tiles, C::THREADS, C::SMEM, st>>>(L, R, D, ga);
  note_launch();
  return check_launch("dgemm_gather_kernel");
}
template <int BM, int BN>
int launch_dmma(const double *L, const double *R, double *D, const GemmArgs &ga, cudaStream_t st) {
  return sequential(ga) ? launch_dmma_as<BM, BN, true>(L, R, D, ga, st) : launch_dmma_as<BM, BN, false>(L, R, D, ga, st);
}

template <int BM, int BN, bool SEQ>
int launch_zmma_as(const double2 *L, const double2 *R, double2 *D, GemmArgs ga, cudaStream_t st) {
  using Z = ZmmaCfg<BM, BN>;
  static std::atomic<uint64_t> attr_set{0};
  once_per_device(attr_set, [] {
    cudaFuncSetAttribute(zgemm_gather_kernel<BM, BN, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Z::SMEM);
  });
  int64_t tiles = 0;
  if (gemm_grid(ga, BM, BN, &tiles)) return TALSH_LIMIT_EXCEEDED;
  zgemm_gather_kernel<BM, BN, SEQ><<<(unsigned)tiles, Z::THREADS, Z::SMEM, st>>>(L, R, D, ga);
  note_launch();
  return check_launch("zgemm_gather_kernel");
}
template <int BM, int BN>
int launch_zmma(const double2 *L, const double2 *R, double2 *D, const GemmArgs &ga, cudaStream_t st) {
  return sequential(ga) ? launch_zmma_as<BM, BN, true>(L, R, D, ga, st) : launch_zmma_as<BM, BN, false>(L, R, D, ga, st);
}

template <typename T, int BM, int BN, bool SEQ>
int launch_fmma_as(const void *L, const void *R, void *D, GemmArgs ga, cudaStream_t st) {
  using C = FmmaCfg<T, BM, BN>;
  static std::atomic<uint64_t> attr_set{0};
  once_per_device(attr_set, [] {
    cudaFuncSetAttribute(fgemm_gather_kernel<T, BM, BN, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
  });
  int64_t tiles = 0;
  if (gemm_grid(ga, BM, BN, &tiles)) return TALSH_LIMIT_EXCEEDED;
  fgemm_gather_kernel<T, BM, BN, SEQ><<<(unsigned)tiles, C::THREADS, C::SMEM, st>>>((const T *)L, (const T *)R, (T *)D, ga);
  note_launch();
  return check_launch("fgemm_gather_kernel");
}
template <typename T, int BM, int BN>
int launch_fmma(const void *L, const void *R, void *D, const GemmArgs &ga, cudaStream_t st) {
  return sequential(ga) ? launch_fmma_as<T, BM, BN, true>(L, R, D, ga, st)
                        : launch_fmma_as<T, BM, BN, false>(L, R, D, ga, st);
}

template <typename T>
int launch_dot(const void *L, const void *R, void *D, const int64_t *kL, const int64_t *kR,
               int64_t K, int cl, int cr, double ar, double ai, int beta, double2 *part,
               cudaStream_t st) {
  const int nb = dot_blocks(K);
  const int64_t chunk = (K + nb - 1) / nb;
  dot_partial_kernel<T><<<nb, kDotThreads, 0, st>>>((const T *)L, (const T *)R, kL, kR, K, chunk, cl, cr, part);
  note_launch();
  dot_final_kernel<T><<<1, kDotThreads, 0, st>>>(part, nb, (T *)D, ar, ai, beta);
  note_launch();
  return check_launch("dot_kernels");
}

int launch_dot_final(int kind, const double2 *part, int n, void *D, double ar, double ai, int beta, cudaStream_t st) {
  switch (kind) {
    case R4: dot_final_kernel<float><<<1, kDotThreads, 0, st>>>(part, n, (float *)D, ar, ai, beta); break;
    case R8: dot_final_kernel<double><<<1, kDotThreads, 0, st>>>(part, n, (double *)D, ar, ai, beta); break;
    case C4: dot_final_kernel<float2><<<1, kDotThreads, 0, st>>>(part, n, (float2 *)D, ar, ai, beta); break;
    default: dot_final_kernel<double2><<<1, kDotThreads, 0, st>>>(part, n, (double2 *)D, ar, ai, beta); break;
  }
  note_launch();
  return check_launch("dot_final_kernel");
}

template <typename T>
int launch_scalar(const void *L, const void *R, void *D, double ar, double ai, int cl, int cr,
                  int beta, cudaStream_t st) {
  scalar_mul_kernel<T><<<1, 1, 0, st>>>((const T *)L, (const T *)R, (T *)D, ar, ai, cl, cr, beta);
  note_launch();
  return check_launch("scalar_mul_kernel");
}

// Operands must be aligned to their element size (16 bytes for C8): the
// kernels move whole elements with vector loads and stores.
bool elements_aligned(int kind, const void *D, const void *L, const void *R) {
  const uintptr_t m = (uintptr_t)kind_size(kind) - 1;
  return ((reinterpret_cast<uintptr_t>(D) | reinterpret_cast<uintptr_t>(L) | reinterpret_cast<uintptr_t>(R)) & m) == 0;
}

// Shape / kind checks shared by the scratch query and the launch.
int check_args(int kind, const int *cptrn, int drank, const int *ddims, int lrank, const int *ldims,
               int rrank, const int *rdims) {
  if (kind_size(kind) == 0) return TALSH_INVALID_ARGS;
  if (drank < 0 || lrank < 0 || rrank < 0 || drank > kMaxRank || lrank > kMaxRank || rrank > kMaxRank)
    return TALSH_INVALID_ARGS;
  if ((lrank + rrank > 0 && cptrn == nullptr) || (drank > 0 && ddims == nullptr) ||
      (lrank > 0 && ldims == nullptr) || (rrank > 0 && rdims == nullptr))
    return TALSH_INVALID_ARGS;
  for (int i = 0; i < drank; ++i) if (ddims[i] <= 0) return TALSH_INVALID_ARGS;
  for (int i = 0; i < lrank; ++i) if (ldims[i] <= 0) return TALSH_INVALID_ARGS;
  for (int i = 0; i < rrank; ++i) if (rdims[i] <= 0) return TALSH_INVALID_ARGS;
  return TALSH_SUCCESS;
}

}  // namespace

// Scratch bytes of tcTensorContract for this shape (0 when none): the offset
// tables and, for a split contracted range, the partial sums and counters.
// `least`, when given, receives what the form without partial sums needs: a call
// with less than the full size but at least that computes the same bits on one
// CTA per tile.
size_t contract_scratch_bytes(int kind, const int *cptrn, int drank, const int *ddims, int lrank,
                              const int *ldims, int rrank, const int *rdims, size_t *least) {
  if (least) *least = 0;
  if (check_args(kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims)) return 0;
  if (lrank == 0 || rrank == 0) return 0;
  Analysis an;
  if (analyze(cptrn, drank, ddims, lrank, ldims, rrank, rdims, an)) return 0;
  const TableParams &T = an.T;
  size_t b = table_bytes(T);
  if (drank == 0) b += (size_t)dot_blocks(T.K) * sizeof(double2);
  if (least) *least = b;
  if (drank == 0) return b;
  const KSplit ks = k_split(kind, T.M, T.N, T.K, T.H);
  return b + (size_t)split_bytes(ks, kind, T.M, T.N, T.H, gemm_edge(kind, T.M, T.N, T.H, ks));
}
size_t contract_scratch_bytes(int kind, const int *cptrn, int drank, const int *ddims, int lrank,
                              const int *ldims, int rrank, const int *rdims) {
  return contract_scratch_bytes(kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims, nullptr);
}

// The argument checks of contract_launch without launching anything.
int contract_validate(int kind, const int *cptrn, int drank, const int *ddims, int lrank, const int *ldims,
                      int rrank, const int *rdims) {
  int rc = check_args(kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims);
  if (rc) return rc;
  if (lrank == 0 && rrank == 0) return drank == 0 ? TALSH_SUCCESS : TALSH_INVALID_ARGS;
  if (lrank == 0 || rrank == 0) {
    const int trank = lrank ? lrank : rrank;
    const int *tdims = lrank ? ldims : rdims;
    const int *tptrn = lrank ? cptrn : cptrn + lrank;
    if (trank != drank) return TALSH_INVALID_ARGS;
    for (int i = 0; i < trank; ++i)
      if (tptrn[i] < 1 || tptrn[i] > drank || ddims[tptrn[i] - 1] != tdims[i]) return TALSH_INVALID_ARGS;
    return TALSH_SUCCESS;
  }
  Analysis an;
  if ((rc = analyze(cptrn, drank, ddims, lrank, ldims, rrank, rdims, an)) != 0) return rc;
  if (an.T.M > 0x7fffffffLL || an.T.N > 0x7fffffffLL || an.T.K > 0x7fffffffLL || an.T.H > 0x7fffffffLL)
    return TALSH_LIMIT_EXCEEDED;
  return TALSH_SUCCESS;
}

int contract_launch(int kind, const int *cptrn, int drank, const int *ddims, int lrank,
                    const int *ldims, int rrank, const int *rdims, void *D, const void *L,
                    const void *R, double alpha_re, double alpha_im, int conj_bits,
                    int accumulative, void *scratch, size_t scratch_bytes, void *stream) {
  int rc = check_args(kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims);
  if (rc) return rc;
  if (D == nullptr || L == nullptr || R == nullptr) return TALSH_INVALID_ARGS;
  if (!elements_aligned(kind, D, L, R)) return TALSH_INVALID_ARGS;
  const bool cplx = kind_is_complex(kind);
  int cl = 0, cr = 0;
  if (cplx) {
    int cb = conj_bits & 7;
    if (cb & 1) cb ^= 7;  // a conjugated destination conjugates both inputs instead
    cl = (cb >> 1) & 1;
    cr = (cb >> 2) & 1;
  }
  const double ar = alpha_re, ai = cplx ? alpha_im : 0.0;
  const int beta = accumulative ? 1 : 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (lrank == 0 && rrank == 0) {
    if (drank != 0) return TALSH_INVALID_ARGS;
    switch (kind) {
      case R4: return launch_scalar<float>(L, R, D, alpha_re, alpha_im, cl, cr, beta, st);
      case R8: return launch_scalar<double>(L, R, D, alpha_re, alpha_im, cl, cr, beta, st);
      case C4: return launch_scalar<float2>(L, R, D, alpha_re, alpha_im, cl, cr, beta, st);
      default: return launch_scalar<double2>(L, R, D, alpha_re, alpha_im, cl, cr, beta, st);
    }
  }
  if (lrank == 0 || rrank == 0) {
    // scalar x tensor: D (+)= permute(T) * (s * alpha), the reference's ADD_TENSOR case.
    const int trank = lrank ? lrank : rrank;
    const int *tdims = lrank ? ldims : rdims;
    const int *tptrn = lrank ? cptrn : cptrn + lrank;
    if (trank != drank) return TALSH_INVALID_ARGS;
    for (int i = 0; i < trank; ++i)
      if (tptrn[i] < 1 || tptrn[i] > drank || ddims[tptrn[i] - 1] != tdims[i]) return TALSH_INVALID_ARGS;
    return permute_scaled_by_device_scalar(kind, trank, tdims, tptrn, lrank ? L : R, D, alpha_re,
                                           alpha_im, lrank ? R : L, lrank ? cr : cl,
                                           lrank ? cl : cr, beta, stream);
  }
  Analysis an;
  if ((rc = analyze(cptrn, drank, ddims, lrank, ldims, rrank, rdims, an)) != 0) return rc;
  order_by_output(an, kind_size(kind), kind_is_complex(kind));
  TableParams T = an.T;
  const size_t need = table_bytes(T) + (drank == 0 ? (size_t)dot_blocks(T.K) * sizeof(double2) : 0);
  if (scratch == nullptr || scratch_bytes < need) return TALSH_INVALID_ARGS;
  if (T.M > 0x7fffffffLL || T.N > 0x7fffffffLL || T.K > 0x7fffffffLL || T.H > 0x7fffffffLL)
    return TALSH_LIMIT_EXCEEDED;
  int64_t *base = (int64_t *)scratch;
  T.es = kind_size(kind);
  T.mL = base; T.mD = T.mL + T.M; T.nR = T.mD + T.M; T.nD = T.nR + T.N; T.kL = T.nD + T.N; T.kR = T.kL + T.K;
  if (T.nh > 0) {
    T.hL = T.kR + T.K; T.hR = T.hL + T.H; T.hD = T.hR + T.H;
  }
  const bool vec_scratch = (uintptr_t)scratch % 16 == 0;  // partial sums are moved 16 bytes at a time
  if (drank == 0 && vec_scratch) {
    // Full contraction: R is walked in L's index order, each operand read once
    // along its own runs.  (Through the offset tables it cost 32 bytes of table
    // traffic per element pair and uncoalesced reads of one operand: 299 us
    // against this form's 66 us for two 20 M element R8 tensors.)
    int o2n[kMaxRank], nparts = 0;
    for (int j = 0; j < rrank; ++j) o2n[j] = -cptrn[lrank + j];
    rc = permute_dot_launch(kind, rrank, rdims, o2n, R, L, cplx ? cr : 0, cplx ? cl : 0, (double2 *)scratch,
                            (int64_t)(need / sizeof(double2)), &nparts, st);
    if (rc != TALSH_NOT_IMPLEMENTED)
      return rc ? rc : launch_dot_final(kind, (const double2 *)scratch, nparts, D, ar, ai, beta, st);
  }
  KSplit ks;
  int edge = 64;
  void *part = nullptr;
  if (drank > 0) {
    ks = k_split(kind, T.M, T.N, T.K, T.H);
    edge = gemm_edge(kind, T.M, T.N, T.H, ks);
    const int64_t extra = split_bytes(ks, kind, T.M, T.N, T.H, edge);
    if (ks.nsplit > 1 && scratch_bytes >= need + (size_t)extra && vec_scratch) {
      const int64_t tiles = ((T.M + edge - 1) / edge) * ((T.N + edge - 1) / edge) * T.H;
      T.ncnt = split_counters(ks, tiles);
      T.cnt = (int *)((char *)scratch + need);
      part = (char *)T.cnt + align_up(4 * T.ncnt, 256);
    } else {  // one CTA per tile
      edge = gemm_edge(kind, T.M, T.N, T.H, KSplit());
    }
  }
  {
    const int64_t total = T.M + T.N + T.K + (T.nh > 0 ? T.H : 0);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 4096));
    build_tables_kernel<<<grid, 256, 0, st>>>(T);
    note_launch();
    if ((rc = check_launch("build_tables_kernel")) != 0) return rc;
  }
  if (drank == 0) {
    double2 *part = (double2 *)((char *)scratch + table_bytes(T));
    switch (kind) {
      case R4: return launch_dot<float>(L, R, D, T.kL, T.kR, T.K, cl, cr, ar, ai, beta, part, st);
      case R8: return launch_dot<double>(L, R, D, T.kL, T.kR, T.K, cl, cr, ar, ai, beta, part, st);
      case C4: return launch_dot<float2>(L, R, D, T.kL, T.kR, T.K, cl, cr, ar, ai, beta, part, st);
      default: return launch_dot<double2>(L, R, D, T.kL, T.kR, T.K, cl, cr, ar, ai, beta, part, st);
    }
  }
  GemmArgs ga;
  std::memset(&ga, 0, sizeof(ga));
  ga.M = (int)T.M; ga.N = (int)T.N; ga.K = (int)T.K;
  ga.mL = T.mL; ga.mD = T.mD; ga.nR = T.nR; ga.nD = T.nD; ga.kL = T.kL; ga.kR = T.kR;
  ga.alpha_re = ar; ga.alpha_im = ai; ga.beta = beta;
  ga.a_along_m = an.a_along_m ? 1 : 0;
  ga.b_along_n = an.b_along_n ? 1 : 0;
  ga.conj_l = cl; ga.conj_r = cr;
  ga.H = (int)T.H;
  if (T.nh > 0) {
    ga.hL = T.hL; ga.hR = T.hR; ga.hD = T.hD;
  }
  ga.nsplit = ks.nsplit; ga.kchunk = ks.kchunk; ga.gsz = ks.gsz;
  ga.cnt = T.cnt;
  ga.part = part;
  switch (kind) {
    case R8: {
      const double *l = (const double *)L, *r = (const double *)R;
      if (edge == 64) return launch_dmma<64, 64>(l, r, (double *)D, ga, st);
      return launch_dmma<32, 32>(l, r, (double *)D, ga, st);
    }
    case R4:
      if (edge == 128) return launch_fmma<float, 128, 128>(L, R, D, ga, st);
      if (edge == 64) return launch_fmma<float, 64, 64>(L, R, D, ga, st);
      return launch_fmma<float, 32, 32>(L, R, D, ga, st);
    case C4: return launch_fmma<float2, 32, 32>(L, R, D, ga, st);
    default:
      if (edge == 64) return launch_zmma<64, 64>((const double2 *)L, (const double2 *)R, (double2 *)D, ga, st);
      return launch_zmma<32, 32>((const double2 *)L, (const double2 *)R, (double2 *)D, ga, st);
  }
}

}  // namespace tb

namespace tb {
// Offset tables (m -> L, D; n -> R, D; k -> L, R) for callers that only need
// the D scatter: bytes for given M, N, K, and a launch that builds them.
size_t contract_tables_bytes(int64_t M, int64_t N, int64_t K) {
  TableParams T;
  std::memset(&T, 0, sizeof(T));
  T.M = M; T.N = N; T.K = K;
  return table_bytes(T);
}

int contract_build_tables(const int *cptrn, int drank, const int *ddims, int lrank, const int *ldims,
                          int rrank, const int *rdims, void *tables, cudaStream_t st, int64_t &M,
                          int64_t &N, int64_t &K, const int64_t **mD, const int64_t **nD) {
  int rc = check_args(R8, cptrn, drank, ddims, lrank, ldims, rrank, rdims);
  if (rc) return rc;
  Analysis an;
  if ((rc = analyze(cptrn, drank, ddims, lrank, ldims, rrank, rdims, an)) != 0) return rc;
  if (an.hyper) return TALSH_NOT_IMPLEMENTED;
  TableParams T = an.T;
  int64_t *base = (int64_t *)tables;
  T.es = kind_size(R8);
  T.mL = base; T.mD = T.mL + T.M; T.nR = T.mD + T.M; T.nD = T.nR + T.N; T.kL = T.nD + T.N; T.kR = T.kL + T.K;
  const int64_t total = T.M + T.N + T.K;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 4096));
  build_tables_kernel<<<grid, 256, 0, st>>>(T);
  note_launch();
  if ((rc = check_launch("build_tables_kernel")) != 0) return rc;
  M = T.M; N = T.N; K = T.K;
  *mD = T.mD;
  *nD = T.nD;
  return TALSH_SUCCESS;
}
}  // namespace tb

extern "C" size_t tcTensorContractScratch(int data_kind, const int *cptrn, int drank,
                                          const int *ddims, int lrank, const int *ldims,
                                          int rrank, const int *rdims) {
  return tb::contract_scratch_bytes(data_kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims);
}


extern "C" int tcTensorContract(int data_kind, const int *cptrn, int drank, const int *ddims,
                                int lrank, const int *ldims, int rrank, const int *rdims, void *D,
                                const void *L, const void *R, double alpha_re, double alpha_im,
                                int conj_bits, int accumulative, void *scratch,
                                size_t scratch_bytes, void *stream) {
  return tb::contract_launch(data_kind, cptrn, drank, ddims, lrank, ldims, rrank, rdims, D, L, R,
                             alpha_re, alpha_im, conj_bits, accumulative, scratch, scratch_bytes,
                             stream);
}

// ---------------------------------------------------------------------------
// Batched contractions: many (small) contractions in one table launch and one
// persistent gather-GEMM launch per tile configuration.  Each task's compact
// descriptor (index groups, strides, GEMM arguments, operand pointers) is
// uploaded once; CTAs walk a flat list of tiles over all tasks of a
// configuration and find their task by binary search in its tile prefix sums.
// ---------------------------------------------------------------------------
namespace tb {
namespace {

constexpr int kBMaxG = 8;  // max dimensions per index group of a batched task

struct BatchDesc {
  int nm, nn, nk, es;
  int32_t mext[kBMaxG], next[kBMaxG], kext[kBMaxG];
  int64_t mstrL[kBMaxG], mstrD[kBMaxG], nstrR[kBMaxG], nstrD[kBMaxG], kstrL[kBMaxG], kstrR[kBMaxG];
  GemmArgs a;
  const void *L, *R;
  void *D;
};

// Tile configurations of the batch: 0 = DMMA 64x64, 1 = DMMA 32x32 (R8),
// Z = complex on the DMMA pipe, S4 / S14 = packed FP32 FMA 64x64 (R4 / C4).
// From kCfgSeq on: the same for tasks whose split range has no partial sums.
enum : int { kCfgD64 = 0, kCfgD32 = 1, kCfgZ64 = 2, kCfgZ32 = 3, kCfgS4 = 4, kCfgS14 = 5, kCfgSeq = 6, kNumCfg = 12 };
// Square tile edge of a configuration.
inline int cfg_tile(int c) { return (c % kCfgSeq == kCfgD32 || c % kCfgSeq == kCfgZ32) ? 32 : 64; }

__global__ void __launch_bounds__(256) batch_tables_kernel(const BatchDesc *descs) {
  const BatchDesc &d = descs[blockIdx.y];
  const int64_t M = d.a.M, N = d.a.N, K = d.a.K;
  const int64_t total = M + N + K;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < d.a.ncnt; i += (int64_t)gridDim.x * 256) d.a.cnt[i] = 0;
  int64_t *mL = const_cast<int64_t *>(d.a.mL), *mD = const_cast<int64_t *>(d.a.mD);
  int64_t *nR = const_cast<int64_t *>(d.a.nR), *nD = const_cast<int64_t *>(d.a.nD);
  int64_t *kL = const_cast<int64_t *>(d.a.kL), *kR = const_cast<int64_t *>(d.a.kR);
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
    int64_t x, y;
    if (i < M) {
      group_offsets((uint32_t)i, d.nm, d.mext, d.mstrL, d.mstrD, x, y);
      mL[i] = x * d.es;
      mD[i] = y;
    } else if (i < M + N) {
      group_offsets((uint32_t)(i - M), d.nn, d.next, d.nstrR, d.nstrD, x, y);
      nR[i - M] = x * d.es;
      nD[i - M] = y;
    } else {
      const int64_t k = i - M - N;
      group_offsets((uint32_t)k, d.nk, d.kext, d.kstrL, d.kstrR, x, y);
      kL[k] = x * d.es;
      kR[k] = y * d.es;
    }
  }
}

// Task owning flat tile w: largest j with prefix[j] <= w.
__device__ __forceinline__ int find_task(const int64_t *prefix, int n, int64_t w) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= w) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Item i of a task: its tiles, repeated for every split of the contracted range.
__device__ __forceinline__ TileWork item_work(const GemmArgs &a, int i) {
  TileWork w;
  w.split = i / a.tiles_mn;
  w.lin = i - w.split * a.tiles_mn;
  w.tm = w.lin % a.tiles_m;
  w.tn = w.lin / a.tiles_m;
  return w;
}

// The item's GEMM arguments, kept in shared memory (in registers they spilled).
__device__ __forceinline__ void stage_args(GemmArgs &to, const GemmArgs &from) {
  static_assert(sizeof(GemmArgs) % 4 == 0, "copied as words");
  const uint32_t *f = reinterpret_cast<const uint32_t *>(&from);
  uint32_t *t = reinterpret_cast<uint32_t *>(&to);
  for (int i = threadIdx.x; i < (int)(sizeof(GemmArgs) / 4); i += blockDim.x) t[i] = f[i];
  __syncthreads();
}

// Dynamic work distribution: CTAs take the next flat tile from a counter; the
// host orders the tasks by decreasing K (longest tiles first).
__device__ __forceinline__ int64_t next_item(unsigned long long *ctr) {
  __shared__ int64_t item;
  __syncthreads();
  if (threadIdx.x == 0) item = (int64_t)atomicAdd(ctr, 1ull);
  __syncthreads();
  return item;
}

template <int BM, int BN, bool SEQ>
__global__ void __launch_bounds__(DmmaCfg<BM, BN>::THREADS, SEQ ? 1 : GemmOcc<BM, BN>::D)
    dmma_batch_kernel(const BatchDesc *descs, const int32_t *list, const int64_t *prefix, int n,
                      int64_t total, unsigned long long *ctr) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ GemmArgs a;
  for (int64_t w = next_item(ctr); w < total; w = next_item(ctr)) {
    const int j = find_task(prefix, n, w);
    const BatchDesc &d = descs[list[j]];
    stage_args(a, d.a);
    dmma_tile<BM, BN, SEQ>((const double *)d.L, (const double *)d.R, (double *)d.D, a, item_work(a, (int)(w - prefix[j])),
                      smem);
  }
}

template <int BM, int BN, bool SEQ>
__global__ void __launch_bounds__(ZmmaCfg<BM, BN>::THREADS, SEQ ? 1 : GemmOcc<BM, BN>::Z)
    zmma_batch_kernel(const BatchDesc *descs, const int32_t *list, const int64_t *prefix, int n,
                      int64_t total, unsigned long long *ctr) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ GemmArgs a;
  for (int64_t w = next_item(ctr); w < total; w = next_item(ctr)) {
    const int j = find_task(prefix, n, w);
    const BatchDesc &d = descs[list[j]];
    stage_args(a, d.a);
    zmma_tile<BM, BN, SEQ>((const double2 *)d.L, (const double2 *)d.R, (double2 *)d.D, a,
                      item_work(a, (int)(w - prefix[j])), smem);
  }
}

template <typename T, bool SEQ>
__global__ void __launch_bounds__(FmmaCfg<T, 64, 64>::THREADS, SEQ ? 1 : FmmaOcc<T, 64>::N)
    fmma_batch_kernel(const BatchDesc *descs, const int32_t *list, const int64_t *prefix, int n,
                      int64_t total, unsigned long long *ctr) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ GemmArgs a;
  for (int64_t w = next_item(ctr); w < total; w = next_item(ctr)) {
    const int j = find_task(prefix, n, w);
    const BatchDesc &d = descs[list[j]];
    stage_args(a, d.a);
    fmma_tile<T, 64, 64, SEQ>((const T *)d.L, (const T *)d.R, (T *)d.D, a, item_work(a, (int)(w - prefix[j])), smem);
  }
}

struct BatchPlan {
  std::vector<BatchDesc> descs;
  std::vector<int> cfg;          // per task: configuration, or -1 = single-task fallback
  std::vector<int64_t> tab_off;  // per task: offset of its tables (int64 elements)
  std::vector<size_t> part_off;  // per task: offset of its partial sums and counters (bytes, from off_part)
  size_t off_part = 0;
  std::vector<size_t> fb_scratch;
  std::vector<size_t> fb_off;
  std::vector<int32_t> list[kNumCfg];
  std::vector<int64_t> prefix[kNumCfg];
  size_t off_desc = 0, off_list[kNumCfg] = {}, off_prefix[kNumCfg] = {}, off_tab = 0, off_fb = 0, off_ctr = 0,
         total = 0;
};

// Tile choices of the autotuner (tcTensorContractBatchTune) per task class:
// kind (R8, C8) x bucket of M x bucket of N, buckets < 16, < 48, < 128, >= 128.
// 0 = not tuned (the shape rule below applies), else the tile edge (32 or 64).
constexpr int kTuneBuckets = 4;
std::atomic<int> g_tune[2][kTuneBuckets][kTuneBuckets];

int tune_bucket(int64_t x) { return x < 16 ? 0 : x < 48 ? 1 : x < 128 ? 2 : 3; }

int batch_cfg_of(int kind, int64_t M, int64_t N) {
  if (kind == R8 || kind == C8) {
    const int t = g_tune[kind == C8][tune_bucket(M)][tune_bucket(N)].load(std::memory_order_relaxed);
    if (t == 32) return kind == R8 ? kCfgD32 : kCfgZ32;
    if (t == 64) return kind == R8 ? kCfgD64 : kCfgZ64;
  }
  switch (kind) {
    case R8: return (M >= 48 && N >= 48) ? kCfgD64 : kCfgD32;
    case C8: return (M >= 48 && N >= 48) ? kCfgZ64 : kCfgZ32;
    case R4: return kCfgS4;
    default: return kCfgS14;
  }
}

// Bytes of a task's partial sums and counters for whichever tile edge it gets, so
// that the scratch of a batch does not depend on what was tuned, when, or on the
// edge the autotuner is trying.
size_t batch_part_bytes(const KSplit &ks, int kind, int64_t M, int64_t N) {
  const int64_t wide = split_bytes(ks, kind, M, N, 1, 64);
  const bool narrow = kind == R8 || kind == C8;
  return (size_t)align_up(narrow ? std::max(wide, split_bytes(ks, kind, M, N, 1, 32)) : wide, 256);
}

// `lean` (one flag per task, or null): no partial sums for that task; each CTA
// of a tile then walks the task's splits itself.
int batch_plan(int ntasks, const tcContractTask *tasks, BatchPlan &bp, const std::vector<char> *lean = nullptr) {
  if (ntasks < 0 || ntasks > 65535 || (ntasks > 0 && tasks == nullptr)) return TALSH_INVALID_ARGS;
  bp.descs.assign(ntasks, BatchDesc());
  bp.cfg.assign(ntasks, -1);
  bp.tab_off.assign(ntasks, 0);
  bp.fb_scratch.assign(ntasks, 0);
  bp.fb_off.assign(ntasks, 0);
  bp.part_off.assign(ntasks, 0);
  int64_t tab = 0;
  size_t part = 0;
  for (int t = 0; t < ntasks; ++t) {
    const tcContractTask &x = tasks[t];
    if (x.drank > TC_BATCH_MAX_RANK || x.lrank > TC_BATCH_MAX_RANK || x.rrank > TC_BATCH_MAX_RANK)
      return TALSH_INVALID_ARGS;
    int rc = check_args(x.data_kind, x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims);
    if (rc) return rc;
    if (x.D == nullptr || x.L == nullptr || x.R == nullptr) return TALSH_INVALID_ARGS;
    if (!elements_aligned(x.data_kind, x.D, x.L, x.R)) return TALSH_INVALID_ARGS;
    Analysis an;
    bool batchable = x.lrank > 0 && x.rrank > 0;  // a full contraction (D of rank 0) is a 1 x 1 GEMM
    if (batchable) {
      if ((rc = analyze(x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims, an)) != 0) return rc;
      batchable = !an.hyper && an.T.nm <= kBMaxG && an.T.nn <= kBMaxG && an.T.nk <= kBMaxG &&
                  an.T.M <= 0x7fffffffLL && an.T.N <= 0x7fffffffLL && an.T.K <= 0x7fffffffLL;
    }
    if (!batchable) {  // scalar operands, hyper-indices: single-task path
      size_t least = 0;
      bp.fb_scratch[t] = contract_scratch_bytes(x.data_kind, x.cptrn, x.drank, x.ddims, x.lrank, x.ldims,
                                                x.rrank, x.rdims, &least);
      if (lean && (*lean)[t]) bp.fb_scratch[t] = least;
      continue;
    }
    order_by_output(an, kind_size(x.data_kind), kind_is_complex(x.data_kind));
    const TableParams &T = an.T;
    BatchDesc &d = bp.descs[t];
    d.nm = T.nm; d.nn = T.nn; d.nk = T.nk; d.es = kind_size(x.data_kind);
    for (int g = 0; g < T.nm; ++g) { d.mext[g] = (int32_t)T.mext[g]; d.mstrL[g] = T.mstrL[g]; d.mstrD[g] = T.mstrD[g]; }
    for (int g = 0; g < T.nn; ++g) { d.next[g] = (int32_t)T.next[g]; d.nstrR[g] = T.nstrR[g]; d.nstrD[g] = T.nstrD[g]; }
    for (int g = 0; g < T.nk; ++g) { d.kext[g] = (int32_t)T.kext[g]; d.kstrL[g] = T.kstrL[g]; d.kstrR[g] = T.kstrR[g]; }
    const bool cplx = kind_is_complex(x.data_kind);
    int cl = 0, cr = 0;
    if (cplx) {
      int cb = x.conj_bits & 7;
      if (cb & 1) cb ^= 7;
      cl = (cb >> 1) & 1;
      cr = (cb >> 2) & 1;
    }
    GemmArgs &a = d.a;
    std::memset(&a, 0, sizeof(a));
    a.M = (int)T.M; a.N = (int)T.N; a.K = (int)T.K;
    a.alpha_re = x.alpha_re; a.alpha_im = cplx ? x.alpha_im : 0.0;
    a.beta = x.accumulative ? 1 : 0;
    a.a_along_m = an.a_along_m ? 1 : 0;
    a.b_along_n = an.b_along_n ? 1 : 0;
    a.conj_l = cl; a.conj_r = cr;
    d.L = x.L; d.R = x.R; d.D = x.D;
    int c = batch_cfg_of(x.data_kind, T.M, T.N);
    const int bm = cfg_tile(c), bn = bm;
    a.tiles_m = (int)((T.M + bm - 1) / bm);
    const int64_t tiles = (int64_t)a.tiles_m * ((T.N + bn - 1) / bn);
    if (tiles > 0x7fffffffLL) return TALSH_LIMIT_EXCEEDED;
    a.tiles_mn = (int)tiles;
    const KSplit ks = k_split(x.data_kind, T.M, T.N, T.K, 1);
    a.nsplit = ks.nsplit; a.kchunk = ks.kchunk; a.gsz = ks.gsz;
    if (lean && (*lean)[t]) {
      if (ks.nsplit > 1) c += kCfgSeq;
    } else {
      a.ncnt = (int)split_counters(ks, tiles);
      bp.part_off[t] = part;
      part += batch_part_bytes(ks, x.data_kind, T.M, T.N);
    }
    bp.cfg[t] = c;
    bp.tab_off[t] = tab;
    tab += 2 * (T.M + T.N + T.K);
    bp.list[c].push_back(t);
  }
  // Longest items (largest K, or K chunk) first, then the item prefix sums.
  auto splits = [&](int t) { return bp.cfg[t] >= kCfgSeq ? 1 : bp.descs[t].a.nsplit; };  // CTAs that share a tile
  auto span = [&](int t) { return splits(t) > 1 ? bp.descs[t].a.kchunk : bp.descs[t].a.K; };
  for (int c = 0; c < kNumCfg; ++c) {
    auto &l = bp.list[c];
    std::stable_sort(l.begin(), l.end(), [&](int x, int y) { return span(x) > span(y); });
    auto &pl = bp.prefix[c];
    if (l.empty()) continue;
    pl.push_back(0);
    for (int t : l) {
      pl.push_back(pl.back() + (int64_t)bp.descs[t].a.tiles_mn * splits(t));
    }
  }
  size_t off = 0;
  auto take = [&](size_t bytes, size_t unit = 256) {
    const size_t o = off = (off + unit - 1) / unit * unit;
    off += bytes;
    return o;
  };
  bp.off_desc = take(sizeof(BatchDesc) * (size_t)std::max(ntasks, 1));
  // The lists take the same room however the tasks fall into them.
  const size_t lists = off + (size_t)ntasks * (sizeof(int32_t) + sizeof(int64_t)) + kNumCfg * (sizeof(int64_t) + 2 * 16);
  for (int c = 0; c < kNumCfg; ++c) {
    bp.off_list[c] = take(sizeof(int32_t) * bp.list[c].size(), 16);
    bp.off_prefix[c] = take(sizeof(int64_t) * bp.prefix[c].size(), 16);
  }
  off = lists;
  bp.off_tab = take(sizeof(int64_t) * (size_t)tab);
  bp.off_ctr = take(sizeof(unsigned long long) * kNumCfg);
  for (int t = 0; t < ntasks; ++t)
    if (bp.cfg[t] < 0) bp.fb_off[t] = take(bp.fb_scratch[t]);
  bp.off_part = take(part);
  bp.total = (off + 255) & ~size_t(255);
  return TALSH_SUCCESS;
}

using BatchKernel = void (*)(const BatchDesc *, const int32_t *, const int64_t *, int, int64_t,
                             unsigned long long *);

// Persistent launch of one tensor-pipe batch kernel: as many CTAs as fit at once.
int launch_tc_batch(BatchKernel k, int threads, size_t smem, const char *name, const BatchPlan &bp, int c,
                    char *base, cudaStream_t st) {
  const int64_t total = bp.prefix[c].back();
  int bps = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k, threads, smem) != cudaSuccess || bps < 1) bps = 1;
  cudaGetLastError();
  const int64_t grid = std::min<int64_t>(total, (int64_t)sm_count_dev() * bps);
  k<<<(unsigned)grid, threads, smem, st>>>(
      (const BatchDesc *)(base + bp.off_desc), (const int32_t *)(base + bp.off_list[c]),
      (const int64_t *)(base + bp.off_prefix[c]), (int)bp.list[c].size(), total,
      (unsigned long long *)(base + bp.off_ctr) + c);
  note_launch();
  return check_launch(name);
}

template <int BM, int BN, bool SEQ>
int launch_dmma_batch(const BatchPlan &bp, int c, char *base, cudaStream_t st) {
  using C = DmmaCfg<BM, BN>;
  static std::atomic<uint64_t> attr{0};
  once_per_device(attr, [] {
    cudaFuncSetAttribute(dmma_batch_kernel<BM, BN, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    cudaFuncSetAttribute(dmma_batch_kernel<BM, BN, SEQ>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
  return launch_tc_batch(dmma_batch_kernel<BM, BN, SEQ>, C::THREADS, C::SMEM, "dmma_batch_kernel", bp, c, base, st);
}

template <int BM, int BN, bool SEQ>
int launch_zmma_batch(const BatchPlan &bp, int c, char *base, cudaStream_t st) {
  using Z = ZmmaCfg<BM, BN>;
  static std::atomic<uint64_t> attr{0};
  once_per_device(attr, [] {
    cudaFuncSetAttribute(zmma_batch_kernel<BM, BN, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Z::SMEM);
    cudaFuncSetAttribute(zmma_batch_kernel<BM, BN, SEQ>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
  return launch_tc_batch(zmma_batch_kernel<BM, BN, SEQ>, Z::THREADS, Z::SMEM, "zmma_batch_kernel", bp, c, base, st);
}

template <typename T, bool SEQ>
int launch_fmma_batch(const BatchPlan &bp, int c, char *base, cudaStream_t st) {
  using C = FmmaCfg<T, 64, 64>;
  static std::atomic<uint64_t> attr{0};
  once_per_device(attr, [] {
    cudaFuncSetAttribute(fmma_batch_kernel<T, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    cudaFuncSetAttribute(fmma_batch_kernel<T, SEQ>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
  return launch_tc_batch(fmma_batch_kernel<T, SEQ>, C::THREADS, C::SMEM, "fmma_batch_kernel", bp, c, base, st);
}

// The persistent launch of configuration c.
template <bool SEQ>
int launch_cfg_as(const BatchPlan &bp, int c, char *base, cudaStream_t st) {
  switch (c % kCfgSeq) {
    case kCfgD64: return launch_dmma_batch<64, 64, SEQ>(bp, c, base, st);
    case kCfgD32: return launch_dmma_batch<32, 32, SEQ>(bp, c, base, st);
    case kCfgZ64: return launch_zmma_batch<64, 64, SEQ>(bp, c, base, st);
    case kCfgZ32: return launch_zmma_batch<32, 32, SEQ>(bp, c, base, st);
    case kCfgS4: return launch_fmma_batch<float, SEQ>(bp, c, base, st);
    default: return launch_fmma_batch<float2, SEQ>(bp, c, base, st);
  }
}
int launch_cfg(const BatchPlan &bp, int c, char *base, cudaStream_t st) {
  return c < kCfgSeq ? launch_cfg_as<false>(bp, c, base, st) : launch_cfg_as<true>(bp, c, base, st);
}

}  // namespace
}  // namespace tb

namespace tb {
namespace {

// The plan for a scratch block of `bytes`: without the partial sums of split
// contracted ranges when those do not fit or the block is not aligned for them
// (batch_run refuses what is smaller still).
int batch_plan_for(int ntasks, const tcContractTask *tasks, BatchPlan &bp, const void *scratch, size_t bytes) {
  const int rc = batch_plan(ntasks, tasks, bp);
  if (rc || (bytes >= bp.total && (uintptr_t)scratch % 16 == 0)) return rc;
  bp = BatchPlan();
  const std::vector<char> lean((size_t)ntasks, 1);
  return batch_plan(ntasks, tasks, bp, &lean);
}

// Points the descriptors at their tables, counters and partial sums in the
// scratch block; returns the largest number of table entries of a task.
int64_t batch_bind(BatchPlan &bp, char *base) {
  int64_t *tabs = (int64_t *)(base + bp.off_tab);
  int64_t max_entries = 0;
  for (size_t t = 0; t < bp.descs.size(); ++t) {
    if (bp.cfg[t] < 0) continue;
    GemmArgs &a = bp.descs[t].a;
    int64_t *p = tabs + bp.tab_off[t];
    a.mL = p; a.mD = p + a.M; a.nR = a.mD + a.M; a.nD = a.nR + a.N; a.kL = a.nD + a.N; a.kR = a.kL + a.K;
    a.cnt = (int *)(base + bp.off_part + bp.part_off[t]);
    a.part = bp.cfg[t] < kCfgSeq ? (char *)a.cnt + align_up(4 * (int64_t)a.ncnt, 256) : nullptr;
    max_entries = std::max<int64_t>(max_entries, (int64_t)a.M + a.N + a.K);
  }
  return max_entries;
}

// Uploads the descriptors, work lists and prefix sums (the scratch bytes below
// off_tab) as one copy, then launches the table build, one persistent kernel
// per configuration and the single-task fallbacks.  `stage`, when given, is a
// pinned host block of at least off_tab bytes that stays untouched until the
// copy has run; otherwise the block is packed in pageable memory.
int batch_run(int ntasks, const tcContractTask *tasks, BatchPlan &bp, void *scratch, size_t scratch_bytes,
              void *stage, cudaStream_t st) {
  if (scratch == nullptr || scratch_bytes < bp.total) return TALSH_INVALID_ARGS;
  char *base = (char *)scratch;
  const int64_t max_entries = batch_bind(bp, base);
  std::vector<char> pageable;
  char *host = (char *)stage;
  if (host == nullptr) {
    pageable.assign(bp.off_tab, 0);
    host = pageable.data();
  }
  std::memcpy(host + bp.off_desc, bp.descs.data(), sizeof(BatchDesc) * ntasks);
  for (int c = 0; c < kNumCfg; ++c) {
    if (bp.list[c].empty()) continue;
    std::memcpy(host + bp.off_list[c], bp.list[c].data(), sizeof(int32_t) * bp.list[c].size());
    std::memcpy(host + bp.off_prefix[c], bp.prefix[c].data(), sizeof(int64_t) * bp.prefix[c].size());
  }
  cudaError_t e = cudaMemcpyAsync(base, host, bp.off_tab, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(base + bp.off_ctr, 0, sizeof(unsigned long long) * kNumCfg, st);
  if (e != cudaSuccess) {
    note_cuda_error("batch descriptor upload", (int)e);
    return TALSH_FAILURE;
  }
  int rc;
  if (max_entries > 0) {
    const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((max_entries + 255) / 256, 16));
    batch_tables_kernel<<<dim3(gx, ntasks), 256, 0, st>>>((const BatchDesc *)(base + bp.off_desc));
    note_launch();
    if ((rc = check_launch("batch_tables_kernel")) != 0) return rc;
  }
  for (int c = 0; c < kNumCfg; ++c)
    if (!bp.list[c].empty() && (rc = launch_cfg(bp, c, base, st)) != 0) return rc;
  for (int t = 0; t < ntasks; ++t) {
    if (bp.cfg[t] >= 0) continue;
    const tcContractTask &x = tasks[t];
    rc = contract_launch(x.data_kind, x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims, x.D, x.L,
                         x.R, x.alpha_re, x.alpha_im, x.conj_bits, x.accumulative,
                         bp.fb_scratch[t] ? base + bp.fb_off[t] : nullptr, bp.fb_scratch[t], (void *)st);
    if (rc) return rc;
  }
  return TALSH_SUCCESS;
}

}  // namespace

// Upper bound of one task's share of a batch's scratch: its descriptor, work
// list and prefix entries, and its offset tables or single-task fallback
// scratch.  A batch needs the sum over its tasks plus batch_fixed_scratch().
// `lean` leaves out the partial sums of a split contracted range.
size_t batch_task_scratch_bound(const tcContractTask &x, bool lean) {
  size_t fb = 0;
  const size_t full = contract_scratch_bytes(x.data_kind, x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank,
                                             x.rdims, &fb);
  Analysis an;
  if (!lean && full > 0 && analyze(x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims, an) == 0) {
    const TableParams &T = an.T;
    if (an.hyper) {  // single-task path inside the batch
      fb = full;
    } else {
      fb += batch_part_bytes(k_split(x.data_kind, T.M, T.N, T.K, 1), x.data_kind, T.M, T.N);
    }
  }
  return sizeof(BatchDesc) + sizeof(int32_t) + sizeof(int64_t) + fb + 256;
}

// Rounding of the blocks (lists and prefix sums to 16 bytes, the others to 256) and the counters.
size_t batch_fixed_scratch() { return (size_t)16 * 256 + 48; }
static_assert(kNumCfg * (2 * 16 + 8 + 8) + 6 * 256 <= 16 * 256 + 48, "the roundings fit");

// Plans a batch, asks `get` for device scratch and a pinned staging block of
// the sizes the plan needs (get returns nullptr to refuse: TRY_LATER), and
// launches it on `stream`.
int batch_launch_with(int ntasks, const tcContractTask *tasks, const std::vector<char> *lean, BatchScratchFn get,
                      void *ctx, void *stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (ntasks == 0) return TALSH_SUCCESS;
  BatchPlan bp;
  int rc = batch_plan(ntasks, tasks, bp, lean);
  if (rc) return rc;
  void *stage = nullptr;
  void *scratch = get(ctx, bp.total, bp.off_tab, &stage);
  if (scratch == nullptr) return TRY_LATER;
  return batch_run(ntasks, tasks, bp, scratch, bp.total, stage, st);
}

}  // namespace tb

extern "C" size_t tcTensorContractBatchScratch(int ntasks, const tcContractTask *tasks) {
  tb::BatchPlan bp;
  if (tb::batch_plan(ntasks, tasks, bp) != TALSH_SUCCESS) return 0;
  return bp.total;
}

extern "C" int tcTensorContractBatch(int ntasks, const tcContractTask *tasks, void *scratch,
                                     size_t scratch_bytes, void *stream) {
  if (ntasks == 0) return TALSH_SUCCESS;
  tb::BatchPlan bp;
  const int rc = tb::batch_plan_for(ntasks, tasks, bp, scratch, scratch_bytes);
  if (rc) return rc;
  return tb::batch_run(ntasks, tasks, bp, scratch, scratch_bytes, nullptr, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Graph-captured batches: the plan, the descriptor upload and the offset
// tables are done once at creation; the GEMM work is captured in one CUDA
// graph -- a reset of the work counters, then the persistent kernel of every
// tile configuration (and the single-task fallbacks) as concurrent branches,
// so one configuration's tail overlaps the others' work -- and replayed with
// one launch.  Each tile still runs the code of the single-task kernels, so a
// replay's results equal tcTensorContractBatch's bit for bit.
// ---------------------------------------------------------------------------
struct tcContractBatchGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int ntasks = 0;
  unsigned launches = 0;
};

extern "C" int tcContractBatchGraphCreate(int ntasks, const tcContractTask *tasks, void *scratch,
                                          size_t scratch_bytes, void *stream, tcContractBatchGraph **out) {
  using namespace tb;
  if (out == nullptr) return TALSH_INVALID_ARGS;
  *out = nullptr;
  if (ntasks < 1) return TALSH_INVALID_ARGS;
  BatchPlan bp;
  int rc = batch_plan_for(ntasks, tasks, bp, scratch, scratch_bytes);
  if (rc) return rc;
  if (scratch == nullptr || scratch_bytes < bp.total) return TALSH_INVALID_ARGS;
  cudaStream_t st = (cudaStream_t)stream;
  char *base = (char *)scratch;
  // Descriptors, lists and prefix sums, then the offset tables, once.
  const int64_t max_entries = batch_bind(bp, base);
  std::vector<char> host(bp.off_tab, 0);
  std::memcpy(host.data() + bp.off_desc, bp.descs.data(), sizeof(BatchDesc) * ntasks);
  for (int c = 0; c < kNumCfg; ++c) {
    if (bp.list[c].empty()) continue;
    std::memcpy(host.data() + bp.off_list[c], bp.list[c].data(), sizeof(int32_t) * bp.list[c].size());
    std::memcpy(host.data() + bp.off_prefix[c], bp.prefix[c].data(), sizeof(int64_t) * bp.prefix[c].size());
  }
  cudaError_t e = cudaMemcpyAsync(base, host.data(), bp.off_tab, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) {
    note_cuda_error("batch graph descriptor upload", (int)e);
    return TALSH_FAILURE;
  }
  if (max_entries > 0) {
    const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((max_entries + 255) / 256, 16));
    batch_tables_kernel<<<dim3(gx, ntasks), 256, 0, st>>>((const BatchDesc *)(base + bp.off_desc));
    note_launch();
    if ((rc = check_launch("batch_tables_kernel")) != 0) return rc;
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) {  // the host block above goes out of scope
    note_cuda_error("batch graph setup", (int)e);
    return TALSH_FAILURE;
  }
  // Capture on a private stream: counters reset, then one branch per
  // configuration and one for the fallbacks, joined at the end.
  cudaStream_t cs = nullptr;
  std::vector<cudaStream_t> br;
  std::vector<cudaEvent_t> ev;
  cudaGraph_t graph = nullptr;
  unsigned launches = 0;
  auto cleanup = [&]() {
    for (auto x : ev) cudaEventDestroy(x);
    for (auto x : br) cudaStreamDestroy(x);
    if (cs) cudaStreamDestroy(cs);
    cudaGetLastError();
  };
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) { cleanup(); return TALSH_FAILURE; }
  std::vector<int> used;
  for (int c = 0; c < kNumCfg; ++c)
    if (!bp.list[c].empty()) used.push_back(c);
  bool fallbacks = false;
  for (int t = 0; t < ntasks; ++t) fallbacks = fallbacks || bp.cfg[t] < 0;
  const int nbr = (int)used.size() + (fallbacks ? 1 : 0);
  br.assign(nbr, nullptr);
  ev.assign(nbr + 1, nullptr);
  for (auto &x : br)
    if (cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking) != cudaSuccess) { cleanup(); return TALSH_FAILURE; }
  for (auto &x : ev)
    if (cudaEventCreateWithFlags(&x, cudaEventDisableTiming) != cudaSuccess) { cleanup(); return TALSH_FAILURE; }
  if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) { cleanup(); return TALSH_FAILURE; }
  e = cudaMemsetAsync(base + bp.off_ctr, 0, sizeof(unsigned long long) * kNumCfg, cs);
  cudaEventRecord(ev[nbr], cs);
  for (int b = 0; b < nbr; ++b) cudaStreamWaitEvent(br[b], ev[nbr], 0);
  const unsigned before = (unsigned)tcKernelLaunchCount();
  for (size_t b = 0; b < used.size() && rc == TALSH_SUCCESS && e == cudaSuccess; ++b) {
    rc = launch_cfg(bp, used[b], base, br[b]);
  }
  for (int t = 0; t < ntasks && fallbacks && rc == TALSH_SUCCESS && e == cudaSuccess; ++t) {
    if (bp.cfg[t] >= 0) continue;
    const tcContractTask &x = tasks[t];
    rc = contract_launch(x.data_kind, x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims, x.D, x.L,
                         x.R, x.alpha_re, x.alpha_im, x.conj_bits, x.accumulative,
                         bp.fb_scratch[t] ? base + bp.fb_off[t] : nullptr, bp.fb_scratch[t], (void *)br[nbr - 1]);
  }
  launches = (unsigned)tcKernelLaunchCount() - before;
  for (int b = 0; b < nbr; ++b) {
    cudaEventRecord(ev[b], br[b]);
    cudaStreamWaitEvent(cs, ev[b], 0);
  }
  const cudaError_t ce = cudaStreamEndCapture(cs, &graph);
  if (rc == TALSH_SUCCESS && (e != cudaSuccess || ce != cudaSuccess)) {
    note_cuda_error("batch graph capture", (int)(e != cudaSuccess ? e : ce));
    rc = TALSH_FAILURE;
  }
  cudaGraphExec_t exec = nullptr;
  if (rc == TALSH_SUCCESS && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) {
    note_error_text("batch graph instantiation failed");
    rc = TALSH_FAILURE;
  }
  cleanup();
  if (rc != TALSH_SUCCESS) {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    return rc;
  }
  tcContractBatchGraph *g = new tcContractBatchGraph();
  g->graph = graph;
  g->exec = exec;
  g->ntasks = ntasks;
  g->launches = launches;
  *out = g;
  return TALSH_SUCCESS;
}

extern "C" int tcContractBatchGraphLaunch(tcContractBatchGraph *g, void *stream) {
  if (g == nullptr) return TALSH_INVALID_ARGS;
  const cudaError_t e = cudaGraphLaunch(g->exec, (cudaStream_t)stream);
  if (e != cudaSuccess) {
    tb::note_cuda_error("tcContractBatchGraphLaunch", (int)e);
    return TALSH_FAILURE;
  }
  tb::note_launch(g->launches);
  return TALSH_SUCCESS;
}

extern "C" int tcContractBatchGraphDestroy(tcContractBatchGraph *g) {
  if (g == nullptr) return TALSH_INVALID_ARGS;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  delete g;
  return TALSH_SUCCESS;
}

// Autotuner: for every class present among the tasks, runs that class's tasks
// as one batch with each candidate tile (32x32, 64x64), `reps` times each,
// timed with events on `stream`, and keeps the faster tile for the class.
extern "C" int tcTensorContractBatchTune(int ntasks, const tcContractTask *tasks, void *scratch,
                                         size_t scratch_bytes, void *stream, int reps) {
  using namespace tb;
  if (ntasks < 0 || (ntasks > 0 && tasks == nullptr) || reps < 1) return TALSH_INVALID_ARGS;
  {  // as tcTensorContractBatch: partial sums are optional, and both edges have them or neither
    BatchPlan bp;
    const std::vector<char> lean((size_t)ntasks, 1);
    if (ntasks > 0 && (batch_plan(ntasks, tasks, bp, &lean) != TALSH_SUCCESS || scratch_bytes < bp.total))
      return TALSH_INVALID_ARGS;
  }
  std::vector<int> cls[2][kTuneBuckets][kTuneBuckets];
  for (int t = 0; t < ntasks; ++t) {
    const tcContractTask &x = tasks[t];
    if (x.data_kind != R8 && x.data_kind != C8) continue;
    if (x.lrank == 0 || x.rrank == 0) continue;
    Analysis an;
    if (analyze(x.cptrn, x.drank, x.ddims, x.lrank, x.ldims, x.rrank, x.rdims, an) != 0 || an.hyper) continue;
    cls[x.data_kind == C8][tune_bucket(an.T.M)][tune_bucket(an.T.N)].push_back(t);
  }
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
    cudaGetLastError();
    if (e0) cudaEventDestroy(e0);
    return TALSH_FAILURE;
  }
  int rc = TALSH_SUCCESS;
  std::vector<tcContractTask> sub;
  for (int k = 0; k < 2 && rc == TALSH_SUCCESS; ++k)
    for (int mb = 0; mb < kTuneBuckets && rc == TALSH_SUCCESS; ++mb)
      for (int nb = 0; nb < kTuneBuckets && rc == TALSH_SUCCESS; ++nb) {
        const std::vector<int> &ids = cls[k][mb][nb];
        if (ids.empty()) continue;
        sub.clear();
        for (int t : ids) sub.push_back(tasks[t]);
        float best_ms = 0.0f;
        int best = 0;
        for (int edge : {32, 64}) {
          g_tune[k][mb][nb].store(edge);
          float ms = 0.0f;
          for (int r = 0; r <= reps && rc == TALSH_SUCCESS; ++r) {  // the first run warms up
            cudaEventRecord(e0, st);
            rc = tcTensorContractBatch((int)sub.size(), sub.data(), scratch, scratch_bytes, stream);
            cudaEventRecord(e1, st);
            if (rc == TALSH_SUCCESS && cudaEventSynchronize(e1) != cudaSuccess) rc = TALSH_FAILURE;
            float dt = 0.0f;
            if (rc == TALSH_SUCCESS && r > 0 && cudaEventElapsedTime(&dt, e0, e1) == cudaSuccess) ms += dt;
          }
          if (rc != TALSH_SUCCESS) break;
          if (best == 0 || ms < best_ms) { best_ms = ms; best = edge; }
        }
        g_tune[k][mb][nb].store(rc == TALSH_SUCCESS ? best : 0);
      }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaGetLastError();
  return rc;
}

// Tile edge the autotuner chose for a class (0: not tuned), or -1 for a bad class.
extern "C" int tcTensorContractBatchTuned(int data_kind, int m_bucket, int n_bucket) {
  using namespace tb;
  if ((data_kind != R8 && data_kind != C8) || m_bucket < 0 || m_bucket >= kTuneBuckets || n_bucket < 0 ||
      n_bucket >= kTuneBuckets)
    return -1;
  return g_tune[data_kind == C8][m_bucket][n_bucket].load();
}

// Forgets every tuned choice (the shape rule applies again).
extern "C" void tcTensorContractBatchTuneReset(void) {
  using namespace tb;
  for (auto &a : g_tune)
    for (auto &b : a)
      for (auto &c : b) c.store(0);
}
