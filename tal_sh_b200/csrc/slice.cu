// Tensor slicing and insertion (tcTensorSlice / tcTensorInsert): copies between
// a dense column-major tensor and a rectangular sub-block of another one.
//
// Reference: talshTensorSlice / talshTensorInsert (talshc.cpp:4008-4268,
// :4269-4528) run only on the CPU there (tensor_block_slice_dlf_r8
// tensor_algebra_cpu.F90:6900-6974, tensor_block_insert_dlf_r8 :7216-7290,
// slice = slice*beta + tensor*alpha with alpha = 1, beta = 1 when
// accumulative else 0); its GPU entry points gpu_tensor_block_slice/insert are
// unimplemented stubs (tensor_algebra_gpu_nvidia.cu:4788-4804).
//
// Layout: leading dimensions that the slice covers completely fuse with the
// first partially covered one into one contiguous run (the same bytes in both
// tensors); the remaining slice dimensions index runs.  Pure data movement
// (memory-bound): 2 * slice volume * element size bytes, 3 * ... when
// accumulating.  The slice is walked element by element (or by 8- or 16-byte
// vectors where every run allows it) in its own order, four in flight per
// thread, each finding its run by 32-bit magic division: lanes stay full for
// any run length.  (A warp per run, one element in flight per lane and 64-bit
// divisions per run, took 56 us for a 71 x 44 x 53 x 60 R8 block, 81 MB, and 62
// us for adding it back; now 36 and 45 us.)
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <cstring>

#include "common.h"

namespace tb {
namespace {

constexpr int kSliceThreads = 256;

struct SliceParams {
  int nrow;                       // run dimensions, at most kMaxRank
  int64_t run;                    // contiguous units per run
  int64_t total;                  // units of the slice
  int64_t base;                   // full-tensor offset of the slice origin
  int64_t full;                   // units of the full tensor
  int64_t rext[kMaxRank];         // slice extents of the run dimensions
  int64_t rstr[kMaxRank];         // full-tensor strides of the run dimensions
  uint32_t mg_run, sh_run, mg[kMaxRank], sh[kMaxRank];  // magic divisors (totals below 2^31)
};

// Round-up magic division of n < 2^31 (Granlund and Montgomery).
void magic(int64_t d, uint32_t &mg, uint32_t &sh) {
  const uint32_t s = d > 1 ? 64 - __builtin_clzll((uint64_t)d - 1) : 0;  // ceil(log2 d)
  mg = d > 1 ? (uint32_t)(((1ull << 32) * ((1ull << s) - (uint64_t)d)) / (uint64_t)d + 1ull) : 1u;
  sh = s;
}
__device__ __forceinline__ uint32_t mdiv(uint32_t n, uint32_t mg, uint32_t sh) { return (__umulhi(n, mg) + n) >> sh; }

// A unit: VEC values of a real type (complex values are two).
template <typename R, int VEC> struct alignas(sizeof(R) * VEC) Unit { R v[VEC]; };

// Arithmetic of unit numbers and full-tensor offsets: 32 bits for both, 32 and
// 64, or 64 for both.
enum : int { kNarrow = 0, kMixed = 1, kWide = 2 };
template <int MODE>
__device__ __forceinline__ int64_t full_offset(const SliceParams &p, int64_t e) {
  if constexpr (MODE == kWide) {
    int64_t r = e / p.run;
    int64_t off = p.base + (e - r * p.run);
    for (int d = 0; d < p.nrow; ++d) {
      const int64_t q = r / p.rext[d];
      off += (r - q * p.rext[d]) * p.rstr[d];
      r = q;
    }
    return off;
  } else {
    using O = std::conditional_t<MODE == kNarrow, uint32_t, int64_t>;
    uint32_t r = mdiv((uint32_t)e, p.mg_run, p.sh_run);
    O off = (O)p.base + ((uint32_t)e - r * (uint32_t)p.run);
    for (int d = 0; d + 1 < p.nrow; ++d) {
      const uint32_t q = mdiv(r, p.mg[d], p.sh[d]);
      off += (O)(r - q * (uint32_t)p.rext[d]) * (O)p.rstr[d];
      r = q;
    }
    return p.nrow > 0 ? off + (O)r * (O)p.rstr[p.nrow - 1] : off;  // r is below the last extent
  }
}

// INSERT = false: slice[e] (+)= full[map(e)]; true: full[map(e)] (+)= slice[e].
template <typename R, int VEC, bool INSERT, bool ACC, int MODE>
__global__ void __launch_bounds__(kSliceThreads) slice_kernel(const Unit<R, VEC> *__restrict__ src,
                                                              Unit<R, VEC> *dst, const SliceParams p) {
  constexpr int U = 4;
  const int64_t step = (int64_t)gridDim.x * (kSliceThreads * U);
  for (int64_t e0 = (int64_t)blockIdx.x * (kSliceThreads * U) + threadIdx.x; e0 < p.total; e0 += step) {
    Unit<R, VEC> x[U], y[U];
    int64_t f[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t e = e0 + u * kSliceThreads;
      if (e >= p.total) continue;
      f[u] = full_offset<MODE>(p, e);
      x[u] = src[INSERT ? e : f[u]];
      if (ACC) y[u] = dst[INSERT ? f[u] : e];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t e = e0 + u * kSliceThreads;
      if (e >= p.total) continue;
      if (ACC) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) x[u].v[j] = y[u].v[j] + x[u].v[j];
      }
      dst[INSERT ? f[u] : e] = x[u];
    }
  }
}

template <typename R, int VEC, bool INSERT, bool ACC>
int launch(const void *src, void *dst, const SliceParams &p, cudaStream_t st) {
  const int64_t want = (p.total + kSliceThreads * 4 - 1) / (kSliceThreads * 4);
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)current_sm_count() * 32));
  const auto *s = (const Unit<R, VEC> *)src;
  auto *d = (Unit<R, VEC> *)dst;
  const int64_t lim = int64_t(1) << 31;
  if (p.total >= lim) slice_kernel<R, VEC, INSERT, ACC, kWide><<<blocks, kSliceThreads, 0, st>>>(s, d, p);
  else if (p.full >= lim) slice_kernel<R, VEC, INSERT, ACC, kMixed><<<blocks, kSliceThreads, 0, st>>>(s, d, p);
  else slice_kernel<R, VEC, INSERT, ACC, kNarrow><<<blocks, kSliceThreads, 0, st>>>(s, d, p);
  note_launch();
  return check_launch(INSERT ? "tensor insert" : "tensor slice");
}

template <typename R, int VEC>
int dispatch(bool insert, bool acc, const void *src, void *dst, const SliceParams &p, cudaStream_t st) {
  if (insert) return acc ? launch<R, VEC, true, true>(src, dst, p, st) : launch<R, VEC, true, false>(src, dst, p, st);
  return acc ? launch<R, VEC, false, true>(src, dst, p, st) : launch<R, VEC, false, false>(src, dst, p, st);
}

int slice_op(bool insert, int kind, int rank, const int *full_dims, const int *slice_dims, const int *offsets,
             const void *src, void *dst, int accumulative, void *stream) {
  if (kind_size(kind) == 0 || rank < 1 || rank > kMaxRank || full_dims == nullptr || slice_dims == nullptr ||
      offsets == nullptr || src == nullptr || dst == nullptr)
    return TALSH_INVALID_ARGS;
  if (!elem_aligned(kind, src) || !elem_aligned(kind, dst)) return TALSH_INVALID_ARGS;
  for (int i = 0; i < rank; ++i)
    if (full_dims[i] <= 0 || slice_dims[i] <= 0 || offsets[i] < 0 || offsets[i] + (int64_t)slice_dims[i] > full_dims[i])
      return TALSH_INVALID_ARGS;
  SliceParams p;
  std::memset(&p, 0, sizeof(p));
  // Run: leading fully covered dimensions plus the first partial one.
  int64_t stride = 1, base = 0;
  int d = 0;
  p.run = 1;
  while (d < rank) {
    base += (int64_t)offsets[d] * stride;
    p.run *= slice_dims[d];
    const bool full = slice_dims[d] == full_dims[d];
    stride *= full_dims[d];
    ++d;
    if (!full) break;
  }
  p.total = p.run;
  for (; d < rank; ++d) {
    base += (int64_t)offsets[d] * stride;
    p.total *= slice_dims[d];
    if (slice_dims[d] > 1) {
      const int k = p.nrow - 1;
      if (k >= 0 && stride == p.rstr[k] * p.rext[k]) {  // continues the previous run dimension
        p.rext[k] *= slice_dims[d];
      } else {
        p.rext[p.nrow] = slice_dims[d];
        p.rstr[p.nrow] = stride;
        p.nrow++;
      }
    }
    stride *= full_dims[d];
  }
  p.base = base;
  // Widest unit that divides every run and starts every run aligned in both tensors.
  const int es = kind_size(kind);
  int vec = 16 / es;
  auto fits = [&](int v) {
    if (((uintptr_t)src | (uintptr_t)dst) % ((uintptr_t)v * es) || p.run % v || p.base % v) return false;
    for (int k = 0; k < p.nrow; ++k)
      if (p.rstr[k] % v) return false;
    return true;
  };
  while (vec > 1 && !fits(vec)) vec /= 2;
  p.run /= vec;
  p.base /= vec;
  p.total /= vec;
  p.full = stride / vec;
  for (int k = 0; k < p.nrow; ++k) p.rstr[k] /= vec;
  magic(p.run, p.mg_run, p.sh_run);
  for (int k = 0; k + 1 < p.nrow; ++k) magic(p.rext[k], p.mg[k], p.sh[k]);
  const bool acc = accumulative != 0;
  cudaStream_t st = (cudaStream_t)stream;
  // values per unit: float 1, 2, 4; double 1, 2
  const bool single = kind == R4 || kind == C4;
  const int n = vec * es / (single ? 4 : 8);
  if (single) {
    if (n == 4) return dispatch<float, 4>(insert, acc, src, dst, p, st);
    if (n == 2) return dispatch<float, 2>(insert, acc, src, dst, p, st);
    return dispatch<float, 1>(insert, acc, src, dst, p, st);
  }
  if (n == 2) return dispatch<double, 2>(insert, acc, src, dst, p, st);
  return dispatch<double, 1>(insert, acc, src, dst, p, st);
}

}  // namespace
}  // namespace tb

extern "C" int tcTensorSlice(int data_kind, int rank, const int *full_dims, const int *slice_dims,
                             const int *offsets, const void *full, void *slice, int accumulative, void *stream) {
  return tb::slice_op(false, data_kind, rank, full_dims, slice_dims, offsets, full, slice, accumulative, stream);
}

extern "C" int tcTensorInsert(int data_kind, int rank, const int *full_dims, const int *slice_dims,
                              const int *offsets, const void *slice, void *full, int accumulative, void *stream) {
  return tb::slice_op(true, data_kind, rank, full_dims, slice_dims, offsets, slice, full, accumulative, stream);
}
