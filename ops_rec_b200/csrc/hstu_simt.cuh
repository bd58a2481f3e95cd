// Register-tiled fp32 building blocks of the CUDA-core attention kernels (forward: hstu_generic.cu, backward:
// hstu_bwd_generic.cu): the path of fp32 inputs, whose 1e-5 tolerance rules out TF32 tensor cores, and of the 16-bit
// calls the tensor-core kernels do not take.
//
// What bounds such a kernel is shared-memory bandwidth, not the FMA pipe: with one element of the result per thread
// every FMA needs an operand from shared memory.  Here 128 threads hold a 32 x BN tile of scores, 4 x BN/16 values each
// (rows 4 ty + r, columns tx + 16 c), so a step of four along the reduction is 4 + BN/16 16-byte loads for 16 BN/16 x 4
// FMAs; the row pitch (dim + 4 floats) puts the 16-byte pieces of eight consecutive rows on different banks.  Tiles
// have 32 rows, not 64: a batch of a few short sequences then still gives every SM two or three CTAs, and the longest
// chain of dependent K tiles - what such a batch's time is - halves.  Tiles of fp32 inputs are fetched with cp.async, the
// next tile of an operand as soon as its last reader is through.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"

namespace hstu {
namespace simt {

constexpr int kRows = 32;      // rows of the resident tile
constexpr int kThreads = 128;  // 16 x 8 threads
constexpr int kMaxDim = 128;

template <typename T> __device__ __forceinline__ float to_float(T x);
template <> __device__ __forceinline__ float to_float<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_float<__half>(__half x) { return __half2float(x); }
template <typename T> __device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_float<__half>(float x) { return __float2half_rn(x); }
template <typename T> __device__ __forceinline__ float rounded(float x) { return to_float<T>(from_float<T>(x)); }

// a / b for b >= 1 with the remainder correction of Markstein ("Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  r = (1 + d) / b with |d| <= 2^-23 (the documented error of rcp.approx), so q = a r is
// within 2^-22 of a / b; its remainder a - q b comes exact out of one FMA, and q + rem r = a / b up to |d| 2^-22 |a / b|
// before the one rounding at the end: half an ulp, and 2^-21 of one.  (Beyond b = 2^126 r is subnormal, which costs up to
// two bits of d: half an ulp, and 2^-17 of one.)  An infinite a or b keeps the uncorrected quotient: what the division
// gives; a zero comes out positive.  The division itself costs 16 % of a training step in fp32 (157 -> 182 us) and changes no error: against 64 bits
// it is the sums of a row that count.
__device__ __forceinline__ float divide(float a, float b) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b));
  const float q = a * r, rem = fmaf(-q, b, a);
  const float c = fmaf(rem, r, q);
  return c == c ? c : q;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Rows [r0, r0 + kTileRows) of head h of a [tokens, heads, dim] tensor -> dst[kTileRows][ld] in fp32, zeros past `len`.
// dim is a multiple of 4 up to kDim and the rows are aligned to four elements.  fp32: cp.async (the caller commits and
// waits); 16-bit: plain loads and stores.
template <typename T, int kTileRows, int kDim>
__device__ __forceinline__ void load_rows(float* dst, int ld, const T* src, long long tok0, int r0, int len, int heads,
                                          int h, int dim) {
  constexpr int kPieces = kDim / 4;                   // 4-element pieces per row
  constexpr int kRowStep = kThreads / kPieces;
  const int d = (threadIdx.x % kPieces) * 4;
  if (d >= dim) return;
#pragma unroll 4
  for (int r = threadIdx.x / kPieces; r < kTileRows; r += kRowStep) {
    const int row = r0 + r;
    const bool in = row < len;
    const T* from = in ? src + ((tok0 + row) * heads + h) * dim + d : src;
    float* to = dst + r * ld + d;
    if constexpr (sizeof(T) == 4) {
      const uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(to));
      const int bytes = in ? 16 : 0;                  // (0: zero-filled, nothing is read)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(addr), "l"(from), "r"(bytes) : "memory");
    } else {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (in) {
        const uint2 u = *reinterpret_cast<const uint2*>(from);
        const T* e = reinterpret_cast<const T*>(&u);
        v = make_float4(to_float<T>(e[0]), to_float<T>(e[1]), to_float<T>(e[2]), to_float<T>(e[3]));
      }
      *reinterpret_cast<float4*>(to) = v;
    }
  }
}

// acc[r][c] = sum over d of A[4 ty + r][d] * B[tx + 16 c][d]; dim a multiple of 4.  Even and odd d are summed apart
// (packed FMAs) and added at the end.
template <int kCols>
__device__ __forceinline__ void dot_tile(const float* a, int lda, const float* b, int ldb, int dim, float (&acc)[4][kCols]) {
  float2 sum[4][kCols];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < kCols; ++c) sum[r][c] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int d = 0; d < dim; d += 4) {
    float4 av[4], bv[kCols];
#pragma unroll
    for (int r = 0; r < 4; ++r) av[r] = *reinterpret_cast<const float4*>(a + r * lda + d);
#pragma unroll
    for (int c = 0; c < kCols; ++c) bv[c] = *reinterpret_cast<const float4*>(b + 16 * c * ldb + d);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        sum[r][c] = __ffma2_rn(make_float2(av[r].x, av[r].y), make_float2(bv[c].x, bv[c].y), sum[r][c]);
        sum[r][c] = __ffma2_rn(make_float2(av[r].z, av[r].w), make_float2(bv[c].z, bv[c].w), sum[r][c]);
      }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < kCols; ++c) acc[r][c] = sum[r][c].x + sum[r][c].y;
}

// Columns of the output a thread owns: kDim / 16 of them, in vectors of up to four.
template <int kDim> struct OutCols {
  static constexpr int kPer = kDim / 16;                    // 2, 4, 8
  static constexpr int kVec = kPer < 4 ? kPer : 4;          // contiguous columns per vector
  static constexpr int kVecs = kPer / kVec;
  static __device__ __forceinline__ int col(int tx, int v) { return v * 64 + tx * kVec; }
};

// acc[r][.] += sum over k < kend of P[4 ty + r][k] * B[k][own columns]; kend a multiple of 4.
template <int kDim>
__device__ __forceinline__ void outer_tile(const float* pm, int ldp, const float* b, int ldb, int kend, int tx,
                                           float (&acc)[4][OutCols<kDim>::kPer]) {
  using C = OutCols<kDim>;
#pragma unroll 2
  for (int k = 0; k < kend; k += 4) {
    float4 pv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) pv[r] = *reinterpret_cast<const float4*>(pm + r * ldp + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float bv[C::kPer];
#pragma unroll
      for (int v = 0; v < C::kVecs; ++v) {
        const float* from = b + (k + kk) * ldb + C::col(tx, v);
        if constexpr (C::kVec == 4) {
          const float4 x = *reinterpret_cast<const float4*>(from);
          bv[4 * v] = x.x, bv[4 * v + 1] = x.y, bv[4 * v + 2] = x.z, bv[4 * v + 3] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(from);
          bv[0] = x.x, bv[1] = x.y;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float pe = kk == 0 ? pv[r].x : kk == 1 ? pv[r].y : kk == 2 ? pv[r].z : pv[r].w;
#pragma unroll
        for (int c = 0; c < C::kPer; ++c) acc[r][c] = fmaf(pe, bv[c], acc[r][c]);
      }
    }
  }
}

// The thread's columns of one output row; dim a multiple of 4, row aligned to four elements.
template <typename T, int kDim>
__device__ __forceinline__ void store_row(T* row, int dim, int tx, const float (&acc)[OutCols<kDim>::kPer]) {
  using C = OutCols<kDim>;
#pragma unroll
  for (int v = 0; v < C::kVecs; ++v) {
    const int col = C::col(tx, v);
    if (col >= dim) continue;
    alignas(16) T e[C::kVec];
#pragma unroll
    for (int i = 0; i < C::kVec; ++i) e[i] = from_float<T>(acc[v * C::kVec + i]);
    if constexpr (sizeof(T) * C::kVec == 16) *reinterpret_cast<uint4*>(row + col) = *reinterpret_cast<const uint4*>(e);
    else if constexpr (sizeof(T) * C::kVec == 8) *reinterpret_cast<uint2*>(row + col) = *reinterpret_cast<const uint2*>(e);
    else *reinterpret_cast<uint32_t*>(row + col) = *reinterpret_cast<const uint32_t*>(e);
  }
}

// Head dims and alignment these kernels take: whole 4-element pieces, at most kMaxDim wide.
inline bool dims_ok(const KParams& p) {
  return p.dqk % 4 == 0 && p.dv % 4 == 0 && p.dqk >= 4 && p.dv >= 4 && p.dqk <= kMaxDim && p.dv <= kMaxDim;
}
inline bool aligned_to(const void* ptr, int dtype) {
  return (reinterpret_cast<uintptr_t>(ptr) & (dtype == HSTU_DTYPE_FP32 ? 15u : 7u)) == 0;
}
inline int tile_dim(const KParams& p) {
  const int d = p.dqk > p.dv ? p.dqk : p.dv;
  return d <= 32 ? 32 : d <= 64 ? 64 : 128;
}

// Launched with programmatic stream serialization: the pre-pass in front only checks the inputs (its status word), so
// the kernel need not wait for it before its end; nor the second backward kernel for the first.
template <typename... P, typename... A>
cudaError_t launch(void (*kern)(P...), dim3 grid, int smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace simt
}  // namespace hstu
