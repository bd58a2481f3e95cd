// in_linear_silu backward: gradients of  (user, value, query, key) = split(silu(x . weight^T + bias))  with respect
// to x, weight and bias, given the forward's saved linear_output.
//
// Reference operator ops_rec::in_linear_silu_backward
// (ascendc/activation/in_linear_silu/torch_extension/in_linear_silu_backward_plugin.cpp:118-152; definition of the
// result in in_linear_silu_backward/test/pytest/test_in_linear_silu_backward.py:125-171):
//     g   = cat(user_grad, value_grad, query_grad, key_grad)                    [m, n]
//     dL  = g * sig * (1 + lo * (1 - sig)),  sig = sigmoid(lo), lo = linear_output      fp32
//     bias_grad = column sums of dL (fp32);  dL is then rounded to the element type
//     x_grad = dL . weight  [m, k];   weight_grad = dL^T . x  [n, k]            fp32 accumulation, one rounding
//
//   silu_grad_kernel   one read of g and linear_output -> dL [m, n] + per-row-block column sums of dL; HBM-bound
//   colsum_kernel      the row-block sums -> bias_grad, in a fixed order (bitwise reproducible; no atomics)
//   launch_product     x_grad = dL . weight and weight_grad = dL^T . x on the forward's tcgen05 pipeline, which reads
//                      dL, weight and x as they lie.  (Forward + backward of 65536 rows of width 1024: 2323 us with transposed
//                      copies of all three and one-CTA tiles, 1760 us)
// All intermediates live in the caller's workspace.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"

namespace hstu {

uint64_t product_partial_bytes(long long m, int n, long long k);
cudaError_t launch_product(const void* a, bool trans_a, const void* b, long long m, int n, long long k, void* out,
                           float* partial, int dtype, uint32_t* status, cudaStream_t stream);

namespace {

constexpr int kBtThreads = 256;
constexpr int kBtCols = 256;     // columns of an element-wise CTA: 32 lanes x 8
constexpr int kSumGroups = 8;    // row-block groups a column sum is added up in

template <typename T> struct Cvt;
template <> struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float2 up(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u)); }
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};
template <> struct Cvt<__half> {
  static __device__ __forceinline__ float2 up(uint32_t u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }
  static __device__ __forceinline__ uint32_t down(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
};

struct SiluGradParams {
  const void* grad[4];     // user / value / query / key gradients, [m, width[i]]
  int width[4], start[5];  // column range of each in the concatenated [m, n]
  const void* lo;          // linear_output [m, n]
  void* dl;                // [m, n]
  float* partial;          // [ceil(m / rows), n] column sums per row block
  long long m;
  int n, rows;             // rows: rows per CTA, a multiple of 32
};

// sigmoid(x) from one ex2 and one reciprocal (each within 2 ulp; the result feeds a 16-bit rounding or a column sum).  Against
// 64 bits bias_grad is 1.0e-7 off for 64 rows, 2.0e-7 for 65536; with a division, and 64-row blocks added one after the
// other, it was 1.3e-7 and 5.9e-7.  An IEEE reciprocal here costs 60 us of forward and backward of 65536 rows.
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

// p.rows x 256 columns of [m, n] per CTA: a thread owns 8 columns and every eighth row of the block, four rows' loads in
// flight.  (An IEEE division per element made this pass issue-bound: two SFU operations and about ten others are left.)
template <typename T>
__global__ void __launch_bounds__(kBtThreads) silu_grad_kernel(const SiluGradParams p) {
  __shared__ float s_part[kBtThreads / 32][kBtCols];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * kBtCols + lane * 8;
  const long long r0 = static_cast<long long>(blockIdx.y) * p.rows;
  const long long r1 = r0 + p.rows < p.m ? r0 + p.rows : p.m;
  float csum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col < p.n) {
    const int which = (col >= p.start[1]) + (col >= p.start[2]) + (col >= p.start[3]);
    const int w = which == 0 ? p.width[0] : which == 1 ? p.width[1] : which == 2 ? p.width[2] : p.width[3];
    const int st = which == 0 ? p.start[0] : which == 1 ? p.start[1] : which == 2 ? p.start[2] : p.start[3];
    const T* g = static_cast<const T*>(which == 0 ? p.grad[0] : which == 1 ? p.grad[1] : which == 2 ? p.grad[2] : p.grad[3]) +
                 (col - st);
    const T* lo = static_cast<const T*>(p.lo) + col;
    T* dl = static_cast<T*>(p.dl) + col;
    for (long long row = r0 + warp; row < r1; row += 32) {
      uint4 gv[4], lv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long long r = row + 8 * i;
        if (r < r1) {
          gv[i] = __ldcs(reinterpret_cast<const uint4*>(g + r * w));
          lv[i] = __ldcs(reinterpret_cast<const uint4*>(lo + r * p.n));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long long r = row + 8 * i;
        if (r >= r1) break;
        const uint32_t gw[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w}, lw[4] = {lv[i].x, lv[i].y, lv[i].z, lv[i].w};
        uint32_t ow[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 g2 = Cvt<T>::up(gw[e]), l2 = Cvt<T>::up(lw[e]);
          const float s0 = sigmoid_f(l2.x), s1 = sigmoid_f(l2.y);
          const float d0 = g2.x * (s0 * (1.f + l2.x * (1.f - s0))), d1 = g2.y * (s1 * (1.f + l2.y * (1.f - s1)));
          csum[2 * e] += d0;
          csum[2 * e + 1] += d1;
          ow[e] = Cvt<T>::down(d0, d1);
        }
        *reinterpret_cast<uint4*>(dl + r * p.n) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
  }
  // column sums of the block: the warps' sums in a fixed order
#pragma unroll
  for (int e = 0; e < 8; ++e) s_part[warp][lane * 8 + e] = csum[e];
  __syncthreads();
  const int c = blockIdx.x * kBtCols + threadIdx.x;
  if (c < p.n) {
    float acc = 0.f;
#pragma unroll
    for (int r = 0; r < kBtThreads / 32; ++r) acc += s_part[r][threadIdx.x];
    p.partial[static_cast<long long>(blockIdx.y) * p.n + c] = acc;
  }
}

// bias_grad[c] = sum over the row blocks: eight groups of consecutive blocks, each in block order, then the groups
__global__ void __launch_bounds__(32 * kSumGroups) colsum_kernel(const float* __restrict__ partial, float* __restrict__ out,
                                                                 long long blocks, int n) {
  __shared__ float s_sum[kSumGroups][32];
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  const long long per = (blocks + kSumGroups - 1) / kSumGroups;
  const long long b1 = (group + 1) * per < blocks ? (group + 1) * per : blocks;
  float acc = 0.f;
  if (c < n) {
#pragma unroll 8
    for (long long b = group * per; b < b1; ++b) acc += partial[b * n + c];
  }
  s_sum[group][lane] = acc;
  __syncthreads();
  if (group == 0 && c < n) {
#pragma unroll
    for (int i = 1; i < kSumGroups; ++i) acc += s_sum[i][lane];
    out[c] = acc;
  }
}

// Rows per CTA of the element-wise pass: 128, or 32 where that leaves fewer than four CTAs per SM of a B200.
inline int block_rows(long long m, int n) {
  const long long ctas = (m + 127) / 128 * ((n + kBtCols - 1) / kBtCols);
  return ctas < 4 * 148 ? 32 : 128;
}

inline uint64_t up256(uint64_t x) { return (x + 255) & ~static_cast<uint64_t>(255); }

inline uint64_t max_u64(uint64_t a, uint64_t b) { return a > b ? a : b; }

}  // namespace

// Workspace bytes of the backward for an [m, k] x, [n, k] weight: dL, the column sums, and (one product after the
// other) the partial sums of a product that is split along its contraction.
uint64_t in_linear_silu_bwd_workspace(long long m, int n, int k) {
  const int rows = block_rows(m, n);
  return up256(static_cast<uint64_t>(m) * n * 2) + up256(static_cast<uint64_t>((m + rows - 1) / rows) * n * 4) +
         up256(max_u64(product_partial_bytes(m, k, n), product_partial_bytes(n, k, m)));
}

// grads: the four output gradients; lo: linear_output; every tensor 16-byte aligned; bias_grad fp32 [n] or null.
cudaError_t launch_in_linear_silu_bwd(const LinSiluParams& shape, const void* x, const void* weight,
                                      const void* const grads[4], const void* lo, void* x_grad, void* weight_grad,
                                      float* bias_grad, void* workspace, int dtype, uint32_t* status,
                                      cudaStream_t stream) {
  const long long m = shape.m;
  const int n = shape.n, k = shape.k;
  if (m == 0) return cudaSuccess;
  SiluGradParams sp;
  sp.rows = block_rows(m, n);
  const long long row_blocks = (m + sp.rows - 1) / sp.rows;
  if (row_blocks > 65535) return cudaErrorInvalidConfiguration;  // (the entry point takes at most 4 194 240 rows)
  char* ws = static_cast<char*>(workspace);
  sp.dl = ws;
  ws += up256(static_cast<uint64_t>(m) * n * 2);
  sp.partial = reinterpret_cast<float*>(ws);
  ws += up256(static_cast<uint64_t>(row_blocks) * n * 4);
  float* partial = reinterpret_cast<float*>(ws);
  for (int i = 0; i < 4; ++i) {
    sp.grad[i] = grads[i];
    sp.width[i] = shape.width[i];
  }
  for (int i = 0; i < 5; ++i) sp.start[i] = shape.start[i];
  sp.lo = lo;
  sp.m = m;
  sp.n = n;
  const dim3 grid((n + kBtCols - 1) / kBtCols, static_cast<unsigned>(row_blocks));
  if (dtype == HSTU_DTYPE_BF16)
    silu_grad_kernel<__nv_bfloat16><<<grid, kBtThreads, 0, stream>>>(sp);
  else
    silu_grad_kernel<__half><<<grid, kBtThreads, 0, stream>>>(sp);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (bias_grad) {
    colsum_kernel<<<(n + 31) / 32, 32 * kSumGroups, 0, stream>>>(sp.partial, bias_grad, row_blocks, n);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  // x_grad [m, k] = dL [m, n] . weight [n, k];  weight_grad [n, k] = dL^T . x [m, k]
  e = launch_product(sp.dl, false, weight, m, k, n, x_grad, partial, dtype, status, stream);
  if (e != cudaSuccess) return e;
  return launch_product(sp.dl, true, x, n, k, m, weight_grad, partial, dtype, status, stream);
}

}  // namespace hstu
