// HSTU jagged forward on CUDA cores: fp32 products and fp32 accumulation for every input type - the path of fp32
// inputs (the 1e-5 tolerance rules out TF32 tensor cores) and of the 16-bit calls hstu_tc.cu does not take.
// One CTA owns a 32-row q-tile of one (sequence, head), walks the K tiles the composite mask leaves visible
// (hstu_dense_forward_jagged_kernel.h:285-289 ends a row at the first fully masked tile; so does this),
// and writes its rows of the jagged output once - no atomics, no zero-initialised output.
//
//   hstu_simt_fwd_kernel   register-tiled (hstu_simt.cuh): head dims that are multiples of 4 up to 128, aligned rows
//   hstu_generic_kernel    any dims up to 512, any alignment: one score per thread and row, operands read from shared
//                          memory for every FMA
//
// Reference arithmetic being reproduced (…/op_kernel/atlas950/hstu_dense_forward_kernel_patten_bsnd.h:258-326,
// regbase_silu.h:21-40): x = alpha * (S + bias); P = x / (1 + exp(-x)) * scale, exactly 0 where masked; P is
// rounded to the input type before P.V; the result is rounded to the input type.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"
#include "hstu_simt.cuh"

namespace hstu {

namespace {

constexpr int GM = 32;       // q rows per CTA
constexpr int GN = 32;       // keys per tile
constexpr int GTHREADS = 256;
constexpr int GROWS = 4;     // rows per thread (GM / 8 warps)
constexpr int GMAXC = 16;    // dv <= 512 -> at most 16 output columns per thread

template <typename T> __device__ __forceinline__ float to_f(T x) { return simt::to_float<T>(x); }
template <typename T> __device__ __forceinline__ T from_f(float x) { return simt::from_float<T>(x); }

constexpr int kFwdKeys = 64;   // keys per tile of the register-tiled kernel

// See hstu_simt.cuh for the tile shape and what bounds it.  K_t is read by the scores only and V_t by the output only,
// so each is fetched again while the other's products run.
template <typename T, int kDim>
__global__ void __launch_bounds__(simt::kThreads) hstu_simt_fwd_kernel(const KParams p) {
  extern __shared__ float smem[];
  constexpr int kCols = kFwdKeys / 16;
  constexpr int kPer = simt::OutCols<kDim>::kPer;
  constexpr int ldq = kDim + 4, ldp = kFwdKeys + 4;
  const int b = blockIdx.x / p.hq, h = blockIdx.x - b * p.hq;
  const int hk = h / p.gqa_ratio;
  const int r0 = static_cast<int>(gridDim.y - 1 - blockIdx.y) * simt::kRows;   // the rows with the most keys first
  const SeqInfo s = load_seq(p, b);
  if (r0 < s.lq) {
    const int dq = p.dqk, dv = p.dv;
    float* Qs = smem;                        // [32][ldq]
    float* Ks = Qs + simt::kRows * ldq;      // [64][ldq]
    float* Vs = Ks + kFwdKeys * ldq;         // [64][kDim]
    float* Ps = Vs + kFwdKeys * kDim;        // [32][ldp]
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const T* k = static_cast<const T*>(p.k);
    const T* v = static_cast<const T*>(p.v);
    const T* bias = static_cast<const T*>(p.bias);
    const T* cmask = static_cast<const T*>(p.mask);
    const bool alpha_first = (p.flags & HSTU_FLAG_ALPHA_BEFORE_BIAS) != 0;
    RowBounds rb[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = r0 + 4 * ty + r;
      rb[r] = row_bounds(s, i, p.mask_type, p.group);
      if (i >= s.lq) rb[r].lim1 = 0, rb[r].lo2 = 1, rb[r].hi2 = 0;   // (a row past the end sees nothing)
    }
    // keys any row of the q-tile sees, rounded up to the q-tile's height
    const int seen = kv_tiles_for_rows(s, r0, simt::kRows, p.mask_type, 32) * 32;
    const int end = seen < s.lk ? seen : s.lk;
    const int ntiles = (end + kFwdKeys - 1) / kFwdKeys;
    float acc[4][kPer];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < kPer; ++c) acc[r][c] = 0.f;
    simt::load_rows<T, simt::kRows, kDim>(Qs, ldq, static_cast<const T*>(p.q), s.q0, r0, s.lq, p.hq, h, dq);
    if (ntiles > 0) simt::load_rows<T, kFwdKeys, kDim>(Ks, ldq, k, s.k0, 0, s.lk, p.hk, hk, dq);
    simt::cp_async_commit();
    if (ntiles > 0) simt::load_rows<T, kFwdKeys, kDim>(Vs, kDim, v, s.k0, 0, s.lk, p.hk, hk, dv);
    simt::cp_async_commit();
    for (int t = 0; t < ntiles; ++t) {
      const int c0 = t * kFwdKeys;
      float bv[4][kCols];
      if (bias) {   // (in flight while the scores are computed)
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            const int i = r0 + 4 * ty + r, j = c0 + tx + 16 * c;
            bv[r][c] = allowed(rb[r], j) ? to_f<T>(bias[static_cast<long long>(b) * p.bias_bstride +
                                                        (static_cast<long long>(h) * p.maxq + i) * p.maxk + j])
                                         : 0.f;
          }
      }
      simt::cp_async_wait<1>();   // K_t (and, first time, Q)
      __syncthreads();
      float sc[4][kCols];
      simt::dot_tile<kCols>(Qs + 4 * ty * ldq, ldq, Ks + tx * ldq, ldq, dq, sc);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int i = r0 + 4 * ty + r, j = c0 + tx + 16 * c;
          // (no branch per element: sixteen of them in a row were a third of a tile's time)
          const bool on = allowed(rb[r], j);
          float x = sc[r][c];
          if (bias) x = alpha_first ? fmaf(x, p.alpha, bv[r][c]) : (x + bv[r][c]) * p.alpha;
          else x *= p.alpha;
          float pv = simt::divide(x, 1.f + expf(-x)) * p.scale;
          if (p.mask_type == HSTU_MASK_CUSTOM)
            pv *= on ? to_f<T>(cmask[((static_cast<long long>(b) * p.hq + h) * p.maxq + i) * p.maxk + j]) : 0.f;
          pv = on ? simt::rounded<T>(pv) : 0.f;
          Ps[(4 * ty + r) * ldp + tx + 16 * c] = pv;
        }
      simt::cp_async_wait<0>();   // V_t
      __syncthreads();            // Ps and V_t are there; K_t is consumed
      if (t + 1 < ntiles) simt::load_rows<T, kFwdKeys, kDim>(Ks, ldq, k, s.k0, c0 + kFwdKeys, s.lk, p.hk, hk, dq);
      simt::cp_async_commit();
      const int left = (end - c0 + 3) & ~3;   // (rows of V between lk and the next multiple of four are zeros)
      simt::outer_tile<kDim>(Ps + 4 * ty * ldp, ldp, Vs, kDim, left < kFwdKeys ? left : kFwdKeys, tx, acc);
      __syncthreads();            // V_t and Ps are consumed
      if (t + 1 < ntiles) simt::load_rows<T, kFwdKeys, kDim>(Vs, kDim, v, s.k0, c0 + kFwdKeys, s.lk, p.hk, hk, dv);
      simt::cp_async_commit();
    }
    simt::cp_async_wait<0>();
    T* out = static_cast<T*>(p.out);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = r0 + 4 * ty + r;
      if (i < s.lq) simt::store_row<T, kDim>(out + ((s.q0 + i) * p.hq + h) * dv, dv, tx, acc[r]);
    }
  }
  // nothing here reads what the pre-pass wrote; the wait makes the stream's next operation find both complete
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename T>
__global__ void __launch_bounds__(GTHREADS) hstu_generic_kernel(const KParams p) {
  extern __shared__ float smem[];
  const int bh = blockIdx.x;
  const int b = bh / p.hq;
  const int h = bh - b * p.hq;
  const int hk = h / p.gqa_ratio;
  const int r0 = blockIdx.y * GM;
  const SeqInfo s = load_seq(p, b);
  if (r0 >= s.lq) return;

  const int dq = p.dqk, dv = p.dv;
  const int ldq = dq + 1;  // +1 float of padding: conflict-free column reads
  float* Qs = smem;                     // [GM][ldq]
  float* Ks = Qs + GM * ldq;            // [GN][ldq]
  float* Vs = Ks + GN * ldq;            // [GN][dv]
  float* Ps = Vs + GN * dv;             // [GM][GN]

  const int tid = threadIdx.x;
  const int tx = tid & 31;
  const int ty = tid >> 5;

  const T* q = static_cast<const T*>(p.q);
  const T* k = static_cast<const T*>(p.k);
  const T* v = static_cast<const T*>(p.v);
  const T* bias = static_cast<const T*>(p.bias);
  const T* cmask = static_cast<const T*>(p.mask);

  for (int idx = tid; idx < GM * dq; idx += GTHREADS) {
    const int r = idx / dq, d = idx - r * dq;
    const int row = r0 + r;
    Qs[r * ldq + d] = row < s.lq ? to_f<T>(q[((s.q0 + row) * p.hq + h) * dq + d]) : 0.f;
  }

  RowBounds rb[GROWS];
#pragma unroll
  for (int r = 0; r < GROWS; ++r) rb[r] = row_bounds(s, r0 + ty * GROWS + r, p.mask_type, p.group);

  float acc[GROWS][GMAXC];
#pragma unroll
  for (int r = 0; r < GROWS; ++r)
#pragma unroll
    for (int c = 0; c < GMAXC; ++c) acc[r][c] = 0.f;

  const int ntiles = kv_tiles_for_rows(s, r0, GM, p.mask_type, GN);
  const int ncol = (dv + 31) >> 5;
  const bool alpha_first = (p.flags & HSTU_FLAG_ALPHA_BEFORE_BIAS) != 0;

  for (int t = 0; t < ntiles; ++t) {
    const int c0 = t * GN;
    __syncthreads();  // previous tile's Ks/Vs/Ps fully consumed (also orders the Qs fill on t == 0)
    for (int idx = tid; idx < GN * dq; idx += GTHREADS) {
      const int r = idx / dq, d = idx - r * dq;
      const int col = c0 + r;
      Ks[r * ldq + d] = col < s.lk ? to_f<T>(k[((s.k0 + col) * p.hk + hk) * dq + d]) : 0.f;
    }
    for (int idx = tid; idx < GN * dv; idx += GTHREADS) {
      const int r = idx / dv, d = idx - r * dv;
      const int col = c0 + r;
      Vs[idx] = col < s.lk ? to_f<T>(v[((s.k0 + col) * p.hk + hk) * dv + d]) : 0.f;
    }
    __syncthreads();

    float sc[GROWS] = {0.f, 0.f, 0.f, 0.f};
    const float* krow = Ks + tx * ldq;
    const float* qrow = Qs + ty * GROWS * ldq;
    for (int d = 0; d < dq; ++d) {
      const float kv = krow[d];
#pragma unroll
      for (int r = 0; r < GROWS; ++r) sc[r] = fmaf(qrow[r * ldq + d], kv, sc[r]);
    }
    const int j = c0 + tx;
#pragma unroll
    for (int r = 0; r < GROWS; ++r) {
      const int i = r0 + ty * GROWS + r;
      float pv = 0.f;
      if (i < s.lq && j < s.lk && allowed(rb[r], j)) {
        float x = sc[r];
        if (bias) {
          const long long boff = static_cast<long long>(b) * p.bias_bstride +
                                 (static_cast<long long>(h) * p.maxq + i) * p.maxk + j;
          const float bv = to_f<T>(bias[boff]);
          x = alpha_first ? fmaf(x, p.alpha, bv) : (x + bv) * p.alpha;
        } else {
          x *= p.alpha;
        }
        pv = x / (1.f + expf(-x)) * p.scale;
        if (p.mask_type == HSTU_MASK_CUSTOM) {
          const long long moff = ((static_cast<long long>(b) * p.hq + h) * p.maxq + i) * p.maxk + j;
          pv *= to_f<T>(cmask[moff]);
        }
        pv = to_f<T>(from_f<T>(pv));
      }
      Ps[(ty * GROWS + r) * GN + tx] = pv;
    }
    __syncthreads();

    const int kend = min(GN, s.lk - c0);
    for (int kk = 0; kk < kend; ++kk) {
      float pr[GROWS];
#pragma unroll
      for (int r = 0; r < GROWS; ++r) pr[r] = Ps[(ty * GROWS + r) * GN + kk];
      const float* vrow = Vs + kk * dv;
#pragma unroll
      for (int c = 0; c < GMAXC; ++c) {
        if (c < ncol) {
          const int col = tx + 32 * c;
          const float vv = col < dv ? vrow[col] : 0.f;
#pragma unroll
          for (int r = 0; r < GROWS; ++r) acc[r][c] = fmaf(pr[r], vv, acc[r][c]);
        }
      }
    }
  }

  T* out = static_cast<T*>(p.out);
#pragma unroll
  for (int r = 0; r < GROWS; ++r) {
    const int i = r0 + ty * GROWS + r;
    if (i >= s.lq) continue;
    T* orow = out + ((s.q0 + i) * p.hq + h) * dv;
#pragma unroll
    for (int c = 0; c < GMAXC; ++c) {
      const int col = tx + 32 * c;
      if (c < ncol && col < dv) orow[col] = from_f<T>(acc[r][c]);
    }
  }
}

size_t generic_smem_bytes(const KParams& p) {
  return sizeof(float) * (static_cast<size_t>(GM + GN) * (p.dqk + 1) + static_cast<size_t>(GN) * p.dv + GM * GN);
}

template <typename T, int kDim>
cudaError_t launch_simt(const KParams& p, cudaStream_t stream) {
  constexpr int smem = 4 * (simt::kRows * (kDim + 4) + kFwdKeys * (kDim + 4) + kFwdKeys * kDim + simt::kRows * (kFwdKeys + 4));
  cudaError_t e = cudaFuncSetAttribute(hstu_simt_fwd_kernel<T, kDim>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid(static_cast<unsigned>(p.batch) * p.hq, (p.maxq + simt::kRows - 1) / simt::kRows, 1);
  return simt::launch(hstu_simt_fwd_kernel<T, kDim>, grid, smem, stream, p);
}

// The register-tiled kernel wherever its loads are possible.  (4 sequences of at most 128 rows, 2 heads of 32, fp32: a call
// took 17 us instead of 39 with the other kernel; 12 us since, with less host work in front of it.)
bool simt_supported(const KParams& p, int dtype) {
  return simt::dims_ok(p) && simt::aligned_to(p.q, dtype) && simt::aligned_to(p.k, dtype) &&
         simt::aligned_to(p.v, dtype) && simt::aligned_to(p.out, dtype);
}

__global__ void divide_kernel(const float* a, const float* b, float* out, long long n) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) out[i] = simt::divide(a[i], b[i]);
}

template <typename T>
cudaError_t launch_t(const KParams& p, int dtype, cudaStream_t stream) {
  if (simt_supported(p, dtype)) {
    switch (simt::tile_dim(p)) {
      case 32: return launch_simt<T, 32>(p, stream);
      case 64: return launch_simt<T, 64>(p, stream);
      default: return launch_simt<T, 128>(p, stream);
    }
  }
  const size_t smem = generic_smem_bytes(p);
  cudaError_t e = cudaFuncSetAttribute(hstu_generic_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  dim3 grid(static_cast<unsigned>(p.batch) * p.hq, (p.maxq + GM - 1) / GM, 1);
  hstu_generic_kernel<T><<<grid, GTHREADS, smem, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace

// simt::divide on arrays, for the tests
cudaError_t launch_divide(const float* a, const float* b, float* out, long long n, cudaStream_t stream) {
  divide_kernel<<<256, 256, 0, stream>>>(a, b, out, n);
  return cudaGetLastError();
}

cudaError_t launch_generic(const KParams& p, int dtype, cudaStream_t stream) {
  switch (dtype) {
    case HSTU_DTYPE_BF16: return launch_t<__nv_bfloat16>(p, dtype, stream);
    case HSTU_DTYPE_FP16: return launch_t<__half>(p, dtype, stream);
    default: return launch_t<float>(p, dtype, stream);
  }
}

}  // namespace hstu
