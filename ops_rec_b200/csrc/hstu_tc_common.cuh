// What the two tensor-core forward kernels (hstu_tc.cu, hstu_short.cu) share: bounded barrier waits, 16-bit packing, the
// element-wise stage of 32 scores, the mask as bits of 32 columns, and the zeroing of V rows behind a sequence's end.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"
#include "ptx_sm100.cuh"

namespace hstu {
namespace {

constexpr long long kWaitLimitCycles = 2000000000ll;  // ~1 s

// The waiting loop of Waiter::wait, one copy for every wait of the kernel (the fast path - the phase is already
// complete - stays inline): less code for the instruction caches, and the warps that spin all spin in the same lines.
__device__ __noinline__ void wait_slow(int* abort_flag, uint32_t* status, uint32_t bar, uint32_t parity) {
  if (*reinterpret_cast<volatile int*>(abort_flag)) return;
  const long long t0 = clock64();
  unsigned spins = 0;
  while (!ptx::mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3ffu) == 0) {
      if (*reinterpret_cast<volatile int*>(abort_flag)) return;
      if (clock64() - t0 > kWaitLimitCycles) {
        *reinterpret_cast<volatile int*>(abort_flag) = 1;
        atomicOr(status, static_cast<uint32_t>(HSTU_ST_PIPE_TIMEOUT));
        return;
      }
    }
  }
}

struct Waiter {
  int* abort_flag;
  uint32_t* status;
  // `polled` is the result of an earlier mbar_try_wait on the same phase (polls of several barriers are issued
  // back to back so that their latencies overlap); only an unsuccessful poll falls into the waiting loop.
  __device__ __forceinline__ void wait_polled(bool polled, uint32_t bar, uint32_t parity) const {
    if (!polled) wait(bar, parity);
  }
  __device__ __forceinline__ bool aborted() const { return *reinterpret_cast<volatile int*>(abort_flag) != 0; }
  __device__ __forceinline__ void wait(uint32_t bar, uint32_t parity) const {
    if (ptx::mbar_try_wait(bar, parity)) return;
    wait_slow(abort_flag, status, bar, parity);
  }
};

template <typename T> struct Pack;
template <> struct Pack<__nv_bfloat16> {
  static constexpr int kFormat = 1;
  static constexpr bool kExact = false;   // SiLU: the tanh form
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  }
};
template <> struct Pack<Bf16Exp> : Pack<__nv_bfloat16> {
  static constexpr bool kExact = true;    // SiLU: exp2 and reciprocal
};
template <> struct Pack<__half> {
  static constexpr int kFormat = 0;
  static constexpr bool kExact = true;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
};

// 32 scores of one row (fp32 bits in sr) -> 16 words of packed P.  Branch-free; the arithmetic runs on the
// packed f32x2 pipe.  x = c_in * s + c_bias * bias covers both orders of alpha and bias (c_bias = c_in gives
// alpha * (s + bias)).
// One tanh.approx per element is the SFU's whole budget (16 results/clk/SM = 1024 clk per 128 x 128 tile).  Moving
// half of the columns to an FMA-pipe polynomial was tried: it is faster only without a range check, and any
// data-dependent branch in this block costs more than it saves, so every element goes through the SFU.
template <typename T, int kBias, bool kMasked>
__device__ __forceinline__ void silu_chunk(const uint32_t (&sr)[32], const uint32_t (&bv)[16], uint32_t (&pr)[16],
                                           float c_in, float c_bias, float scale, uint32_t visible) {
  constexpr bool kExact = Pack<T>::kExact;  // exp2 + rcp (two MUFU ops); else the tanh form (one)
  const float2 cin2 = make_float2(c_in, c_in);
  const float2 cb2 = make_float2(c_bias, c_bias);
  const float2 sc2 = make_float2(scale, scale);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    float2 x = make_float2(__uint_as_float(sr[2 * e]), __uint_as_float(sr[2 * e + 1]));
    if (kBias == 1)
      x = __ffma2_rn(x, cin2, __fmul2_rn(Pack<T>::unpack(bv[e]), cb2));
    else
      x = __fmul2_rn(x, cin2);
    const float2 r = __fmul2_rn(x, sc2);
    float2 o;
    if (kExact) {
      // sigmoid form: o = y*scale / (1 + 2^(-y log2 e))
      const float2 ny = __fmul2_rn(x, make_float2(-1.4426950408889634f, -1.4426950408889634f));
      const float2 d = __fadd2_rn(make_float2(ptx::ex2_approx(ny.x), ptx::ex2_approx(ny.y)), make_float2(1.f, 1.f));
      o = __fmul2_rn(r, make_float2(ptx::rcp_approx(d.x), ptx::rcp_approx(d.y)));
    } else {
      // tanh form on x = y/2: o = x*scale*(1 + tanh x)
      o = __ffma2_rn(r, make_float2(ptx::tanh_approx(x.x), ptx::tanh_approx(x.y)), r);
    }
    if (kBias == 3) o = __fmul2_rn(o, Pack<T>::unpack(bv[e]));  // custom mask: its values multiply (fp32)
    if (kMasked) {  // a select, not a multiply: scores of rows past the sequence end may be Inf or NaN
      o.x = (visible & (1u << (2 * e))) ? o.x : 0.f;
      o.y = (visible & (2u << (2 * e))) ? o.y : 0.f;
    }
    pr[e] = Pack<T>::pack(o.x, o.y);
  }
}

// Bit e set <=> column j0 + e is visible to the row described by rb (columns j0 .. j0 + 31).
__device__ __forceinline__ uint32_t low_bits(int n) {  // n lowest bits set, n clamped to [0, 32]
  return n <= 0 ? 0u : (n >= 32 ? 0xffffffffu : ((1u << n) - 1u));
}
__device__ __forceinline__ uint32_t visible_bits(const RowBounds& rb, int j0) {
  return low_bits(rb.lim1 - j0) | (low_bits(rb.hi2 + 1 - j0) & ~low_bits(rb.lo2 - j0));
}

// Zeroes `pieces` 16-byte pieces from shared-memory address `first` on, in each of `boxes` regions `box_bytes` apart
// (the rows of a V tile behind a sequence end); called by the 128 threads of a P/O group, `tid` = 0..127.
__device__ __noinline__ void zero_v_rows(uint32_t first, int pieces, int tid, int boxes, int box_bytes) {
  for (int i = tid; i < pieces; i += kTileM)
    for (int b = 0; b < boxes; ++b) ptx::st_shared_zero16(first + b * box_bytes + i * 16);
  ptx::fence_proxy_async();
}

}  // namespace
}  // namespace hstu
