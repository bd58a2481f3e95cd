// in_linear_silu forward on Blackwell tensor cores: mixed = x . weight^T + bias;  linear_output = mixed;
// (user, value, query, key) = split(silu(mixed)) - the step that produces the attention's q / k / v in an HSTU layer.
//
// Reference operator ops_rec::distance_in_linear_silu
// (ascendc/activation/in_linear_silu/torch_extension/in_linear_silu_plugin.cpp:36-98; definition of the result in
// in_linear_silu_forward/test/pytest/test_in_linear_silu.py:36-50: addmm in the input type, SiLU of that ROUNDED
// value, split along the last dimension).  x [m, k] and weight [n, k] are bf16 / fp16, bias [n] fp32.
//
// One CTA PAIR (cluster of two, cta_group::2) per 256 x 256 tile of mixed (n tiles fastest, so the pairs that run together
// share their x rows; the weight stays in L2).  The tile size is set by the L2 -> shared-memory traffic: a 128 x 128 tile
// needs 1 byte per 64 FLOPs (measured: 531 TFLOP/s, the L2 limit), a 256 x 256 tile half of that.  Shared by a pair, the
// tile takes half of each CTA's tensor memory, so there are two of them: the epilogue of one tile runs under the main
// loop of the next.  In each CTA:
//   warp 0   TMA producer: 64-wide K chunks of this CTA's 128 rows of x and 128 rows of the weight, a 5-stage ring; the
//            bytes of both CTAs are counted on the leader's barrier
//   warp 1   MMA issuer (of the leader, rank 0): tcgen05.mma cta_group::2, M256 N256 K16, fp32 accumulators in TMEM
//            (each CTA its 128 rows x 256 columns)
//   warp 2   TMEM allocation
//   warps 4-7 / 8-11 epilogue of columns 0..127 / 128..255 (thread = row): TMEM -> + bias -> round -> linear_output; SiLU
//            of the rounded value -> the output its 16-column group belongs to (the split sizes are multiples of 16)
// The two products of the backward run on the same pipeline with operands read where they lie: x_grad = dL . weight has
// an N-contiguous B, weight_grad = dL^T . x an M-contiguous A as well (MN-major descriptors, no transposed copies).
// Rows / columns / K past the matrix edges are zero-filled by TMA and never stored.  Tensor bound: 2 m n k FLOPs.
// Every mbarrier wait is bounded (then: status bit in the caller's status word, CTA-wide abort flag).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"
#include "ptx_sm100.cuh"

namespace hstu {

bool make_matrix_map(CUtensorMap* m, const void* base, long long rows, long long cols, int dtype, int box_rows);
bool make_store_map(CUtensorMap* m, void* base, long long rows, long long cols, long long ld, int dtype, int box_cols);

namespace {

constexpr int kLsThreads = 384;
constexpr int kLsTile = 256;                    // tile edge of a CTA pair
constexpr int kLsHalf = 128;                    // each CTA's rows of A and of B
constexpr int kLsStages = 5;
constexpr int kLsChunkBytes = kLsHalf * 128;    // 128 x 64 16-bit values of one operand
constexpr int kLsPairs = 74;                    // CTA pairs of a B200 (148 SMs): what a product is split for
constexpr long long kLsWaitLimit = 2000000000ll;

struct LsBars {
  uint64_t full[kLsStages], empty[kLsStages];
  uint64_t acc_full[2], acc_free[2];   // per accumulator buffer (acc_free: the leader's counts both CTAs' epilogue warps)
  uint64_t done;   // every product this pair has issued is complete
  uint32_t tmem_base;
  int abort_flag;
  int epi_stop[2];   // the abort flag as the epilogue warps agree to have seen it (per tile parity)
};

template <typename T> struct LsPack;
template <> struct LsPack<__nv_bfloat16> {
  static constexpr int kFormat = 1;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
  }
  // SiLU in the tanh form, one SFU operation per element: v sigmoid(v) = h (1 + tanh h), h = v / 2.  The error of
  // tanh.approx (2^-11) stays below half a unit in the last place of the bf16 result wherever the result is not tiny.
  static __device__ __forceinline__ uint32_t silu2(float2 v) {
    const float2 h = __fmul2_rn(v, make_float2(0.5f, 0.5f));
    const float2 o = __ffma2_rn(h, make_float2(ptx::tanh_approx(h.x), ptx::tanh_approx(h.y)), h);
    return pack(o.x, o.y);
  }
};
template <> struct LsPack<__half> {
  static constexpr int kFormat = 0;
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
  static __device__ __forceinline__ uint32_t silu2(float2 v) {
    return pack(__fdividef(v.x, 1.f + __expf(-v.x)), __fdividef(v.y, 1.f + __expf(-v.y)));
  }
};

__device__ __forceinline__ void ls_wait(LsBars* bars, uint32_t* status, uint32_t bar, uint32_t parity) {
  if (ptx::mbar_try_wait(bar, parity)) return;
  if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) return;
  const long long t0 = clock64();
  unsigned spins = 0;
  while (!ptx::mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3ffu) == 0) {
      if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) return;
      if (clock64() - t0 > kLsWaitLimit) {
        *reinterpret_cast<volatile int*>(&bars->abort_flag) = 1;
        if (status) atomicOr(status, static_cast<uint32_t>(HSTU_ST_PIPE_TIMEOUT));
        return;
      }
    }
  }
}

constexpr int kLsStageBytes = 8 * 2 * 4096;   // per epilogue warp, twice: 32 rows x 32 columns of linear_output and of SiLU
constexpr int kLsRingBytes = kLsStages * 2 * kLsChunkBytes;

// kForward: the operator itself, A = x and B = weight, both K-major.  The other modes are bare products for the backward
// (in_linear_silu_bwd.cu), written to p.linear ([m, n], rounded) or, split along K, as fp32 partial sums to `partial`:
//   kGradX  A [m, k] K-major, B [k, n] (N-contiguous);   kGradW  A [k, m] (M-contiguous), B [k, n] (N-contiguous)
//
// Persistent: the pairs walk the units (tile, part of K) u, u + pairs, ...  The operand ring runs on across units and
// the accumulators alternate between two TMEM buffers, so the tensor cores go on while the epilogue warps turn a tile's
// accumulators into outputs; the results leave through TMA stores from a staging block per warp.
enum LsMode { kForward, kGradX, kGradW };

template <typename T, int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kLsThreads, 1)
in_linear_silu_kernel(const LinSiluParams p, const __grid_constant__ CUtensorMap tm_a,
                      const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_lin,
                      const __grid_constant__ CUtensorMap tm_o0, const __grid_constant__ CUtensorMap tm_o1,
                      const __grid_constant__ CUtensorMap tm_o2, const __grid_constant__ CUtensorMap tm_o3,
                      const long long tiles, const int splits, float* const partial) {
  constexpr bool kPlain = kMode != kForward;
  constexpr bool kMnA = kMode == kGradW, kMnB = kMode != kForward;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  LsBars* bars = reinterpret_cast<LsBars*>(base_ptr + kLsRingBytes + kLsStageBytes);
  float* s_bias = reinterpret_cast<float*>(base_ptr + kLsRingBytes + kLsStageBytes + 256);   // [256]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = ptx::cluster_rank();
  const long long pair0 = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int n_tiles = (p.n + kLsTile - 1) / kLsTile;
  const int chunks = (p.k + 63) / 64;
  const int per_split = (chunks + splits - 1) / splits;   // (the launcher leaves no part empty)
  const long long units = tiles * splits;

  if (tid == 0) {
    ptx::prefetch_tensormap(&tm_a);
    ptx::prefetch_tensormap(&tm_b);
    ptx::prefetch_tensormap(&tm_lin);
    if (!kPlain) {
      ptx::prefetch_tensormap(&tm_o0);
      ptx::prefetch_tensormap(&tm_o1);
      ptx::prefetch_tensormap(&tm_o2);
      ptx::prefetch_tensormap(&tm_o3);
    }
    for (int i = 0; i < kLsStages; ++i) {
      ptx::mbar_init(ptx::smem_u32(&bars->full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&bars->empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(ptx::smem_u32(&bars->acc_full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&bars->acc_free[i]), 2 * 8);   // every epilogue warp of the pair
    }
    ptx::mbar_init(ptx::smem_u32(&bars->done), 1);
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 2) {
    ptx::tmem_alloc_pair(ptx::smem_u32(&bars->tmem_base), 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();   // both CTAs' barriers exist
  ptx::tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

  if (warp == 0) {
    if (lane == 0) {
      uint32_t g = 0;   // chunks requested so far (over all units of this pair)
      for (long long u = pair0; u < units; u += pairs) {
        const long long t = u / splits;
        const int c_begin = static_cast<int>(u % splits) * per_split;
        const int c_end = c_begin + per_split < chunks ? c_begin + per_split : chunks;
        const int n0 = static_cast<int>(t % n_tiles) * kLsTile + static_cast<int>(rank) * kLsHalf;
        const int m0 = static_cast<int>(t / n_tiles) * kLsTile + static_cast<int>(rank) * kLsHalf;
        for (int c = c_begin; c < c_end; ++c, ++g) {
          const uint32_t s = g % kLsStages;
          ls_wait(bars, p.status, ptx::smem_u32(&bars->empty[s]), ((g / kLsStages) & 1u) ^ 1u);
          if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) break;
          const uint32_t full = ptx::smem_u32(&bars->full[s]);
          if (rank == 0) ptx::mbar_expect_tx(full, 4 * kLsChunkBytes);   // both operands of both CTAs
          const uint32_t lead = ptx::map_to_rank(full, 0);
          const uint32_t sa = base + s * 2 * kLsChunkBytes, sb = sa + kLsChunkBytes;
          if (kMnA) {
            ptx::tma_load_2d_pair(sa, &tm_a, lead, m0, c * 64);
            ptx::tma_load_2d_pair(sa + kLsChunkBytes / 2, &tm_a, lead, m0 + 64, c * 64);
          } else {
            ptx::tma_load_2d_pair(sa, &tm_a, lead, c * 64, m0);
          }
          if (kMnB) {
            ptx::tma_load_2d_pair(sb, &tm_b, lead, n0, c * 64);
            ptx::tma_load_2d_pair(sb + kLsChunkBytes / 2, &tm_b, lead, n0 + 64, c * 64);
          } else {
            ptx::tma_load_2d_pair(sb, &tm_b, lead, c * 64, n0);
          }
        }
        if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) break;
      }
      // drain (matters only after an abort): the last loads have landed before either CTA leaves the cluster barrier at the
      // end.  The leader's barriers count those of both CTAs, but the other CTA may have requested more than the leader
      // has, on barriers it cannot wait for: it gives them a millisecond.
      if (rank != 0 && *reinterpret_cast<volatile int*>(&bars->abort_flag)) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) {}
      }
      if (rank == 0) {
        for (uint32_t back = 0; back < kLsStages && back < g; ++back) {
          const uint32_t c = g - 1 - back;
          const uint32_t bar = ptx::smem_u32(&bars->full[c % kLsStages]);
          for (int spin = 0; spin < (1 << 22) && !ptx::mbar_try_wait(bar, (c / kLsStages) & 1u); ++spin) {}
        }
      }
    }
  } else if (warp == 1) {
    // (an elected thread, not `lane == 0`: the compiler then keeps descriptors and barrier addresses in uniform registers)
    if (rank == 0 && ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::umma_idesc_f16(LsPack<T>::kFormat, kLsTile, kLsTile, kMnB, kMnA);
      constexpr uint64_t kDescK = ptx::umma_desc_sw128_hi(16, 1024);
      constexpr uint64_t kDescMn = ptx::umma_desc_sw128_hi(kLsChunkBytes / 2, 1024);   // two 64-wide column blocks
      uint32_t g = 0, it = 0;
      for (long long u = pair0; u < units; u += pairs, ++it) {
        const int c_begin = static_cast<int>(u % splits) * per_split;
        const int c_end = c_begin + per_split < chunks ? c_begin + per_split : chunks;
        const uint32_t buf = it & 1u;
        // the epilogues have read what this buffer held
        if (it > 1) ls_wait(bars, p.status, ptx::smem_u32(&bars->acc_free[buf]), ((it >> 1) - 1u) & 1u);
        ptx::tc_fence_after();
        for (int c = c_begin; c < c_end; ++c, ++g) {
          const uint32_t s = g % kLsStages;
          ls_wait(bars, p.status, ptx::smem_u32(&bars->full[s]), (g / kLsStages) & 1u);
          if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) break;
          ptx::tc_fence_after();
          const uint32_t sa = base + s * 2 * kLsChunkBytes;
          const uint64_t a = (kMnA ? kDescMn : kDescK) | static_cast<uint64_t>(sa >> 4);
          const uint64_t b = (kMnB ? kDescMn : kDescK) | static_cast<uint64_t>((sa + kLsChunkBytes) >> 4);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t off_a = static_cast<uint64_t>((ks * (kMnA ? 2048 : 32)) >> 4);
            const uint64_t off_b = static_cast<uint64_t>((ks * (kMnB ? 2048 : 32)) >> 4);
            ptx::mma_ss_pair(tmem + buf * kLsTile, a + off_a, b + off_b, idesc, (c > c_begin || ks > 0) ? 1u : 0u);
          }
          ptx::mma_commit_pair(ptx::smem_u32(&bars->empty[s]));
        }
        if (*reinterpret_cast<volatile int*>(&bars->abort_flag)) break;
        ptx::mma_commit_pair(ptx::smem_u32(&bars->acc_full[buf]));
      }
      ptx::mma_commit_pair(ptx::smem_u32(&bars->done));
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue (thread = row of the tile)
    // Each warp turns 32 rows x 32 columns at a time: TMEM -> registers -> (+ bias, round, SiLU) -> its staging block
    // -> TMA stores (one 32-column box of linear_output, 64-byte swizzle; the SiLU values as two 16-column boxes,
    // because a split boundary may fall between them).  The TMEM load of the next 32 columns is in flight while the
    // current ones are computed; two staging blocks, so a round does not wait for the previous round's stores.
    const int colh = ((warp - 4) >> 2) * kLsHalf;   // this warp's columns of the tile: [colh, colh + 128)
    const uint32_t lane_base = (static_cast<uint32_t>((warp & 3) * 32) << 16) + colh;
    const uint32_t swz = (lane >> 1) & 3;      // 64-byte swizzle: 16-byte chunk index ^ address bits [7, 9)
    const int etid = tid - 128;                // 0..255 among the epilogue threads
    uint32_t it = 0, round = 0;   // round: 32-column chunks this warp has staged
    for (long long u = pair0; u < units; u += pairs, ++it) {
      const long long t = u / splits;
      const int n0 = static_cast<int>(t % n_tiles) * kLsTile;
      const long long m0 = (t / n_tiles) * kLsTile;
      const long long row0 = m0 + rank * kLsHalf + (warp & 3) * 32;   // first row of this warp
      const uint32_t buf = it & 1u;
      // The eight warps meet at barriers once per tile, so they must leave the loop together: one thread samples the
      // abort flag before the first barrier, everybody acts on that sample after it.
      if (etid == 0) bars->epi_stop[buf] = *reinterpret_cast<volatile int*>(&bars->abort_flag);
      ptx::named_bar_sync(1, 8 * 32);   // (also: every warp has read the previous tile's bias values)
      if (*reinterpret_cast<volatile int*>(&bars->epi_stop[buf])) break;
      if (!kPlain) {
        // the bias values of this tile's columns (zeros without a bias / past the last column)
        s_bias[etid] = (p.bias && n0 + etid < p.n) ? p.bias[n0 + etid] : 0.f;
        ptx::named_bar_sync(1, 8 * 32);
      }
      ls_wait(bars, p.status, ptx::smem_u32(&bars->acc_full[buf]), (it >> 1) & 1u);
      ptx::tc_fence_after();
      // a wait gave up (status word set) since the sample: the accumulators hold nothing valid - touch nothing, store
      // nothing, and leave at the next tile's barrier
      if (__any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&bars->abort_flag))) continue;
      const int left = (p.n - n0 - colh + 31) / 32;
      const int nch = left < 0 ? 0 : left < kLsHalf / 32 ? left : kLsHalf / 32;   // uniform over the warp
      const uint32_t src = tmem + buf * kLsTile + lane_base;
      auto release = [&] {   // this warp has read the last columns it needs: the buffer's next products may overwrite them
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_rank(ptx::smem_u32(&bars->acc_free[buf]), 0));
      };
      uint32_t acc[2][32];
      if (nch == 0) release();
      else ptx::tmem_ld32(src, acc[0]);
#pragma unroll 1
      for (int ch2 = 0; ch2 < kLsHalf / 32; ch2 += 2) {
#pragma unroll
        for (int u2 = 0; u2 < 2; ++u2) {
          const int ch = ch2 + u2;
          if (ch >= nch) break;
          const int c0 = n0 + colh + ch * 32;
          const uint32_t st_lin = base + kLsRingBytes + ((warp - 4) * 2 + (round & 1u)) * 4096;   // 32 rows x 64 bytes, 64-byte swizzle
          const uint32_t st_act = st_lin + 2048;                                        // 2 x (32 rows x 32 bytes)
          ptx::tmem_wait_ld_dep(acc[u2]);
          if (ch + 1 < nch) ptx::tmem_ld32(src + (ch + 1) * 32, acc[u2 ^ 1]);
          else release();
          if (kPlain && splits > 1) {   // fp32 partial sums (n is a multiple of 16)
            const long long row = row0 + lane;
            if (row < p.m) {
              float* to = partial + ((u % splits) * p.m + row) * p.n + c0;
#pragma unroll
              for (int e = 0; e < 8; ++e)
                if (c0 + 4 * e < p.n)
                  *reinterpret_cast<uint4*>(to + 4 * e) =
                      make_uint4(acc[u2][4 * e], acc[u2][4 * e + 1], acc[u2][4 * e + 2], acc[u2][4 * e + 3]);
            }
            continue;
          }
          uint32_t lin[16], act[16];
          // packed f32x2 arithmetic; the rounded values come back out of the packed pair (one conversion each way)
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float2 sum = make_float2(__uint_as_float(acc[u2][2 * e]), __uint_as_float(acc[u2][2 * e + 1]));
            if (!kPlain) sum = __fadd2_rn(sum, *reinterpret_cast<const float2*>(&s_bias[colh + ch * 32 + 2 * e]));
            lin[e] = LsPack<T>::pack(sum.x, sum.y);
            if (!kPlain) act[e] = LsPack<T>::silu2(LsPack<T>::unpack(lin[e]));   // SiLU of the rounded value
          }
          // the stores that last used this staging block (two rounds ago: at most the latest one may still be reading)
          if (lane < 3) ptx::bulk_wait_read<1>();   // (lanes 0..2 issue one store each)
          __syncwarp();
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(st_lin + lane * 64 + ((q4 ^ swz) << 4)),
                         "r"(lin[4 * q4]), "r"(lin[4 * q4 + 1]), "r"(lin[4 * q4 + 2]), "r"(lin[4 * q4 + 3])
                         : "memory");
            if (!kPlain)   // columns 0..15 of the chunk in the first block, 16..31 in the second
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(st_act + (q4 >> 1) * 1024 + lane * 32 + (q4 & 1) * 16),
                           "r"(act[4 * q4]), "r"(act[4 * q4 + 1]), "r"(act[4 * q4 + 2]), "r"(act[4 * q4 + 3])
                           : "memory");
          }
          ptx::fence_proxy_async();
          __syncwarp();
          // three lanes issue one store each (an issue costs its thread ~100 cycles); rows and columns past the
          // matrix edge are clipped by the tensor maps.  Every round commits a group, an empty one too: the wait above
          // counts rounds.
          if (lane < 3) {
            const int cg = c0 + 16 * (lane - 1);   // the 16-column group decides the SiLU output tensor (n, splits: multiples of 16)
            const bool rows = row0 < p.m;
            if (rows && lane == 0) {
              ptx::tma_store_2d(&tm_lin, st_lin, c0, static_cast<int>(row0));
            } else if (rows && lane > 0 && !kPlain && cg < p.n) {
              const int which = (cg >= p.start[1]) + (cg >= p.start[2]) + (cg >= p.start[3]);
              const CUtensorMap* tm = which == 0 ? &tm_o0 : which == 1 ? &tm_o1 : which == 2 ? &tm_o2 : &tm_o3;
              ptx::tma_store_2d(tm, st_act + (lane - 1) * 1024, cg - p.start[which], static_cast<int>(row0));
            }
            ptx::bulk_commit();
          }
          ++round;
        }
      }
    }
    if (lane < 3) ptx::bulk_wait<0>();   // this thread's TMA stores have completed
  }

  ptx::tc_fence_before();
  __syncthreads();
  // (matters only after an abort: otherwise the epilogues have waited for every product)
  if (tid == 0)
    for (int spin = 0; spin < (1 << 22) && !ptx::mbar_try_wait(ptx::smem_u32(&bars->done), 0); ++spin) {}
  __syncwarp();
  ptx::cluster_sync();   // neither CTA leaves while the other's loads, products or arrivals may still touch it
  if (warp == 2) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem, 512);
  }
}

long long tiles_of(long long m, int n) {
  return static_cast<long long>((n + kLsTile - 1) / kLsTile) * ((m + kLsTile - 1) / kLsTile);
}

template <typename T, int kMode>
cudaError_t launch_t(const LinSiluParams& p, const CUtensorMap& ma, const CUtensorMap& mb, int splits, float* partial,
                     int dtype, cudaStream_t stream) {
  constexpr bool kPlain = kMode != kForward;
  // store maps: linear_output [m, n], and the four SiLU outputs [m, width[i]] (a width of 0: never addressed)
  CUtensorMap ml, mo[4];
  if (!make_store_map(&ml, p.linear, p.m, p.n, p.n, dtype, 32)) return cudaErrorNotSupported;
  for (int i = 0; i < 4; ++i) {
    const bool used = !kPlain && p.width[i] > 0;
    if (!make_store_map(&mo[i], used ? p.out[i] : p.linear, p.m, used ? p.width[i] : p.n, used ? p.width[i] : p.n, dtype,
                        16))
      return cudaErrorNotSupported;
  }
  constexpr int smem = 1024 + kLsRingBytes + kLsStageBytes + 256 + kLsTile * 4;
  static_assert(smem <= 232448, "shared memory budget");
  static_assert(sizeof(LsBars) <= 256, "barrier block too large");
  auto kern = in_linear_silu_kernel<T, kMode>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const long long tiles = tiles_of(p.m, p.n);
  if ((p.m + kLsTile - 1) / kLsTile > 0x7fffffll) return cudaErrorInvalidConfiguration;   // (TMA row coordinates are int)
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const long long pairs = sms / 2, units = tiles * splits;
  const unsigned grid = 2 * static_cast<unsigned>(units < pairs ? units : pairs);
  kern<<<dim3(grid), kLsThreads, smem, stream>>>(p, ma, mb, ml, mo[0], mo[1], mo[2], mo[3], tiles, splits, partial);
  return cudaGetLastError();
}

template <typename T>
__global__ void __launch_bounds__(256) sum_partials_kernel(const float* __restrict__ partial, T* __restrict__ out,
                                                           long long count4, int splits) {
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;   // four values each
  if (i >= count4) return;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float4 v = reinterpret_cast<const float4*>(partial)[s * count4 + i];
    sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
  }
  reinterpret_cast<uint2*>(out)[i] = make_uint2(LsPack<T>::pack(sum.x, sum.y), LsPack<T>::pack(sum.z, sum.w));
}

template <typename T, int kMode>
cudaError_t product_t(const LinSiluParams& p, const CUtensorMap& ma, const CUtensorMap& mb, int splits, float* partial,
                      int dtype, cudaStream_t stream) {
  cudaError_t e = launch_t<T, kMode>(p, ma, mb, splits, partial, dtype, stream);
  if (e != cudaSuccess || splits == 1) return e;
  const long long count4 = p.m * p.n / 4;   // (n is a multiple of 16)
  sum_partials_kernel<T><<<static_cast<unsigned>((count4 + 255) / 256), 256, 0, stream>>>(partial, static_cast<T*>(p.linear),
                                                                                         count4, splits);
  return cudaGetLastError();
}

}  // namespace

// Returns cudaSuccess, a CUDA error, or cudaErrorNotSupported when the tensor maps could not be encoded.
cudaError_t launch_in_linear_silu(const LinSiluParams& p, const void* x, const void* weight, int dtype,
                                  cudaStream_t stream) {
  if (p.m == 0) return cudaSuccess;
  CUtensorMap mx, mw;
  if (!make_matrix_map(&mx, x, p.m, p.k, dtype, kLsHalf) || !make_matrix_map(&mw, weight, p.n, p.k, dtype, kLsHalf))
    return cudaErrorNotSupported;
  return dtype == HSTU_DTYPE_BF16 ? launch_t<__nv_bfloat16, kForward>(p, mx, mw, 1, nullptr, dtype, stream)
                                  : launch_t<__half, kForward>(p, mx, mw, 1, nullptr, dtype, stream);
}

// How many parts a product [m, n] with contraction length k is cut into along k: as many as give every CTA pair a unit,
// at least eight 64-wide chunks each (a part costs a write and a read of its fp32 partial sums).  Products with more
// than half as many tiles as pairs stay whole.
int product_splits(long long m, int n, long long k) {
  const long long tiles = tiles_of(m, n), chunks = (k + 63) / 64;
  long long s = kLsPairs / (tiles > 0 ? tiles : 1);
  if (s > chunks / 8) s = chunks / 8;
  if (s < 2) return 1;
  const long long per = (chunks + s - 1) / s;
  return static_cast<int>((chunks + per - 1) / per);   // (no empty part)
}
uint64_t product_partial_bytes(long long m, int n, long long k) {
  const int s = product_splits(m, n, k);
  return s > 1 ? static_cast<uint64_t>(s) * static_cast<uint64_t>(m) * n * 4 : 0;
}

// The backward's products, out [m, n] = a . b in the element type (fp32 accumulation, one rounding; n a multiple of 16,
// bases 16-byte aligned, tensors contiguous); partial: product_partial_bytes(m, n, k) bytes.
// trans_a: a is [k, m] and read transposed, else [m, k].  b is [k, n].  What lies past k reads as zeros.
cudaError_t launch_product(const void* a, bool trans_a, const void* b, long long m, int n, long long k, void* out,
                           float* partial, int dtype, uint32_t* status, cudaStream_t stream) {
  if (m == 0 || n == 0) return cudaSuccess;
  CUtensorMap ma, mb;
  if (!(trans_a ? make_matrix_map(&ma, a, k, m, dtype, 64) : make_matrix_map(&ma, a, m, k, dtype, kLsHalf)) ||
      !make_matrix_map(&mb, b, k, n, dtype, 64))
    return cudaErrorNotSupported;
  LinSiluParams p = {};
  p.linear = out;
  p.m = m;
  p.n = n;
  p.k = static_cast<int>(k);
  p.start[4] = n;
  p.status = status;
  const int splits = product_splits(m, n, k);
  if (dtype == HSTU_DTYPE_BF16)
    return trans_a ? product_t<__nv_bfloat16, kGradW>(p, ma, mb, splits, partial, dtype, stream)
                   : product_t<__nv_bfloat16, kGradX>(p, ma, mb, splits, partial, dtype, stream);
  return trans_a ? product_t<__half, kGradW>(p, ma, mb, splits, partial, dtype, stream)
                 : product_t<__half, kGradX>(p, ma, mb, splits, partial, dtype, stream);
}

}  // namespace hstu
