// HSTU jagged attention forward on the sm_100a tensor cores for batches of short sequences (bf16 / fp16, head dims up to
// 128): several small independent chains per SM instead of hstu_tc.cu's two coupled ones.
//
// What bounds such a batch is the chain of dependent steps of a tile - S = Q.K^T, P = silu(..), O += P.V, and the output at
// its end - not any unit of the SM: a tile of a sequence of 300 rows visits two or three 128-key tiles, each step waits for
// tensor cores, then SFU, then tensor cores, and a call of few queries per sequence (hstu_paged) fills one of the two Q
// tiles of an item only.  Here a CTA is one chain: one 128-row Q tile at a time, K tiles of 64 keys, 192 threads, 128 (D = 64)
// or 256 (D = 128) columns of tensor memory - so an SM holds four of them (three with a staged bias, two at D = 128), and
// while one waits the others compute.  64 keys rather than 128: half the columns of tensor memory per chain, and less of a
// tile lies behind the diagonal or the sequence end.  (4 heads of 64: 2048 sequences of mean 80 151 ->
// 103 us, 1024 of mean 300 243 -> 188, but 4096 of mean 271 with a shared bias, three chains on an SM, 1176 -> 1167, no more
// than the noise; the latter's histories in a paged cache, 16-80 queries each: 720 -> 540 us with a gather in front of it,
// 386 us without.  What a step takes - measured inside the kernel, four chains on an SM - is 1 700 cycles of P, 800 of the
// two products and their hand-overs, and a tile's start and end add some 8 000.)
//
//   warps 0-3  P / O (thread = row = TMEM lane): scores -> P, output store
//   warp 4     one thread: draws tiles (scheduler), requests Q, K / V ring and bias tiles by TMA
//   warp 5     TMEM allocation; one thread issues the MMAs
//
// Element-wise stage, masks, work list and numerics are hstu_tc.cu's, except that a staged bias is added in registers
// (which needs no identity products and no special case at the end of a sequence).  Every mbarrier wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"
#include "hstu_tc_common.cuh"
#include "ptx_sm100.cuh"

namespace hstu {

bool make_kv_tile_map(CUtensorMap* m, const void* base, long long tokens, int heads, int dim, int dtype, int box_rows);

namespace {

constexpr int kShThreads = 192;
constexpr int kShKeys = 64;        // keys per K / V tile
constexpr int kShItems = 3;        // depth of the tile ring between the scheduler and the other roles
constexpr int kShReaders = 4 + 1;  // P / O warps, MMA issuer
constexpr int kShColO = 64;        // TMEM columns: S 0..63 (P in place), O from here

template <int D, bool kBias>
struct ShCfg {
  static constexpr int kHalves = D / 64;
  static constexpr int kQHalf = kTileM * 128, kKvHalf = kShKeys * 128;   // bytes of a 64-wide half tile
  static constexpr int kQBytes = kHalves * kQHalf, kKvBytes = kHalves * kKvHalf;
  static constexpr int kStages = kBias ? 3 : 4;                          // K / V ring slots (one tile each)
  static constexpr int kBiasBytes = kTileM * kShKeys * 2;                // a staged bias tile: 128 rows x 64 keys
  static constexpr int kBiasBufs = D == 64 ? 2 : 1;
  static constexpr int kBiasTotal = kBias ? kBiasBufs * kBiasBytes : 0;
  static constexpr int kPerSm = D == 128 ? 2 : kBias ? 3 : 4;            // CTAs per SM
  static constexpr int kTmemCols = D == 128 ? 256 : 128;
  static constexpr int kSmemBytes = 1024 + kQBytes + kStages * kKvBytes + kBiasTotal + 1024;
  static_assert(kPerSm * (kSmemBytes + 1024) <= 228 * 1024, "shared memory of an SM");
  static_assert(kPerSm * kTmemCols <= 512, "tensor memory of an SM");
};

struct ShTile {
  SeqInfo s;
  int b, h, hk, r0;   // r0: first row of the Q tile
  int n;              // K tiles it visits
  int valid;          // 0 = end of work
  // The keys of a sequence are one segment, or - hstu_paged - two: the cached keys [0, split) and the targets
  // [split, lk).  A tile lies in one segment: tiles j < n_first start at key 64 j, the others at split + 64 (j - n_first).
  int split, n_first;
  int pages;            // hstu_paged: pages of the sequence,
  long long first_slot; //   and the first of them in page_ids
};

struct ShBars {
  uint64_t q_full, q_free, s_full, p_full, o_full, o_free, done;
  uint64_t bias_full[2], bias_free[2];
  uint64_t kv_full[4], kv_free[4];
  uint64_t item_full[kShItems], item_free[kShItems];
  ShTile item[kShItems];
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(ShBars) <= 1024, "barrier block too large");

// This thread's 64 scores -> P, in place.  kMasked: the mask or the segment's end (`left` keys away) cuts through the tile.
template <typename T, bool kBias, bool kMasked>
__device__ __forceinline__ void short_p(uint32_t t_s, uint32_t bias_row, uint32_t bias_swz, const RowBounds& rb, int c0,
                                        int left, float c_in, float scale) {
#pragma unroll
  for (int ch = 0; ch < 2; ++ch) {
    uint32_t sr[32], bv[16], pr[16];
    ptx::tmem_ld32(t_s + ch * 32, sr);
    uint32_t vis = 0xffffffffu;
    bool all_on = true, all_off = false;
    if (kMasked) {
      vis = visible_bits(rb, c0 + ch * 32) & low_bits(left - ch * 32);
      all_on = __all_sync(0xffffffffu, vis == 0xffffffffu);
      all_off = __all_sync(0xffffffffu, vis == 0u);
    }
    if (kBias) {
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(bv[4 * q4]), "=r"(bv[4 * q4 + 1]), "=r"(bv[4 * q4 + 2]), "=r"(bv[4 * q4 + 3])
                     : "r"(bias_row + (((ch * 4 + q4) ^ bias_swz) << 4))
                     : "memory");
    }
    ptx::tmem_wait_ld_dep(sr);
    if (all_off) {
#pragma unroll
      for (int e = 0; e < 16; ++e) pr[e] = 0u;
    } else if (all_on) {
      silu_chunk<T, kBias ? 1 : 0, false>(sr, bv, pr, c_in, c_in, scale, 0u);
    } else {
      silu_chunk<T, kBias ? 1 : 0, true>(sr, bv, pr, c_in, c_in, scale, vis);
    }
    ptx::tmem_st16(t_s + ch * 16, pr);   // (columns whose scores this thread has read)
  }
}

template <int D, typename T, bool kBias>
__global__ void __launch_bounds__(kShThreads, ShCfg<D, kBias>::kPerSm)
hstu_short_kernel(const KParams p, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_bias,
                  const __grid_constant__ CUtensorMap tm_cache) {
  using C = ShCfg<D, kBias>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = ptx::smem_u32(smem_raw);
  const uint32_t sm_q = (raw + 1023u) & ~1023u;
  const uint32_t sm_ring = sm_q + C::kQBytes;
  const uint32_t sm_bias = sm_ring + C::kStages * C::kKvBytes;
  ShBars* bars = reinterpret_cast<ShBars*>(smem_raw + (sm_bias + C::kBiasTotal - raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Waiter w{&bars->abort_flag, p.ws_header};
  const int halves_qk = C::kHalves == 1 ? 1 : (p.dqk + 63) >> 6;
  const int halves_v = C::kHalves == 1 ? 1 : (p.dv + 63) >> 6;

  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&tm_q);
    ptx::prefetch_tensormap(&tm_k);
    ptx::prefetch_tensormap(&tm_v);
    if (p.paged_split) ptx::prefetch_tensormap(&tm_cache);
    if (kBias) ptx::prefetch_tensormap(&tm_bias);
    ptx::mbar_init(ptx::smem_u32(&bars->q_full), 1);
    ptx::mbar_init(ptx::smem_u32(&bars->q_free), 1);
    ptx::mbar_init(ptx::smem_u32(&bars->s_full), 1);
    ptx::mbar_init(ptx::smem_u32(&bars->p_full), 4);    // the P / O warps
    ptx::mbar_init(ptx::smem_u32(&bars->o_full), 1);
    ptx::mbar_init(ptx::smem_u32(&bars->o_free), 4);
    ptx::mbar_init(ptx::smem_u32(&bars->done), 1);
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(ptx::smem_u32(&bars->bias_full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&bars->bias_free[i]), 4);
    }
    for (int i = 0; i < C::kStages; ++i) {
      ptx::mbar_init(ptx::smem_u32(&bars->kv_full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&bars->kv_free[i]), 1);
    }
    for (int i = 0; i < kShItems; ++i) {
      ptx::mbar_init(ptx::smem_u32(&bars->item_full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&bars->item_free[i]), kShReaders);
    }
    bars->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 5) {
    ptx::tmem_alloc(ptx::smem_u32(&bars->tmem_base), C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

  if (warp == 4) {
    // ------------------------------------------------------------------ scheduler and TMA producer
    if (lane == 0) {
      // (only this thread reads what the pre-pass - and hstu_paged's gather in front of it - wrote to global memory)
      asm volatile("griddepcontrol.wait;" ::: "memory");
      long long num_items = p.ws_header[1];
      if (num_items > p.item_capacity) num_items = p.item_capacity;   // (inconsistent offsets: never read past the list)
      // The list's items are q-pairs (256 rows).  Many items: a CTA takes both Q tiles of a pair, and the look-up of a pair
      // is spread over the two before it - counter, entry, offsets - so that none of it delays the loads of K and V.  Few
      // (under eight per CTA): every Q tile is drawn by itself, the later one - more keys - first, and only once the current
      // tile's loads are requested: balance counts for more.
      const bool many = num_items >= 8ll * gridDim.x;
      uint32_t u_next = 0;          // many: the number drawn ahead
      uint32_t e_b = 0, e_hp = 0;   // many: the entry read ahead
      bool e_ok = false;
      // (inline: the compiler's form of a one-lane atomicAdd waits for the result at once)
      auto draw = [&] {
        uint32_t u;
        asm volatile("atom.global.add.u32 %0, [%1], 1;" : "=r"(u) : "l"(&p.ws_header[2]) : "memory");
        return u;
      };
      auto read_entry = [&](uint32_t u) {
        e_ok = u < num_items;
        if (e_ok) {
          e_b = p.items[2ll * u];
          e_hp = p.items[2ll * u + 1];
        }
      };
      // what decode() will read of the next sequence, on its way to the L1
      auto prefetch_next = [&] {
        if (!e_ok || e_b >= static_cast<uint32_t>(p.batch)) return;
        auto line = [&](const void* base, long long i) {
          if (base) asm volatile("prefetch.global.L1 [%0];" ::"l"(static_cast<const char*>(base) + i * p.index_bytes));
        };
        line(p.offq, e_b);
        line(p.offq, e_b + 1ll);
        line(p.offk, e_b);
        line(p.offk, e_b + 1ll);
        line(p.ctx, e_b);
        line(p.tgt, e_b);
        if (p.paged_split) line(p.page_offsets, e_b);
      };
      bool second = false;   // the pair's other tile is still to come
      ShTile pair = {};
      auto decode = [&]() -> ShTile {
        ShTile t = {};
        if (second) {
          second = false;
          t = pair;
          t.r0 -= kTileM;
        } else {
          uint32_t u = 0;
          if (!many) {
            u = draw();
            read_entry(u >> 1);
          }
          if (!e_ok) return t;
          t.b = static_cast<int>(e_b);
          t.h = static_cast<int>(e_hp >> 16);
          t.r0 = static_cast<int>(e_hp & 0xffffu) * kPairM;
          // an entry that does not name a (sequence, head) of this call does nothing (inconsistent offsets only)
          const bool bad = t.b < 0 || t.b >= p.batch || t.h >= p.hq;
          if (bad) t.b = 0, t.h = 0;
          t.hk = t.h / p.gqa_ratio;
          t.s = load_seq(p, t.b);
          if (bad) t.s.lq = t.s.lk = 0;
          if (p.paged_split) {
            long long pg0 = load_index(p.page_offsets, p.index_bytes, t.b), pg1 = load_index(p.page_offsets, p.index_bytes, t.b + 1);
            if (pg0 < 0) pg0 = 0;
            if (pg1 > p.num_page_ids) pg1 = p.num_page_ids;
            t.first_slot = pg0;
            t.pages = pg1 > pg0 ? static_cast<int>(pg1 - pg0) : 0;
          }
          if (!many) {
            t.r0 += (1 - static_cast<int>(u & 1)) * kTileM;
          } else if (t.r0 + kTileM < t.s.lq) {   // the later tile now, the first one next
            t.r0 += kTileM;
            second = true;
            pair = t;
          }
          if (many) {
            read_entry(u_next);
            u_next = draw();
          }
        }
        const int seen = kv_tiles_for_rows(t.s, t.r0, kTileM, p.mask_type, 1);   // keys [0, seen) are visited
        t.split = p.paged_split ? t.s.lk - t.s.tgt : t.s.lk;
        t.n_first = ((seen < t.split ? seen : t.split) + kShKeys - 1) / kShKeys;
        t.n = t.n_first + (seen > t.split ? (seen - t.split + kShKeys - 1) / kShKeys : 0);
        t.valid = 1;
        return t;
      };
      // page `i` of the tile's sequence (-1: the table has none)
      auto page = [&](const ShTile& t, int i) -> long long {
        return p.paged_split && i < t.pages ? load_index(p.page_ids, p.index_bytes, t.first_slot + i) : -1;
      };
      uint32_t q_uses = 0, ring_pos = 0, bias_pos = 0;
      if (many) {
        read_entry(draw());
        u_next = draw();
      }
      ShTile t = decode();
      for (uint32_t k = 0;; ++k) {
        const uint32_t slot = k % kShItems;
        long long pid_next = page(t, 0);   // (read ahead of its use, here and below)
        w.wait(ptx::smem_u32(&bars->item_free[slot]), ((k / kShItems) & 1u) ^ 1u);
        if (w.aborted()) break;   // a wait gave up somewhere: every role leaves when it sees the flag
        bars->item[slot] = t;
        ptx::mbar_arrive(ptx::smem_u32(&bars->item_full[slot]));
        if (!t.valid) break;
        if (t.n > 0) {
          const uint32_t qf = ptx::smem_u32(&bars->q_full);
          w.wait(ptx::smem_u32(&bars->q_free), (q_uses & 1u) ^ 1u);
          if (w.aborted()) break;
          ptx::mbar_expect_tx(qf, halves_qk * C::kQHalf);
          const int qrow = static_cast<int>(t.s.q0) + t.r0;
#pragma unroll
          for (int hf = 0; hf < C::kHalves; ++hf)
            if (hf < halves_qk) ptx::tma_load_3d(sm_q + hf * C::kQHalf, &tm_q, qf, hf * 64, t.h, qrow);
          ++q_uses;
          long long pid = 0;
          for (int j = 0; j < t.n; ++j) {
            const bool from_cache = p.paged_split && j < t.n_first;
            int row = static_cast<int>(t.s.k0) + j * kShKeys, in_page = 0;
            if (from_cache) {
              in_page = (j * kShKeys) % p.page_size;
              if (in_page == 0) {
                pid = pid_next;   // (an id outside the cache reads as zeros: the coordinate lies past the tensor)
                if (pid < 0 || pid >= p.num_pages) pid = p.num_pages;
                pid_next = page(t, (j * kShKeys) / p.page_size + 1);
              }
            } else if (p.paged_split) {
              row = static_cast<int>(t.s.q0) + t.s.lq - t.s.tgt + (j - t.n_first) * kShKeys;
            }
#pragma unroll
            for (int kv = 0; kv < 2; ++kv) {
              const uint32_t stage = ring_pos % C::kStages;
              const uint32_t full = ptx::smem_u32(&bars->kv_full[stage]);
              w.wait(ptx::smem_u32(&bars->kv_free[stage]), ((ring_pos / C::kStages) & 1u) ^ 1u);
              if (w.aborted()) break;
              const int halves = kv == 0 ? halves_qk : halves_v;
              ptx::mbar_expect_tx(full, halves * C::kKvHalf);
              const CUtensorMap* tm = from_cache ? &tm_cache : (kv == 0 ? &tm_k : &tm_v);
              const int trow = from_cache ? static_cast<int>((pid * 2 + kv) * p.page_size) + in_page : row;
#pragma unroll
              for (int hf = 0; hf < C::kHalves; ++hf)
                if (hf < halves) ptx::tma_load_3d(sm_ring + stage * C::kKvBytes + hf * C::kKvHalf, tm, full, hf * 64, t.hk, trow);
              ++ring_pos;
              if (kBias && kv == 0) {
                const uint32_t bb = bias_pos % C::kBiasBufs;
                const uint32_t bfull = ptx::smem_u32(&bars->bias_full[bb]);
                w.wait(ptx::smem_u32(&bars->bias_free[bb]), ((bias_pos / C::kBiasBufs) & 1u) ^ 1u);
                if (w.aborted()) break;
                ptx::mbar_expect_tx(bfull, C::kBiasBytes);
                const int brow = t.b * (p.bias_bstride ? p.hq * p.maxq : 0) + t.h * p.maxq + t.r0;
                ptx::tma_load_2d(sm_bias + bb * C::kBiasBytes, &tm_bias, bfull, j * kShKeys, brow);
                ++bias_pos;
              }
            }
            if (w.aborted()) break;
            if (j == 0 && many && !second) prefetch_next();
          }
        }
        t = decode();
      }
      // Drain (matters only after an abort): every load this thread issued has landed before the CTA exits.
      auto drain = [&](uint64_t* bar, uint32_t uses) {
        if (uses == 0) return;
        for (int spin = 0; spin < (1 << 22) && !ptx::mbar_try_wait(ptx::smem_u32(bar), (uses - 1) & 1u); ++spin) {}
      };
      drain(&bars->q_full, q_uses);
      for (uint32_t s = 0; s < C::kStages; ++s) drain(&bars->kv_full[s], (ring_pos + C::kStages - 1 - s) / C::kStages);
      if (kBias)
        for (uint32_t s = 0; s < C::kBiasBufs; ++s)
          drain(&bars->bias_full[s], (bias_pos + C::kBiasBufs - 1 - s) / C::kBiasBufs);
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer
    if (ptx::elect_one()) {
      constexpr uint32_t idesc_qk = ptx::umma_idesc_f16(Pack<T>::kFormat, kTileM, kShKeys, 0);
      const uint32_t idesc_pv = ptx::umma_idesc_f16(Pack<T>::kFormat, kTileM, p.dv, 1);
      const bool half_k = p.dqk <= D / 2;   // the upper half of the contraction holds nothing but zeros
      constexpr uint64_t kDescK = ptx::umma_desc_sw128_hi(16, 1024);
      constexpr uint64_t kDescV = ptx::umma_desc_sw128_hi(C::kKvHalf, 1024);
      const uint64_t qbase = kDescK | static_cast<uint64_t>(sm_q >> 4);
      const uint32_t bar_s = ptx::smem_u32(&bars->s_full), bar_p = ptx::smem_u32(&bars->p_full);
      uint32_t ring_pos = 0, q_uses = 0, p_uses = 0, o_uses = 0;
      for (uint32_t k = 0;; ++k) {
        const uint32_t slot = k % kShItems;
        w.wait(ptx::smem_u32(&bars->item_full[slot]), (k / kShItems) & 1u);
        if (w.aborted()) break;
        const int n = bars->item[slot].n, valid = bars->item[slot].valid, lk = bars->item[slot].s.lk;
        const int split = bars->item[slot].split, n_first = bars->item[slot].n_first;
        ptx::mbar_arrive(ptx::smem_u32(&bars->item_free[slot]));
        if (!valid) break;
        if (n == 0) continue;
        // S = Q . K(j)^T.  Issued right behind P(j - 1).V(j - 1), whose P it overwrites: products of one thread run in
        // order.
        auto qk = [&](int j) {
          const uint32_t st = ring_pos % C::kStages;
          w.wait(ptx::smem_u32(&bars->kv_full[st]), (ring_pos / C::kStages) & 1u);
          if (j == 0) w.wait(ptx::smem_u32(&bars->q_full), q_uses & 1u);
          if (w.aborted()) return;
          ptx::tc_fence_after();
          const uint64_t kbase = kDescK | static_cast<uint64_t>((sm_ring + st * C::kKvBytes) >> 4);
          auto one = [&](int ks) {
            const uint64_t qoff = static_cast<uint64_t>(((ks >> 2) * C::kQHalf + (ks & 3) * 32) >> 4);
            const uint64_t koff = static_cast<uint64_t>(((ks >> 2) * C::kKvHalf + (ks & 3) * 32) >> 4);
            ptx::mma_ss(tmem, qbase + qoff, kbase + koff, idesc_qk, ks > 0 ? 1u : 0u);
          };
#pragma unroll
          for (int ks = 0; ks < D / 32; ++ks) one(ks);
          if (!half_k) {
#pragma unroll
            for (int ks = D / 32; ks < D / 16; ++ks) one(ks);
          }
          ptx::mma_commit(bar_s);
          ptx::mma_commit(ptx::smem_u32(&bars->kv_free[st]));
          ++ring_pos;
          if (j == n - 1) {
            ptx::mma_commit(ptx::smem_u32(&bars->q_free));
            ++q_uses;
          }
        };
        qk(0);
        for (int j = 0; j < n; ++j) {
          // O (+)= P(j) . V(j); the P / O warps have waited for a V tile that a sequence end cuts before they hand P over
          const uint32_t st = ring_pos % C::kStages;
          w.wait(ptx::smem_u32(&bars->kv_full[st]), (ring_pos / C::kStages) & 1u);
          if (j == 0) w.wait(ptx::smem_u32(&bars->o_free), (o_uses & 1u) ^ 1u);
          w.wait(bar_p, p_uses & 1u);
          if (w.aborted()) break;
          ptx::tc_fence_after();
          const uint64_t vbase = kDescV | static_cast<uint64_t>((sm_ring + st * C::kKvBytes) >> 4);
          // (16-key products wholly behind the segment's end are left out)
          const int keys = j < n_first ? split - j * kShKeys : lk - split - (j - n_first) * kShKeys;
#pragma unroll
          for (int ks = 0; ks < kShKeys / 16; ++ks)
            ptx::mma_ts_if(ks * 16 < keys ? 1u : 0u, tmem + kShColO, tmem + ks * 8,
                           vbase + static_cast<uint64_t>((ks * 2048) >> 4), idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          ptx::mma_commit(ptx::smem_u32(&bars->kv_free[st]));
          ++p_uses;
          ++ring_pos;
          if (j == n - 1) {
            ptx::mma_commit(ptx::smem_u32(&bars->o_full));
            ++o_uses;
          } else {
            qk(j + 1);
          }
        }
        if (w.aborted()) break;
      }
      // all MMAs (and the arrivals of their commits) complete before the CTA tears down
      ptx::mma_commit(ptx::smem_u32(&bars->done));
      for (int spin = 0; spin < (1 << 22) && !ptx::mbar_try_wait(ptx::smem_u32(&bars->done), 0); ++spin) {}
    }
  } else {
    // ------------------------------------------------------------------ P / O (thread = row)
    const int row = threadIdx.x;
    const uint32_t t_s = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    constexpr bool kExact = Pack<T>::kExact;
    const float c_in = kExact ? p.alpha : 0.5f * p.alpha;   // (the tanh form: on half the argument)
    auto arrive_warp = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(bar));
    };
    // (the warp's lanes act on one answer: what follows a wait is warp-wide)
    auto stopped = [&] { return __any_sync(0xffffffffu, w.aborted()) != 0; };
    uint32_t s_uses = 0, o_uses = 0, ring_base = 0, bias_pos = 0;
    for (uint32_t k = 0;; ++k) {
      const uint32_t slot = k % kShItems;
      w.wait(ptx::smem_u32(&bars->item_full[slot]), (k / kShItems) & 1u);
      if (stopped()) break;
      const ShTile& in = bars->item[slot];
      const int valid = in.valid, n = in.n, r0 = in.r0, lq = in.s.lq, lk = in.s.lk;
      const int split = in.split, n_first = in.n_first;
      const int i_row = r0 + row;
      const bool row_ok = i_row < lq;
      RowBounds rb = {0, 1, 0};
      T* orow = nullptr;
      int full_end = 0;   // tiles that end at or before this key are visible to every row of the Q tile (tile_is_full's rule)
      if (valid) {
        const SeqInfo s = in.s;
        if (lq > 0) rb = row_bounds(s, row_ok ? i_row : lq - 1, p.mask_type, p.group);
        orow = static_cast<T*>(p.out) + ((s.q0 + i_row) * p.hq + in.h) * p.dv;
        full_end = lk;
        if (p.mask_type == HSTU_MASK_TRIL) {
          const int causal = r0 + (lk - lq) + 1;
          if (causal < full_end) full_end = causal;
          const int r1 = r0 + kTileM - 1 < lq - 1 ? r0 + kTileM - 1 : lq - 1;
          if (s.tgt > 0 && p.group > 0 && r1 >= lq - s.tgt && lk - s.tgt < full_end) full_end = lk - s.tgt;
        }
      }
      arrive_warp(&bars->item_free[slot]);
      if (!valid) break;
      bool ok = true;
      for (int j = 0; j < n; ++j) {
        const int c0 = j < n_first ? j * kShKeys : split + (j - n_first) * kShKeys;
        const int rem = (j < n_first ? split : lk) - c0;
        const uint32_t bb = bias_pos % C::kBiasBufs;
        if (kBias) w.wait(ptx::smem_u32(&bars->bias_full[bb]), (bias_pos / C::kBiasBufs) & 1u);
        if (rem < kShKeys && (rem & 15)) {
          // the V tile holds foreign rows behind the segment's end: P is 0 there, but 0 x NaN is not.  The rows
          // up to the next multiple of 16 (at most 120 pieces of 16 bytes per half) are zeroed; the products stop there.
          const uint32_t pos = ring_base + 2u * j + 1u, st = pos % C::kStages;
          w.wait(ptx::smem_u32(&bars->kv_full[st]), (pos / C::kStages) & 1u);
          if (row < (16 - (rem & 15)) * 8) {
#pragma unroll
            for (int hf = 0; hf < C::kHalves; ++hf)
              ptx::st_shared_zero16(sm_ring + st * C::kKvBytes + hf * C::kKvHalf + rem * 128 + row * 16);
            ptx::fence_proxy_async();
          }
        }
        w.wait(ptx::smem_u32(&bars->s_full), s_uses & 1u);
        ok = !stopped();
        if (!ok) break;
        ++s_uses;
        ptx::tc_fence_after();
        const uint32_t brow = sm_bias + bb * C::kBiasBytes + row * 128, bswz = row & 7;
        if (c0 + kShKeys <= full_end && rem >= kShKeys)
          short_p<T, kBias, false>(t_s, brow, bswz, rb, c0, rem, c_in, p.scale);
        else
          short_p<T, kBias, true>(t_s, brow, bswz, rb, c0, rem, c_in, p.scale);
        if (kBias) ptx::fence_proxy_async();   // the bias tile's buffer goes back to TMA: its reads come first
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
        arrive_warp(&bars->p_full);
        if (kBias) {
          if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->bias_free[bb]));
          ++bias_pos;
        }
      }
      if (!ok) break;
      ring_base += 2u * n;
      if (n == 0) {   // nothing visible: zeros
        if (row_ok)
          for (int c = 0; c < p.dv; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
        continue;
      }
      w.wait(ptx::smem_u32(&bars->o_full), o_uses & 1u);
      if (stopped()) break;
      ++o_uses;
      ptx::tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < D / 32; ++ch) {
        if (ch * 32 >= p.dv) continue;
        uint32_t orr[32];
        ptx::tmem_ld32(t_s + kShColO + ch * 32, orr);
        ptx::tmem_wait_ld_dep(orr);
        if (row_ok) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 u;
            u.x = Pack<T>::pack(__uint_as_float(orr[q4 * 8 + 0]), __uint_as_float(orr[q4 * 8 + 1]));
            u.y = Pack<T>::pack(__uint_as_float(orr[q4 * 8 + 2]), __uint_as_float(orr[q4 * 8 + 3]));
            u.z = Pack<T>::pack(__uint_as_float(orr[q4 * 8 + 4]), __uint_as_float(orr[q4 * 8 + 5]));
            u.w = Pack<T>::pack(__uint_as_float(orr[q4 * 8 + 6]), __uint_as_float(orr[q4 * 8 + 7]));
            if (ch * 32 + q4 * 8 < p.dv) *reinterpret_cast<uint4*>(orow + ch * 32 + q4 * 8) = u;
          }
        }
      }
      ptx::tc_fence_before();
      arrive_warp(&bars->o_free);
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, C::kTmemCols);
  }
}

template <int D, typename T, bool kBias>
cudaError_t launch_inst(const KParams& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                        const CUtensorMap& mb, const CUtensorMap& mc, int num_sms, cudaStream_t stream) {
  using C = ShCfg<D, kBias>;
  auto kern = hstu_short_kernel<D, T, kBias>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
  if (e != cudaSuccess) return e;
  const long long want = 2 * p.item_capacity, most = static_cast<long long>(num_sms) * C::kPerSm;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(want < 1 ? 1 : want < most ? want : most));
  cfg.blockDim = dim3(kShThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // start while the pre-pass is still running
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p, mq, mk, mv, mb, mc);
}

}  // namespace

// Whether a call goes to this kernel rather than hstu_tc.cu's (asked for calls that one supports, without a custom mask,
// the bias absent or tiled by TMA).  A chain here takes longer per key than there (half the keys per step), an SM holds
// more of them: short sequences gain always, longer ones when there are chains enough to fill the SMs, very long ones
// never, except where the other kernel's second Q tile would stay empty.  Measured, us there -> here, 4 heads of width D,
// bf16, B200:
//   D = 64   2000 sequences of mean 300: 417 -> 318, with a bias 470 -> 450; 870 of mean 600: 499 -> 430; 220 of 2400: equal
//            without, 1439 -> 1579 with a bias; 14 of mean 600: 21 -> 30; 27 of mean 300: equal
//            hstu_paged, 16-80 queries per sequence: 512 of mean 1000: 238 -> 184; 64 of 1000: 53 -> 61
//   D = 128  8700 of mean 60: 649 -> 481; 3500 of mean 150: 460 -> 487; 220 of 2400: 1453 -> 2105
//            hstu_paged: 2048 of mean 300: 510 -> 433; 512 of 1000: 292 -> 270; 8 of 1000: 38 -> 44
//
// Means do not show a single long sequence, whose chain is what such a batch then waits for: its last Q tile - both of a
// pair, one after the other, in calls of many items - takes 1.65 us per 64 keys here, 125 us of 8192 keys there.  So the
// longest chain the call allows has to fit the time the other kernel needs for the batch as such, about 2 us a pair and
// 9 us per 1000 keys of its sequences on each SM; with hstu_paged that kernel has the gather in front of it.  (max_seq_len_k
// stands for the longest length, which only the device knows.)  D = 64, 512 sequences of mean 80: 36 here, 47 there; and one
// more of 1024: 39 / 49, of 2048: 65 / 53, of 8192: 234 / 157; 2048 of mean 80 and one of 2048: 122 / 157, of 4096:
// 206 / 172; 1024 of mean 300 and one of 2048: 193 / 249, of 8192: 409 / 313; 300 of mean 800 and one of 8192: 271 / 330.
// hstu_paged, 512 of mean 350 and one of 4096: 104 / 126, of 16384: 306 / 224.  No call takes the other kernel less than
// some 5.5 us beside its launches: a few sequences of at most 192 rows 10.6 here, 11.5 there; of 256: 12.3 / 11.7.
static bool short_rule(const KParams& p, long long mean_k, bool in_place) {
  const bool wide = p.dqk > 64 || p.dv > 64;
  const long long mean_q = p.total_q / p.batch;
  if (mean_k >= (wide ? 96 : 320)) {
    const long long tiles = p.hq * (p.total_q / kTileM > p.batch ? p.total_q / kTileM : p.batch);
    if (tiles < kFewItems) return false;
    if (mean_q >= 96 && (wide || mean_k >= 1024)) return false;
  }
  const long long in_pairs = p.total_q / kPairM + p.batch / 2;
  const double pairs = static_cast<double>(p.hq) * (in_pairs > p.batch ? in_pairs : p.batch);
  const bool many = pairs >= 8.0 * 148 * (wide ? 2 : p.bias ? 3 : 4) && p.maxq > kTileM;
  const double chain_us = p.maxk * (in_place ? 0.011 : many ? 0.05 : 0.026);
  const double batch_us = (in_place ? 4.0 : 0.0) + pairs / 148 * (2.0 + 0.009 * mean_k);
  return chain_us <= (batch_us > 5.5 ? batch_us : 5.5);
}
bool short_preferred(const KParams& p) {
  if (p.paged_split) return true;                     // (decided by short_paged_split)
  if (p.batch <= 0 || p.paged_direct) return false;   // (cache pages beside staging tensors: hstu_tc.cu)
  return short_rule(p, p.total_k / p.batch, false);
}

// Whether an hstu_paged call can run here without staging anything: K / V tiles of 64 keys lie in one page, and no bias - a
// bias tile of the targets would start at any column, TMA wants multiples of 16 bytes.
bool short_paged_split(const KParams& p) {
  const uintptr_t align = reinterpret_cast<uintptr_t>(p.kv_cache) | reinterpret_cast<uintptr_t>(p.k_new) |
                          reinterpret_cast<uintptr_t>(p.v_new);
  if (p.batch <= 0 || p.mask_type == HSTU_MASK_CUSTOM || p.bias || p.page_size % kShKeys != 0 || (align & 15u) != 0 ||
      p.num_pages > 0x7fffff00ll / 2 / p.page_size)
    return false;
  // (the cached keys are not known here: all pages, each sequence's last one half full)
  return short_rule(p, (p.num_page_ids * p.page_size + p.total_q) / p.batch - p.page_size / 2, true);
}

// Returns cudaSuccess, a CUDA error, or cudaErrorNotSupported when a tensor map could not be encoded.
cudaError_t launch_short(const KParams& p, int dtype, const CUtensorMap& mq, const CUtensorMap& mb, int num_sms,
                         cudaStream_t stream) {
  CUtensorMap mk, mv, mbs = mb;
  const long long rows = p.paged_split ? p.total_q : p.total_k;
  if (!make_kv_tile_map(&mk, p.paged_split ? p.k_new : p.k, rows, p.hk, p.dqk, dtype, kShKeys) ||
      !make_kv_tile_map(&mv, p.paged_split ? p.v_new : p.v, rows, p.hk, p.dv, dtype, kShKeys))
    return cudaErrorNotSupported;
  CUtensorMap mc = mk;
  if (p.paged_split &&
      !make_kv_tile_map(&mc, p.kv_cache, p.num_pages * 2 * p.page_size, p.hk, p.dqk, dtype, kShKeys))
    return cudaErrorNotSupported;
#define HSTU_SHORT_CASE(DD, TT)                                                     \
  return p.bias ? launch_inst<DD, TT, true>(p, mq, mk, mv, mbs, mc, num_sms, stream) \
                : launch_inst<DD, TT, false>(p, mq, mk, mv, mbs, mc, num_sms, stream)
  const bool wide = p.dqk > 64 || p.dv > 64;
  if (dtype == HSTU_DTYPE_BF16) {
    if (!tanh_silu(p)) {
      if (wide) { HSTU_SHORT_CASE(128, Bf16Exp); }
      HSTU_SHORT_CASE(64, Bf16Exp);
    }
    if (wide) { HSTU_SHORT_CASE(128, __nv_bfloat16); }
    HSTU_SHORT_CASE(64, __nv_bfloat16);
  }
  if (wide) { HSTU_SHORT_CASE(128, __half); }
  HSTU_SHORT_CASE(64, __half);
#undef HSTU_SHORT_CASE
}

}  // namespace hstu
