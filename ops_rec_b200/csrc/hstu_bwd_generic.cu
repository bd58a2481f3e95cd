// HSTU jagged backward on CUDA cores: fp32 products and fp32 accumulation for every input type, any head dims,
// every mask form.  Two kernels, both without atomics (bitwise reproducible), each in a register-tiled form with tiles
// of 32 rows (hstu_simt_bwd_*, hstu_simt.cuh: head dims that are multiples of 4 up to 128, aligned rows) and a form for
// everything else with tiles of 16 rows:
//
//   hstu_bwd_dq_kernel    one CTA per (sequence, query head, q-tile): walks the visible K tiles, recomputes
//                         S = Q.K^T and dP = dO.V^T, forms dS, writes that tile of d_bias, accumulates dQ = dS.K.
//                         It also writes the zeros of its d_bias rows outside the visible region, so the caller
//                         need not clear d_bias (the reference adapter clears it with zeros_like,
//                         hstu_v1/torch_extension/hstu_jagged_plugin.cpp:113-118).
//   hstu_bwd_dkv_kernel   one CTA per (sequence, key/value head, key tile): walks the query heads of the group
//                         and the q-tiles that can see the keys, recomputes S and dP, accumulates dV = P^T.dO and
//                         dK = dS^T.Q.
//
// Element-wise stage as in the reference kernel (hstu_backward_v1/op_kernel/vector_score.h:159-209):
//   x = alpha (S + bias);  sg = sigmoid(x) * M;  P = x * sg * scale;  dS = dP * scale * alpha * sg * (1 + x - x sg)
// with P and dS rounded to the input type before the products that consume them; d_bias = dS.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "hstu_common.cuh"
#include "hstu_simt.cuh"

namespace hstu {

namespace {

constexpr int BT = 16;          // tile edge (rows and keys)
constexpr int BTHREADS = 256;   // BT x BT threads
constexpr int BMAXC = 32;       // dims <= 512 -> at most 32 columns per thread

template <typename T> __device__ __forceinline__ float ld_f(const T* p) { return simt::to_float<T>(*p); }
template <typename T> __device__ __forceinline__ T cvt_f(float x) { return simt::from_float<T>(x); }

template <typename T> __device__ __forceinline__ float round_to(float x) {
  T t = cvt_f<T>(x);
  return ld_f<T>(&t);
}

// rows [r0, r0 + BT) of a [tokens, heads, dim] tensor, head h -> dst[BT][ld] (zeros past `len`)
template <typename T>
__device__ __forceinline__ void load_tile(float* dst, int ld, const T* src, long long tok0, int r0, int len, int heads,
                                          int h, int dim) {
  for (int idx = threadIdx.x; idx < BT * dim; idx += BTHREADS) {
    const int r = idx / dim, d = idx - r * dim;
    const int row = r0 + r;
    dst[r * ld + d] = row < len ? ld_f<T>(src + ((tok0 + row) * heads + h) * dim + d) : 0.f;
  }
}

template <typename T>
__device__ __forceinline__ float bias_at(const KParams& p, int b, int h, int i, int j) {
  return ld_f<T>(static_cast<const T*>(p.bias) + static_cast<long long>(b) * p.bias_bstride +
                 (static_cast<long long>(h) * p.maxq + i) * p.maxk + j);
}
// P (rounded) and dS (rounded) of element (i, j) from the raw dot products s = q_i.k_j and dp = dO_i.v_j.
// d_bias gets dS for the reference's x = alpha (S + bias) and dX for the alpha-before-bias variant.
// bv: bias_at(i, j) of a visible element (unused without a bias)
template <typename T>
__device__ __forceinline__ void score_grad(const KParams& p, int b, int h, int i, int j, bool visible, float s, float dp,
                                           float bv, float* p_out, float* ds_out, float* dbias_out) {
  // (selects, no branch around the arithmetic: a thread has up to sixteen elements in a row)
  const bool alpha_first = (p.flags & HSTU_FLAG_ALPHA_BEFORE_BIAS) != 0;
  float x = s;
  if (p.bias) x = alpha_first ? fmaf(x, p.alpha, bv) : (x + bv) * p.alpha;
  else x *= p.alpha;
  float m = 1.f;
  if (p.mask_type == HSTU_MASK_CUSTOM && visible) {
    const long long moff = ((static_cast<long long>(b) * p.hq + h) * p.maxq + i) * p.maxk + j;
    m = ld_f<T>(static_cast<const T*>(p.mask) + moff);
  }
  const float sg = simt::divide(1.f, 1.f + expf(-x));
  const float dx = dp * p.scale * m * sg * (1.f + x * (1.f - sg));
  const float pv = visible ? round_to<T>(x * sg * p.scale * m) : 0.f;
  const float ds = visible ? round_to<T>(dx * p.alpha) : 0.f;
  const float db = visible ? (alpha_first ? round_to<T>(dx) : round_to<T>(dx * p.alpha)) : 0.f;
  *p_out = pv;
  *ds_out = ds;
  *dbias_out = db;
}

template <typename T>
__global__ void __launch_bounds__(BTHREADS) hstu_bwd_dq_kernel(const BwdParams bp) {
  extern __shared__ float smem[];
  const KParams& p = bp.f;
  const int bh = blockIdx.x;
  const int b = bh / p.hq;
  const int h = bh - b * p.hq;
  const int hk = h / p.gqa_ratio;
  const int r0 = blockIdx.y * BT;
  const SeqInfo s = load_seq(p, b);
  const int tid = threadIdx.x;
  const int tx = tid & (BT - 1), ty = tid >> 4;
  T* dbias = static_cast<T*>(bp.dbias);
  const long long brow0 = (static_cast<long long>(b) * p.hq + h) * p.maxq;  // first bias row of (b, h)

  const int ntiles = kv_tiles_for_rows(s, r0, BT, p.mask_type, BT);
  if (dbias) {
    // zeros of this CTA's d_bias rows: everything right of the visited tiles (all columns when none is visited)
    const int first = ntiles * BT;
    const int width = p.maxk - first;
    if (width > 0) {
      for (int idx = tid; idx < BT * width; idx += BTHREADS) {
        const int r = idx / width, c = idx - r * width;
        if (r0 + r < p.maxq) dbias[(brow0 + r0 + r) * p.maxk + first + c] = cvt_f<T>(0.f);
      }
    }
  }
  if (ntiles == 0) return;

  const int dq = p.dqk, dv = p.dv;
  const int ldq = dq + 1, ldv = dv + 1;  // +1 float: conflict-free column reads
  float* Qs = smem;               // [BT][ldq]
  float* Gs = Qs + BT * ldq;      // [BT][ldv]   dO rows
  float* Ks = Gs + BT * ldv;      // [BT][ldq]
  float* Vs = Ks + BT * ldq;      // [BT][ldv]
  float* Ds = Vs + BT * ldv;      // [BT][BT]    dS

  load_tile<T>(Qs, ldq, static_cast<const T*>(p.q), s.q0, r0, s.lq, p.hq, h, dq);
  load_tile<T>(Gs, ldv, static_cast<const T*>(bp.dout), s.q0, r0, s.lq, p.hq, h, dv);

  const int i = r0 + ty;
  const RowBounds rb = row_bounds(s, i < s.lq ? i : s.lq - 1, p.mask_type, p.group);
  float acc[BMAXC];
#pragma unroll
  for (int c = 0; c < BMAXC; ++c) acc[c] = 0.f;
  const int ncol = (dq + BT - 1) / BT;

  for (int t = 0; t < ntiles; ++t) {
    const int c0 = t * BT;
    __syncthreads();  // the previous tile's Ks / Vs / Ds are consumed (and, for t == 0, Qs / Gs are filled)
    load_tile<T>(Ks, ldq, static_cast<const T*>(p.k), s.k0, c0, s.lk, p.hk, hk, dq);
    load_tile<T>(Vs, ldv, static_cast<const T*>(p.v), s.k0, c0, s.lk, p.hk, hk, dv);
    __syncthreads();
    float sc = 0.f, dp = 0.f;
    for (int d = 0; d < dq; ++d) sc = fmaf(Qs[ty * ldq + d], Ks[tx * ldq + d], sc);
    for (int d = 0; d < dv; ++d) dp = fmaf(Gs[ty * ldv + d], Vs[tx * ldv + d], dp);
    const int j = c0 + tx;
    const bool visible = i < s.lq && j < s.lk && allowed(rb, j);
    float pv, ds, db;
    score_grad<T>(p, b, h, i, j, visible, sc, dp, visible && p.bias ? bias_at<T>(p, b, h, i, j) : 0.f, &pv, &ds, &db);
    Ds[ty * BT + tx] = ds;
    if (dbias && i < p.maxq && j < p.maxk) dbias[(brow0 + i) * p.maxk + j] = cvt_f<T>(db);
    __syncthreads();
    for (int kk = 0; kk < BT; ++kk) {
      const float d = Ds[ty * BT + kk];
#pragma unroll
      for (int c = 0; c < BMAXC; ++c) {
        if (c < ncol) {
          const int col = tx + BT * c;
          acc[c] = fmaf(d, col < dq ? Ks[kk * ldq + col] : 0.f, acc[c]);
        }
      }
    }
  }
  if (i < s.lq) {
    T* row = static_cast<T*>(bp.dq) + ((s.q0 + i) * p.hq + h) * dq;
#pragma unroll
    for (int c = 0; c < BMAXC; ++c) {
      const int col = tx + BT * c;
      if (c < ncol && col < dq) row[col] = cvt_f<T>(acc[c]);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(BTHREADS) hstu_bwd_dkv_kernel(const BwdParams bp) {
  extern __shared__ float smem[];
  const KParams& p = bp.f;
  const int bh = blockIdx.x;
  const int b = bh / p.hk;
  const int hk = bh - b * p.hk;
  const int c0 = blockIdx.y * BT;
  const SeqInfo s = load_seq(p, b);
  if (c0 >= s.lk) return;
  const int tid = threadIdx.x;
  const int tx = tid & (BT - 1), ty = tid >> 4;

  const int dq = p.dqk, dv = p.dv;
  const int ldq = dq + 1, ldv = dv + 1;
  float* Ks = smem;               // [BT][ldq]
  float* Vs = Ks + BT * ldq;      // [BT][ldv]
  float* Qs = Vs + BT * ldv;      // [BT][ldq]
  float* Gs = Qs + BT * ldq;      // [BT][ldv]
  float* Ps = Gs + BT * ldv;      // [BT][BT]  P  (row = query)
  float* Ds = Ps + BT * BT;       // [BT][BT]  dS (row = query)

  load_tile<T>(Ks, ldq, static_cast<const T*>(p.k), s.k0, c0, s.lk, p.hk, hk, dq);
  load_tile<T>(Vs, ldv, static_cast<const T*>(p.v), s.k0, c0, s.lk, p.hk, hk, dv);

  float acc_k[BMAXC], acc_v[BMAXC];
#pragma unroll
  for (int c = 0; c < BMAXC; ++c) acc_k[c] = acc_v[c] = 0.f;
  const int ncol_k = (dq + BT - 1) / BT, ncol_v = (dv + BT - 1) / BT;
  const int ktile = c0 / BT;
  const int j = c0 + tx;

  for (int hh = 0; hh < p.gqa_ratio; ++hh) {
    const int h = hk * p.gqa_ratio + hh;
    for (int r0 = 0; r0 < s.lq; r0 += BT) {
      if (kv_tiles_for_rows(s, r0, BT, p.mask_type, BT) <= ktile) continue;  // no row of this q-tile sees these keys
      __syncthreads();  // the previous Qs / Gs / Ps / Ds are consumed (and, first time, Ks / Vs are filled)
      load_tile<T>(Qs, ldq, static_cast<const T*>(p.q), s.q0, r0, s.lq, p.hq, h, dq);
      load_tile<T>(Gs, ldv, static_cast<const T*>(bp.dout), s.q0, r0, s.lq, p.hq, h, dv);
      __syncthreads();
      const int i = r0 + ty;
      const RowBounds rb = row_bounds(s, i < s.lq ? i : s.lq - 1, p.mask_type, p.group);
      float sc = 0.f, dp = 0.f;
      for (int d = 0; d < dq; ++d) sc = fmaf(Qs[ty * ldq + d], Ks[tx * ldq + d], sc);
      for (int d = 0; d < dv; ++d) dp = fmaf(Gs[ty * ldv + d], Vs[tx * ldv + d], dp);
      const bool visible = i < s.lq && j < s.lk && allowed(rb, j);
      float pv, ds, db;
      score_grad<T>(p, b, h, i, j, visible, sc, dp, visible && p.bias ? bias_at<T>(p, b, h, i, j) : 0.f, &pv, &ds, &db);
      Ps[ty * BT + tx] = pv;
      Ds[ty * BT + tx] = ds;
      __syncthreads();
      // this thread now owns key `ty` and the columns tx, tx + 16, ...
      for (int ii = 0; ii < BT; ++ii) {
        const float pe = Ps[ii * BT + ty], de = Ds[ii * BT + ty];
#pragma unroll
        for (int c = 0; c < BMAXC; ++c) {
          const int col = tx + BT * c;
          if (c < ncol_v) acc_v[c] = fmaf(pe, col < dv ? Gs[ii * ldv + col] : 0.f, acc_v[c]);
          if (c < ncol_k) acc_k[c] = fmaf(de, col < dq ? Qs[ii * ldq + col] : 0.f, acc_k[c]);
        }
      }
    }
  }
  const int key = c0 + ty;
  if (key < s.lk) {
    T* krow = static_cast<T*>(bp.dk) + ((s.k0 + key) * p.hk + hk) * dq;
    T* vrow = static_cast<T*>(bp.dv) + ((s.k0 + key) * p.hk + hk) * dv;
#pragma unroll
    for (int c = 0; c < BMAXC; ++c) {
      const int col = tx + BT * c;
      if (c < ncol_k && col < dq) krow[col] = cvt_f<T>(acc_k[c]);
      if (c < ncol_v && col < dv) vrow[col] = cvt_f<T>(acc_v[c]);
    }
  }
}

// ------------------------------------------------------------------------------------ register-tiled form
// Rows of the streamed tile: 64, or 32 at width 128 (two CTAs on an SM instead of one).
template <int kDim> constexpr int kStream = kDim > 64 ? 32 : 64;

template <typename T, int kDim>
__global__ void __launch_bounds__(simt::kThreads) hstu_simt_bwd_dq_kernel(const BwdParams bp) {
  extern __shared__ float smem[];
  constexpr int kN = kStream<kDim>, kCols = kN / 16, kPer = simt::OutCols<kDim>::kPer;
  constexpr int ld = kDim + 4, ldp = kN + 4;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const KParams& p = bp.f;
  const int b = blockIdx.x / p.hq, h = blockIdx.x - b * p.hq;
  const int hk = h / p.gqa_ratio;
  const int r0 = static_cast<int>(gridDim.y - 1 - blockIdx.y) * simt::kRows;   // the rows with the most keys first
  const SeqInfo s = load_seq(p, b);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T* dbias = static_cast<T*>(bp.dbias);
  const long long brow0 = (static_cast<long long>(b) * p.hq + h) * p.maxq;
  const int seen = kv_tiles_for_rows(s, r0, simt::kRows, p.mask_type, 32) * 32;
  const int end = seen < s.lk ? seen : s.lk;
  const int ntiles = (end + kN - 1) / kN;
  if (dbias) {
    // zeros of this CTA's d_bias rows: everything right of the visited tiles (all columns when none is visited)
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < simt::kRows && r0 + r < p.maxq; r += simt::kThreads / 32)
      for (int c = ntiles * kN + lane; c < p.maxk; c += 32) dbias[(brow0 + r0 + r) * p.maxk + c] = cvt_f<T>(0.f);
  }
  if (r0 < s.lq) {
    const int dq = p.dqk, dv = p.dv;
    float* Qs = smem;                     // [32][ld]
    float* Gs = Qs + simt::kRows * ld;    // [32][ld]   dO rows
    float* Ks = Gs + simt::kRows * ld;    // [kN][ld]
    float* Vs = Ks + kN * ld;             // [kN][ld]
    float* Ds = Vs + kN * ld;             // [32][ldp]  dS
    const T* k = static_cast<const T*>(p.k);
    const T* v = static_cast<const T*>(p.v);
    RowBounds rb[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = r0 + 4 * ty + r;
      rb[r] = row_bounds(s, i, p.mask_type, p.group);
      if (i >= s.lq) rb[r].lim1 = 0, rb[r].lo2 = 1, rb[r].hi2 = 0;   // (a row past the end sees nothing)
    }
    float acc[4][kPer];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < kPer; ++c) acc[r][c] = 0.f;
    if (ntiles > 0) {
      simt::load_rows<T, simt::kRows, kDim>(Qs, ld, static_cast<const T*>(p.q), s.q0, r0, s.lq, p.hq, h, dq);
      simt::load_rows<T, simt::kRows, kDim>(Gs, ld, static_cast<const T*>(bp.dout), s.q0, r0, s.lq, p.hq, h, dv);
      simt::load_rows<T, kN, kDim>(Ks, ld, k, s.k0, 0, s.lk, p.hk, hk, dq);
      simt::load_rows<T, kN, kDim>(Vs, ld, v, s.k0, 0, s.lk, p.hk, hk, dv);
      simt::cp_async_commit();
    }
    for (int t = 0; t < ntiles; ++t) {
      const int c0 = t * kN;
      float bv[4][kCols];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int i = r0 + 4 * ty + r, j = c0 + tx + 16 * c;
          bv[r][c] = p.bias && allowed(rb[r], j) ? bias_at<T>(p, b, h, i, j) : 0.f;
        }
      simt::cp_async_wait<0>();
      __syncthreads();
      float sc[4][kCols], dp[4][kCols];
      simt::dot_tile<kCols>(Qs + 4 * ty * ld, ld, Ks + tx * ld, ld, dq, sc);
      simt::dot_tile<kCols>(Gs + 4 * ty * ld, ld, Vs + tx * ld, ld, dv, dp);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int i = r0 + 4 * ty + r, j = c0 + tx + 16 * c;
          float pv, ds, db;
          score_grad<T>(p, b, h, i, j, allowed(rb[r], j), sc[r][c], dp[r][c], bv[r][c], &pv, &ds, &db);
          Ds[(4 * ty + r) * ldp + tx + 16 * c] = ds;
          if (dbias && i < p.maxq && j < p.maxk) dbias[(brow0 + i) * p.maxk + j] = cvt_f<T>(db);
        }
      __syncthreads();   // Ds is there; V_t is consumed
      if (t + 1 < ntiles) simt::load_rows<T, kN, kDim>(Vs, ld, v, s.k0, c0 + kN, s.lk, p.hk, hk, dv);
      const int left = (end - c0 + 3) & ~3;   // (rows of K between lk and the next multiple of four are zeros)
      simt::outer_tile<kDim>(Ds + 4 * ty * ldp, ldp, Ks, ld, left < kN ? left : kN, tx, acc);
      __syncthreads();   // K_t and Ds are consumed
      if (t + 1 < ntiles) simt::load_rows<T, kN, kDim>(Ks, ld, k, s.k0, c0 + kN, s.lk, p.hk, hk, dq);
      simt::cp_async_commit();
    }
    simt::cp_async_wait<0>();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = r0 + 4 * ty + r;
      if (i < s.lq) simt::store_row<T, kDim>(static_cast<T*>(bp.dq) + ((s.q0 + i) * p.hq + h) * dq, dq, tx, acc[r]);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (the pre-pass: nothing here reads what it wrote)
}

template <typename T, int kDim>
__global__ void __launch_bounds__(simt::kThreads) hstu_simt_bwd_dkv_kernel(const BwdParams bp) {
  extern __shared__ float smem[];
  constexpr int kN = kStream<kDim>, kCols = kN / 16, kPer = simt::OutCols<kDim>::kPer;
  constexpr int ld = kDim + 4, ldp = kN + 4;
  const KParams& p = bp.f;
  const int b = blockIdx.x / p.hk, hk = blockIdx.x - b * p.hk;
  const int c0 = blockIdx.y * simt::kRows;   // (the first keys are seen by the most queries)
  const SeqInfo s = load_seq(p, b);
  if (c0 < s.lk) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int dq = p.dqk, dv = p.dv;
    float* Ks = smem;                     // [32][ld]
    float* Vs = Ks + simt::kRows * ld;    // [32][ld]
    float* Qs = Vs + simt::kRows * ld;    // [kN][ld]
    float* Gs = Qs + kN * ld;             // [kN][ld]   dO rows
    float* Ps = Gs + kN * ld;             // [32][ldp]  P^T  (row = key)
    float* Ds = Ps + simt::kRows * ldp;   // [32][ldp]  dS^T (row = key)
    const T* q = static_cast<const T*>(p.q);
    const T* g = static_cast<const T*>(bp.dout);
    // Query tiles that see a key of this tile, one after the other: u = (query head of the group) * per_head + tile.
    const int per_head = (s.lq + kN - 1) / kN, count = per_head * p.gqa_ratio, ktile = c0 / simt::kRows;
    auto next = [&](int u) {
      while (u < count && kv_tiles_for_rows(s, (u % per_head) * kN, kN, p.mask_type, simt::kRows) <= ktile) ++u;
      return u;
    };
    float acc_k[4][kPer], acc_v[4][kPer];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < kPer; ++c) acc_k[r][c] = acc_v[r][c] = 0.f;
    int u = next(0);
    if (u < count) {
      const int h = hk * p.gqa_ratio + u / per_head, r0 = (u % per_head) * kN;
      simt::load_rows<T, simt::kRows, kDim>(Ks, ld, static_cast<const T*>(p.k), s.k0, c0, s.lk, p.hk, hk, dq);
      simt::load_rows<T, simt::kRows, kDim>(Vs, ld, static_cast<const T*>(p.v), s.k0, c0, s.lk, p.hk, hk, dv);
      simt::load_rows<T, kN, kDim>(Qs, ld, q, s.q0, r0, s.lq, p.hq, h, dq);
      simt::load_rows<T, kN, kDim>(Gs, ld, g, s.q0, r0, s.lq, p.hq, h, dv);
      simt::cp_async_commit();
    }
    while (u < count) {
      const int h = hk * p.gqa_ratio + u / per_head, r0 = (u % per_head) * kN;
      const int un = next(u + 1);
      const int hn = hk * p.gqa_ratio + un / per_head, rn = (un % per_head) * kN;
      RowBounds rb[kCols];
      float bv[4][kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int i = r0 + tx + 16 * c;
        rb[c] = row_bounds(s, i, p.mask_type, p.group);
        if (i >= s.lq) rb[c].lim1 = 0, rb[c].lo2 = 1, rb[c].hi2 = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int j = c0 + 4 * ty + r;
          bv[r][c] = p.bias && allowed(rb[c], j) ? bias_at<T>(p, b, h, i, j) : 0.f;
        }
      }
      simt::cp_async_wait<0>();
      __syncthreads();
      float sc[4][kCols], dp[4][kCols];
      simt::dot_tile<kCols>(Ks + 4 * ty * ld, ld, Qs + tx * ld, ld, dq, sc);
      simt::dot_tile<kCols>(Vs + 4 * ty * ld, ld, Gs + tx * ld, ld, dv, dp);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const int i = r0 + tx + 16 * c, j = c0 + 4 * ty + r;
          float pv, ds, db;
          score_grad<T>(p, b, h, i, j, allowed(rb[c], j), sc[r][c], dp[r][c], bv[r][c], &pv, &ds, &db);
          Ps[(4 * ty + r) * ldp + tx + 16 * c] = pv;
          Ds[(4 * ty + r) * ldp + tx + 16 * c] = ds;
        }
      __syncthreads();
      const int left = (s.lq - r0 + 3) & ~3, kend = left < kN ? left : kN;   // (rows past the end are zeros)
      simt::outer_tile<kDim>(Ps + 4 * ty * ldp, ldp, Gs, ld, kend, tx, acc_v);
      __syncthreads();   // dO_i is consumed
      if (un < count) simt::load_rows<T, kN, kDim>(Gs, ld, g, s.q0, rn, s.lq, p.hq, hn, dv);
      simt::outer_tile<kDim>(Ds + 4 * ty * ldp, ldp, Qs, ld, kend, tx, acc_k);
      __syncthreads();   // Q_i and Ds are consumed
      if (un < count) simt::load_rows<T, kN, kDim>(Qs, ld, q, s.q0, rn, s.lq, p.hq, hn, dq);
      simt::cp_async_commit();
      u = un;
    }
    simt::cp_async_wait<0>();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int j = c0 + 4 * ty + r;
      if (j >= s.lk) continue;
      simt::store_row<T, kDim>(static_cast<T*>(bp.dk) + ((s.k0 + j) * p.hk + hk) * dq, dq, tx, acc_k[r]);
      simt::store_row<T, kDim>(static_cast<T*>(bp.dv) + ((s.k0 + j) * p.hk + hk) * dv, dv, tx, acc_v[r]);
    }
  }
  // the dQ pass wrote nothing this one reads; the wait makes the stream's next operation find both complete
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename T, int kDim>
cudaError_t launch_simt_bwd(const BwdParams& bp, cudaStream_t stream) {
  const KParams& p = bp.f;
  constexpr int kN = kStream<kDim>;
  constexpr int tiles = 2 * (simt::kRows + kN) * (kDim + 4), part = simt::kRows * (kN + 4);
  constexpr int smem_q = 4 * (tiles + part), smem_kv = 4 * (tiles + 2 * part);
  cudaError_t e = cudaFuncSetAttribute(hstu_simt_bwd_dq_kernel<T, kDim>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_q);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(hstu_simt_bwd_dkv_kernel<T, kDim>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_kv);
  if (e != cudaSuccess) return e;
  const dim3 grid_q(static_cast<unsigned>(p.batch) * p.hq, (p.maxq + simt::kRows - 1) / simt::kRows, 1);
  e = simt::launch(hstu_simt_bwd_dq_kernel<T, kDim>, grid_q, smem_q, stream, bp);
  if (e != cudaSuccess) return e;
  const dim3 grid_k(static_cast<unsigned>(p.batch) * p.hk, (p.maxk + simt::kRows - 1) / simt::kRows, 1);
  return simt::launch(hstu_simt_bwd_dkv_kernel<T, kDim>, grid_k, smem_kv, stream, bp);
}

// The register-tiled kernels wherever their loads are possible.  (16 sequences of 50-500 rows, 2 heads of 64, fp32, forward
// and backward: 158 us, 1239 us with the other kernels.)
bool simt_bwd_supported(const BwdParams& bp, int dtype) {
  return simt::dims_ok(bp.f) && simt::aligned_to(bp.f.q, dtype) && simt::aligned_to(bp.f.k, dtype) &&
         simt::aligned_to(bp.f.v, dtype) && simt::aligned_to(bp.dout, dtype) && simt::aligned_to(bp.dq, dtype) &&
         simt::aligned_to(bp.dk, dtype) && simt::aligned_to(bp.dv, dtype);
}

template <typename T>
cudaError_t launch_bwd_t(const BwdParams& bp, int dtype, cudaStream_t stream) {
  const KParams& p = bp.f;
  if (simt_bwd_supported(bp, dtype)) {
    switch (simt::tile_dim(p)) {
      case 32: return launch_simt_bwd<T, 32>(bp, stream);
      case 64: return launch_simt_bwd<T, 64>(bp, stream);
      default: return launch_simt_bwd<T, 128>(bp, stream);
    }
  }
  const size_t tile = static_cast<size_t>(BT) * (p.dqk + 1) + static_cast<size_t>(BT) * (p.dv + 1);
  const size_t smem_q = sizeof(float) * (2 * tile + BT * BT);
  const size_t smem_kv = sizeof(float) * (2 * tile + 2 * BT * BT);
  cudaError_t e = cudaFuncSetAttribute(hstu_bwd_dq_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem_q));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(hstu_bwd_dkv_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem_kv));
  if (e != cudaSuccess) return e;
  dim3 grid_q(static_cast<unsigned>(p.batch) * p.hq, (p.maxq + BT - 1) / BT, 1);
  hstu_bwd_dq_kernel<T><<<grid_q, BTHREADS, smem_q, stream>>>(bp);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  dim3 grid_k(static_cast<unsigned>(p.batch) * p.hk, (p.maxk + BT - 1) / BT, 1);
  hstu_bwd_dkv_kernel<T><<<grid_k, BTHREADS, smem_kv, stream>>>(bp);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_bwd_generic(const BwdParams& bp, int dtype, cudaStream_t stream) {
  switch (dtype) {
    case HSTU_DTYPE_BF16: return launch_bwd_t<__nv_bfloat16>(bp, dtype, stream);
    case HSTU_DTYPE_FP16: return launch_bwd_t<__half>(bp, dtype, stream);
    default: return launch_bwd_t<float>(bp, dtype, stream);
  }
}

}  // namespace hstu
