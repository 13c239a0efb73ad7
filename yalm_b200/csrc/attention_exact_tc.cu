// Prefill attention on tcgen05 WITHOUT rounding the softmax weights (see attention_exact.cu for the
// arithmetic and for what a query sees: a sliding window or everything before it, pooled blocks that
// lie wholly before the window, kept first positions beside it): S = Q.K^T from the 16-bit q and k
// with 32-bit sums; scale, masks, maxima, exponentials and their sum in 32 bits; each weight as three
// 16-bit terms, p = hi + mid + lo, and O += lo.V + mid.V + hi.V into the same 32-bit accumulators.
//
// The form is attention_tc.cu's: 256 query tokens of one head per block as two tiles of 128 rows, a TMA
// producer, one issuing warp per tile, one softmax warpgroup per tile with a query row per thread,
// keys and values in blocks of 64 through TMA rings that serve both tiles.  What differs is tensor
// memory: the terms of P take 96 columns of a tile where the rounded form takes 32, so a tile has one
// S buffer (hi and mid go back over its 64 columns, lo into 32 of its own) beside its O, and the
// block's products come in the order S(i), P.V(i), S(i + 1); while one tile's rows are in their
// softmax the other tile's products run.  Bound by the tensor cores: three P.V products a block.
//
// The keys of a block of queries come from up to five places, each a run of key blocks of 64 rows:
// pooled rows; kept first positions that lie before the earliest window, cached or of this step; the
// ring, walked in blocks of its rows as in attention_tc.cu; and the step's own rows.  V's rows that no query
// of the block sees are cleared between copy and product (ta_clear_foreign_rows).
// The mma.sync kernel that these head sizes took before: 196 us for 2,048 tokens of 16 heads of 128
// behind a window of 1,024 with pooled blocks; here 62. Three causal prompts of 2,150 tokens in all: 132 -> 50.
#include "api.h"
#include "attention_tc.cuh"

namespace yalm {

constexpr int XT_THREADS = 352;
constexpr int XT_MMA_B = 10;       // the warp that issues tile B's products (warp 1: tile A's)
constexpr int XT_STAGES = 3;
constexpr float XT_RAISE = 8.f;    // a block's maximum may exceed the reference by this much (log2)
constexpr int XT_TILE_COLS = 256;  // tensor memory columns of a tile: S / hi, mid 64; lo 32; O HD

struct ExactTcArgs {
  const int *q_start, *seq_slot, *slot_pos, *page_table, *pool_table;
  int pps, n_pages, capacity;                     // the cache
  int pool, pool_pps, pool_pages, pool_capacity;  // pooled rows (pool 0: none)
  int keep;                                       // > 0: positions below it stay visible
  int H, G, window;
  float scale_log2;
  int* status;
};

__device__ __forceinline__ void xt_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// two neighbouring 16-bit values as floats
template <typename T> __device__ __forceinline__ float2 xt_unpack(uint32_t u);
template <> __device__ __forceinline__ float2 xt_unpack<__nv_bfloat16>(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
template <> __device__ __forceinline__ float2 xt_unpack<__half>(uint32_t u) {
  return __half22float2(*reinterpret_cast<const __half2*>(&u));
}

template <int HD, typename T16>
__global__ void __launch_bounds__(XT_THREADS)
attn_exact_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_step,
                     const __grid_constant__ CUtensorMap map_pk, const __grid_constant__ CUtensorMap map_pv,
                     const ExactTcArgs a, T16* __restrict__ out) {
  constexpr uint32_t FMT = std::is_same<T16, __nv_bfloat16>::value ? 1u : 0u;   // operand format
  constexpr int SUB = HD / 64;                     // 64-column sub-tiles of a head
  constexpr int Q_BYTES = TA_BM * HD * 2;          // one query tile
  constexpr int KV_BYTES = TA_BN * HD * 2;         // one block of K or of V
  constexpr int TMEM_COLS = 2 * XT_TILE_COLS;
  static_assert(64 + 32 + HD <= XT_TILE_COLS, "a tile's columns");
  extern __shared__ uint8_t xt_smem[];
  __shared__ __align__(8) uint64_t q_full, s_full[2], p_ready[2], pv_done[2];
  __shared__ __align__(8) uint64_t k_full[XT_STAGES], k_empty[XT_STAGES], v_full[XT_STAGES], v_empty[XT_STAGES];
  __shared__ __align__(8) uint64_t v_landed;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // heads run fastest, then sequences; a sequence's blocks come from its end: long blocks start first
  const int b = blockIdx.y, h = blockIdx.x;
  const int g = h / (a.H / a.G), H = a.H, G = a.G, window = a.window;
  const int qs = __shfl_sync(0xffffffffu, a.q_start[b], 0);      // written by a host copy: safe early
  const int q_len = __shfl_sync(0xffffffffu, a.q_start[b + 1], 0) - qs;
  const int slot = __shfl_sync(0xffffffffu, a.seq_slot[b], 0);
  // (positions are written by the advance kernel alone, which lets nothing start before it has ended)
  const int past = __shfl_sync(0xffffffffu, a.slot_pos[slot], 0);
  const int n_blocks = (q_len + 2 * TA_BM - 1) / (2 * TA_BM);
  if ((int)blockIdx.z >= n_blocks) return;
  const int m0 = (n_blocks - 1 - (int)blockIdx.z) * 2 * TA_BM;
  int t_m0[2], t_rows[2], t_kb0[2], t_kb1[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    t_m0[x] = m0 + x * TA_BM;
    t_rows[x] = max(0, min(TA_BM, q_len - t_m0[x]));
  }
  // ---- the runs of key blocks: [pooled | front, cached | front, step | ring | step]
  const int j_lo = first_visible(past + m0, window);             // the earliest position inside a window
  const int last_pos = past + m0 + t_rows[0] + t_rows[1] - 1;
  const int n_pooled = a.pool > 0 && window > 0 ? max(0, last_pos - window + 1) / a.pool : 0;
  const int n_front = a.keep > 0 ? min(a.keep, j_lo) : 0;        // kept positions before that
  const int front_cached = min(n_front, past);
  const int e_pool = (n_pooled + TA_BN - 1) / TA_BN;
  const int e_fc = e_pool + (front_cached + TA_BN - 1) / TA_BN;
  const int e_fs = e_fc + (n_front - front_cached + TA_BN - 1) / TA_BN;
  const int cap = a.capacity, n_rb = (cap + TA_BN - 1) / TA_BN;
  const int last_row = past > 0 ? (past - 1) % cap : 0;          // the newest row of the ring
  int n_ring = 0, rb0 = 0, step0 = 0;
  bool whole = false;                                            // the first ring block is also the newest one's
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    const int lo = max(first_visible(past + t_m0[x], window), past - cap);
    int first;
    if (lo < past) {
      const int r = lo % cap, rb = r / TA_BN;
      if (x == 0) {
        rb0 = rb;
        n_ring = last_row / TA_BN - rb + 1 + (r <= last_row ? 0 : n_rb);
        whole = n_ring > n_rb;
        n_ring = min(n_ring, n_rb);
      }
      first = whole ? 0 : rb - rb0 + (rb < rb0 ? n_rb : 0);
    } else {
      const int sb = (lo - past) / TA_BN;
      if (x == 0) step0 = sb * TA_BN;
      first = n_ring + sb - step0 / TA_BN;
    }
    // tile B starts where its window does, unless something before its window stays visible to it
    t_kb0[x] = e_fs > 0 || a.keep > 0 ? 0 : e_fs + first;
    t_kb1[x] = t_rows[x] > 0 ? e_fs + n_ring + (t_m0[x] + t_rows[x] - step0 + TA_BN - 1) / TA_BN : t_kb0[x];
  }
  const int e_ring = e_fs + n_ring;
  const int n_it = t_rows[1] > 0 ? t_kb1[1] : t_kb1[0];          // tile A starts at block 0

  const uint32_t base = (smem_u32(xt_smem) + 1023u) & ~1023u;
  const uint32_t q_s = base;                                     // tiles A and B
  const uint32_t k_s = q_s + 2 * Q_BYTES;
  const uint32_t v_s = k_s + XT_STAGES * KV_BYTES;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&q_full), 1);
    for (int x = 0; x < 2; ++x) {
      mbar_init(smem_u32(&s_full[x]), 1);
      mbar_init(smem_u32(&p_ready[x]), TA_BM);
      mbar_init(smem_u32(&pv_done[x]), 1);
    }
    mbar_init(smem_u32(&v_landed), 1);
    for (int s = 0; s < XT_STAGES; ++s) {
      mbar_init(smem_u32(&k_full[s]), 1);
      mbar_init(smem_u32(&k_empty[s]), 2);
      mbar_init(smem_u32(&v_full[s]), 1);
      mbar_init(smem_u32(&v_empty[s]), 2);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  volatile int* abort_p = &abort_flag;
  pdl_launch_dependents();

  if (warp == 0) {
    // ---------------- TMA producer: the whole warp runs the loop, lane 0 issues
    const bool issuer = lane == 0;
    pdl_wait();
    if (issuer) {
      const int n_tiles = t_rows[1] > 0 ? 2 : 1;
      mbar_expect_tx(smem_u32(&q_full), n_tiles * Q_BYTES);
      for (int x = 0; x < n_tiles; ++x)
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
          ta_tma_load_2d(q_s + x * Q_BYTES + sub * (TA_BM * 128), &map_q, h * HD + sub * 64, qs + t_m0[x],
                         smem_u32(&q_full));
    }
    // the stage of V whose rows no query of this block sees are still to be cleared (-1: none), and how many were
    int pending = -1, cleared = 0;
    uint64_t pending_live = 0;
    auto clear_pending = [&]() {
      const int s = pending;
      pending = -1;
      return ta_clear_foreign_rows<HD>(v_s + s * KV_BYTES, pending_live, smem_u32(&v_landed), cleared++ & 1,
                                       smem_u32(&v_full[s]), lane, abort_p);
    };
    for (int it = 0; it < n_it; ++it) {
      // the block's first row in its maps, the columns of K and of V, and which of its rows some query of
      // this block sees: row i of lane i, rows 32 + i beside it
      const CUtensorMap *mk = &map_k, *mv = &map_v;
      int row, col_k = 0, col_v = 0;
      bool seen[2];
      if (it < e_pool) {
        mk = &map_pk;
        mv = &map_pv;
        row = a.pool_table != nullptr
                  ? (g * a.pool_pages + a.pool_table[(size_t)slot * a.pool_pps + it]) * KV_PAGE
                  : (slot * G + g) * a.pool_capacity + it * TA_BN;
#pragma unroll
        for (int i = 0; i < 2; ++i) seen[i] = it * TA_BN + 32 * i + lane < n_pooled;
      } else if (it < e_fc || (it >= e_fs && it < e_ring)) {
        int cb = it - e_pool;                                    // the block of the cache's rows
        if (it >= e_fs) {
          cb = rb0 + it - e_fs;
          if (cb >= n_rb) cb -= n_rb;
        }
        row = a.page_table != nullptr ? (g * a.n_pages + a.page_table[(size_t)slot * a.pps + cb]) * KV_PAGE
                                      : (slot * G + g) * cap + cb * TA_BN;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = cb * TA_BN + 32 * i + lane;
          seen[i] = it < e_fc ? r < front_cached
                              : r < cap && past - 1 - last_row + r - (r > last_row ? cap : 0) >= j_lo;
        }
      } else {
        mk = mv = &map_step;
        col_k = g * HD;
        col_v = (G + g) * HD;
        const int t = it < e_fs ? (it - e_fc) * TA_BN : step0 + (it - e_ring) * TA_BN;
        row = qs + t;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int key = past + t + 32 * i + lane;
          seen[i] = it < e_fs ? key < n_front : key >= j_lo && key <= last_pos;
        }
      }
      const uint64_t live = (uint64_t)__ballot_sync(0xffffffffu, seen[1]) << 32 | __ballot_sync(0xffffffffu, seen[0]);
      const int s = it % XT_STAGES;
      const uint32_t phase = ((it / XT_STAGES) & 1) ^ 1u;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&k_empty[s]), phase, abort_p))) break;
      if (issuer) {
        mbar_expect_tx(smem_u32(&k_full[s]), KV_BYTES);
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
          ta_tma_load_2d(k_s + s * KV_BYTES + sub * (TA_BN * 128), mk, col_k + sub * 64, row, smem_u32(&k_full[s]));
      }
      // (the stages waited for above and below held block it - 3, whose products need no later block)
      if (pending >= 0 && !clear_pending()) break;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&v_empty[s]), phase, abort_p))) break;
      if (~live) {
        pending = s;
        pending_live = live;
      }
      if (issuer) {
        const uint32_t bar = ~live ? smem_u32(&v_landed) : smem_u32(&v_full[s]);
        mbar_expect_tx(bar, KV_BYTES);
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
          ta_tma_load_2d(v_s + s * KV_BYTES + sub * (TA_BN * 128), mv, col_v + sub * 64, row, bar);
      }
    }
    if (pending >= 0) clear_pending();
  } else if (warp == 1 || warp == XT_MMA_B) {
    // ---------------- MMA issuers, one per tile: the whole warp runs the loop, lane 0 issues
    const int x = warp == 1 ? 0 : 1;
    const uint32_t leader = lane == 0 ? 1u : 0u;
    // S: M = 128 queries, N = 64 keys, both operands K-major;  O += P.V: N = HD, V MN-major
    const uint32_t idesc_s = (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(TA_BN >> 3) << 17) |
                             ((uint32_t)(TA_BM >> 4) << 24);
    const uint32_t idesc_pv = (1u << 4) | (FMT << 7) | (FMT << 10) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) |
                              ((uint32_t)(TA_BM >> 4) << 24);
    const uint64_t q_desc = ta_desc_k(q_s + x * Q_BYTES);
    const uint32_t my_s = tmem_base + x * XT_TILE_COLS, my_o = my_s + 96;
    const int my_kb0 = x ? t_kb0[1] : t_kb0[0], my_kb1 = x ? t_kb1[1] : t_kb1[0];
    const uint32_t bar_s = smem_u32(&s_full[x]), bar_p = smem_u32(&p_ready[x]), bar_pv = smem_u32(&pv_done[x]);
    auto mine = [&](int kb) { return kb >= my_kb0 && kb < my_kb1; };
    // S of block `it`, once its keys have landed.  A stage is free once both issuers have committed it
    // (also the one whose tile does not see the block: it waits for the stage all the same, so that
    // a stage gets one arrival per issuer and filling).
    auto product_s = [&](int it) {
      const int s = it % XT_STAGES;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&k_full[s]), (it / XT_STAGES) & 1, abort_p))) return false;
      if (mine(it)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t k_desc = ta_desc_k(k_s + s * KV_BYTES);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          ta_umma_by(leader, my_s, q_desc + (uint64_t)(((ks / 4) * (TA_BM * 128) + (ks % 4) * 32) >> 4),
                     k_desc + (uint64_t)(((ks / 4) * (TA_BN * 128) + (ks % 4) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
        ta_commit_by(leader, bar_s);
      }
      ta_commit_by(leader, smem_u32(&k_empty[s]));
      return true;
    };
    bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&q_full), 0, abort_p));
    if (ok && n_it > 0) ok = product_s(0);
    for (int it = 0; it < n_it && ok; ++it) {
      const int s = it % XT_STAGES;
      const bool pv = mine(it);
      if (pv) {
        // P of this block is in tensor memory, S has been read, O is rescaled
        ok = __all_sync(0xffffffffu, mbar_wait(bar_p, (uint32_t)(it - my_kb0) & 1u, abort_p));
        if (!ok) break;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&v_full[s]), (it / XT_STAGES) & 1, abort_p));
      if (!ok) break;
      if (pv) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t v_desc = ta_desc_mn(v_s + s * KV_BYTES, TA_BN * 128);
        // the smallest terms first
#pragma unroll
        for (int term = 2; term >= 0; --term)
#pragma unroll
          for (int kk = 0; kk < TA_BN / 16; ++kk)
            ta_umma_tmem_a_by(leader, my_o, my_s + term * 32 + kk * 8, v_desc + (uint64_t)((kk * 16 * 128) >> 4),
                              idesc_pv, (it == my_kb0 && term == 2 && kk == 0) ? 0u : 1u);
        ta_commit_by(leader, bar_pv);
      }
      ta_commit_by(leader, smem_u32(&v_empty[s]));
      // the tensor core runs its instructions in order: S of the next block goes over this block's P
      if (it + 1 < n_it) ok = product_s(it + 1);
    }
  } else {
    // ---------------- softmax: one query row per thread; warps 2-5 tile A, 6-9 tile B
    const int x = warp >= 6 ? 1 : 0;
    const int quarter = warp & 3;                                // the TMEM lanes this warp may touch
    const int row = quarter * 32 + lane;
    const int my_m0 = x ? t_m0[1] : t_m0[0], my_rows = x ? t_rows[1] : t_rows[0];
    const int my_kb0 = x ? t_kb0[1] : t_kb0[0], my_kb1 = x ? t_kb1[1] : t_kb1[0];
    const int p = past + my_m0 + row;                            // this row's position
    const int p_hi = past + my_m0 + TA_BM - 1;
    const int p_lo = first_visible(p, window);                   // the first key of this row's window
    const int pooled_seen = n_pooled > 0 ? max(0, p - window + 1) / a.pool : 0;
    const uint32_t my_s = tmem_base + x * XT_TILE_COLS + ((uint32_t)(quarter * 32) << 16), my_o = my_s + 96;
    const uint32_t bar_s = smem_u32(&s_full[x]), bar_p = smem_u32(&p_ready[x]), bar_pv = smem_u32(&pv_done[x]);
    const float scale_log2 = a.scale_log2;
    float m_ref = -INFINITY, l_run = 0.f;
    pdl_wait();
    bool ok = true;
    const int n_x = my_kb1 - my_kb0;
    for (int i_blk = 0; i_blk < n_x; ++i_blk) {
      const int it = my_kb0 + i_blk;
      // every wait is decided per warp (the loads from tensor memory below are warp-wide)
      ok = __all_sync(0xffffffffu, mbar_wait(bar_s, i_blk & 1, abort_p));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[TA_BN];
      {
        uint32_t raw[TA_BN];
        ta_ld32_issue(my_s, raw);                                // both halves in flight, one wait
        ta_ld32_issue(my_s + 32, raw + 32);
        ta_ld_wait32(raw);
        ta_ld_after32(raw + 32);
#pragma unroll
        for (int i = 0; i < TA_BN; ++i) s[i] = __uint_as_float(raw[i]);
      }
      // masks: keys [lo, hi) of the block by index inside it, or position by position where the newest
      // row of the ring cuts the block in two
      if (it < e_fs) {
        const int hi = it < e_pool ? min(pooled_seen, n_pooled) - it * TA_BN
                     : it < e_fc ? front_cached - (it - e_pool) * TA_BN
                                 : n_front - past - (it - e_fc) * TA_BN;
        if (hi < TA_BN) {
#pragma unroll
          for (int i = 0; i < TA_BN; ++i) s[i] = i < hi ? s[i] : -INFINITY;
        }
      } else if (it < e_ring) {
        int cb = rb0 + it - e_fs;
        if (cb >= n_rb) cb -= n_rb;
        const int row0 = cb * TA_BN, newest = past - 1 - last_row;
        const int j0 = newest + row0 - (row0 > last_row ? cap : 0);
        const bool inside = j0 >= first_visible(p_hi, window) && j0 >= 0 &&
                            (last_row < row0 || last_row >= row0 + TA_BN - 1) && row0 + TA_BN <= cap;
        if (!inside) {
#pragma unroll
          for (int i = 0; i < TA_BN; ++i) {
            const int r = row0 + i;
            const int key = newest + r - (r > last_row ? cap : 0);
            s[i] = r < cap && key >= j_lo && (key >= p_lo || (key < a.keep && key >= 0)) ? s[i] : -INFINITY;
          }
        }
      } else {
        const int j0 = past + step0 + (it - e_ring) * TA_BN;
        if (!(j0 + TA_BN - 1 <= past + my_m0 && j0 >= first_visible(p_hi, window))) {
#pragma unroll
          for (int i = 0; i < TA_BN; ++i) {
            const int key = j0 + i;
            s[i] = key <= p && key >= j_lo && (key >= p_lo || key < a.keep) ? s[i] : -INFINITY;
          }
        }
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};                    // four chains instead of one
#pragma unroll
      for (int i = 4; i < TA_BN; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;
      const bool raise = m_blk > m_ref + XT_RAISE;               // always true for the first live block
      const float m_new = raise ? m_blk : m_ref;
      const float corr = raise ? ta_ex2(m_ref - m_new) : 1.f;
      const bool any_raise = __any_sync(0xffffffffu, raise);
      if (i_blk > 0 && any_raise) {                              // uniform over the warp; rare
        // O is rescaled once the previous block's product has been added to it
        ok = __all_sync(0xffffffffu, mbar_wait(bar_pv, (i_blk - 1) & 1, abort_p));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c = 0; c < HD; c += 32) {
          float v[32];
          ta_ld32(my_o + c, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] *= corr;
          ta_st32(my_o + c, v);
        }
      }
      m_ref = m_new;
      const float neg = m_ref > -INFINITY ? -m_ref : 0.f;
      float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const float2 scale2 = make_float2(scale_log2, scale_log2), neg2 = make_float2(neg, neg);
      const float2 minus = make_float2(-1.f, -1.f);
      // the terms of P, two keys per 32-bit column: hi and mid over the S columns they came from (S has been
      // read), lo beside them
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {                           // pairs of keys, in packed arithmetic
          const int i = part * 32 + 2 * j;
          const float2 t = __ffma2_rn(make_float2(s[i], s[i + 1]), scale2, neg2);
          const float2 e = make_float2(ta_ex2(t.x), ta_ex2(t.y));
          ls[j & 1] = __fadd2_rn(ls[j & 1], e);
          hi[j] = pack2<T16>(e.x, e.y);
          const float2 r = __ffma2_rn(xt_unpack<T16>(hi[j]), minus, e);       // exact
          mid[j] = pack2<T16>(r.x, r.y);
          const float2 r2 = __ffma2_rn(xt_unpack<T16>(mid[j]), minus, r);     // exact
          lo[j] = pack2<T16>(r2.x, r2.y);
        }
        xt_st16(my_s + part * 16, hi);
        xt_st16(my_s + 32 + part * 16, mid);
        xt_st16(my_s + 64 + part * 16, lo);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      l_run = l_run * corr + ((ls[0].x + ls[0].y) + (ls[1].x + ls[1].y));
      // P is complete for this row, S has been read, O is rescaled: the issuer may go on
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(bar_p);
    }
    if (ok && n_x > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar_pv, (n_x - 1) & 1, abort_p));
    if (ok && n_x > 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = 1.0f / l_run;
      T16* op = out + ((size_t)(qs + my_m0 + row) * H + h) * HD;
#pragma unroll 1
      for (int c = 0; c < HD; c += 32) {
        float v[32];
        ta_ld32(my_o + c, v);                                    // by the whole warp
        if (row < my_rows) {
#pragma unroll
          for (int c8 = 0; c8 < 32; c8 += 8) {
            uint4 u;
            u.x = pack2<T16>(v[c8 + 0] * inv, v[c8 + 1] * inv);
            u.y = pack2<T16>(v[c8 + 2] * inv, v[c8 + 3] * inv);
            u.z = pack2<T16>(v[c8 + 4] * inv, v[c8 + 5] * inv);
            u.w = pack2<T16>(v[c8 + 6] * inv, v[c8 + 7] * inv);
            *reinterpret_cast<uint4*>(op + c + c8) = u;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) atomicOr(a.status, ERR_WAIT_TIMEOUT);
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}

template <int HD, typename T16>
static int launch_exact_tc(const void* q, const void* kv_step, const void* k_cache, const void* v_cache,
                           long long cache_rows, const void* pool_k, const void* pool_v, long long pool_rows,
                           const ExactTcArgs& a, void* out, int n_tokens, int n_seqs, int max_q_len,
                           cudaStream_t stream) {
  constexpr bool half = std::is_same<T16, __half>::value;
  CUtensorMap mq, mk, mv, ms, mpk, mpv;
  int rc = ta_make_map(&mq, q, n_tokens, (long long)a.H * HD, TA_BM, half);
  if (!rc) rc = ta_make_map(&mk, k_cache, cache_rows, HD, TA_BN, half);
  if (!rc) rc = ta_make_map(&mv, v_cache, cache_rows, HD, TA_BN, half);
  if (!rc) rc = ta_make_map(&ms, kv_step, n_tokens, (long long)2 * a.G * HD, TA_BN, half);
  mpk = mk;
  mpv = mv;
  if (!rc && a.pool > 0) rc = ta_make_map(&mpk, pool_k, pool_rows, HD, TA_BN, half);
  if (!rc && a.pool > 0) rc = ta_make_map(&mpv, pool_v, pool_rows, HD, TA_BN, half);
  if (rc) return rc;
  // two query tiles, the K and V rings, slack to align to 1024
  const size_t smem = (size_t)2 * TA_BM * HD * 2 + (size_t)2 * XT_STAGES * TA_BN * HD * 2 + 1024;
  static bool attr_set = false;
  if (!attr_set) {
    const cudaError_t e =
        cudaFuncSetAttribute(attn_exact_tc_kernel<HD, T16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const dim3 grid(a.H, n_seqs, (max_q_len + 2 * TA_BM - 1) / (2 * TA_BM));
  launch_pdl(attn_exact_tc_kernel<HD, T16>, grid, dim3(XT_THREADS), smem, stream, mq, mk, mv, ms, mpk, mpv, a,
             (T16*)out);
  YALM_LAUNCH_CHECK();
  return 0;
}

}  // namespace yalm

using namespace yalm;

// yalm_attention_exact_prefill for head sizes 64 and 128 (same arguments and meaning, plus the sizes of
// the caches: n_slots, and n_tokens, and the status word for the bounded waits).  q_start, seq_slot and
// slot_pos are read before the wait on the previous kernel, the page tables after it.
extern "C" int yalm_attention_exact_tc(const void* q, const void* kv_step, const void* k_cache, const void* v_cache,
                                       const int* q_start, const int* seq_slot, const int* slot_pos, void* out,
                                       int dtype, int n_tokens, int n_seqs, int max_q_len, int n_slots, int H, int G,
                                       int hd, int capacity, int window, float scale, const int* page_table,
                                       int pages_per_slot, int n_pages, const void* pool_k, const void* pool_v,
                                       int pool, int pool_capacity, const int* pool_table, int pool_pps,
                                       int pool_pages, int keep_first, int* status, cudaStream_t stream) {
  if (n_seqs <= 0 || max_q_len <= 0 || n_tokens <= 0) return 0;
  if (hd != 64 && hd != 128) return -2;
  if (G <= 0 || H % G != 0 || window < 0 || (pool > 0 && window <= 0)) return -3;
  if (keep_first < 0 || (keep_first > 0 && (window <= 0 || pool > 0))) return -3;
  if (dtype != DT_BF16 && dtype != DT_F16) return -3;
  if (capacity <= 0 || n_slots <= 0 || (pool > 0 && pool_capacity <= 0)) return -4;
  if (n_seqs > 65535 || (max_q_len + 2 * TA_BM - 1) / (2 * TA_BM) > 65535) return -4;
  const long long rows = page_table != nullptr ? (long long)G * n_pages * KV_PAGE : (long long)n_slots * G * capacity;
  const long long prows = pool <= 0 ? 0
                          : pool_table != nullptr ? (long long)G * pool_pages * KV_PAGE
                                                  : (long long)n_slots * G * pool_capacity;
  if (rows <= 0 || rows > 0x7fffffffLL || prows > 0x7fffffffLL || (pool > 0 && prows <= 0)) return -4;
  if (((uintptr_t)q | (uintptr_t)kv_step | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out |
       (pool > 0 ? (uintptr_t)pool_k | (uintptr_t)pool_v : 0)) & 15)
    return -6;
  const ExactTcArgs a = {q_start, seq_slot, slot_pos, page_table, pool_table, pages_per_slot, n_pages, capacity,
                         pool > 0 ? pool : 0, pool_pps, pool_pages, pool_capacity, keep_first, H, G, window,
                         1.4426950408889634f * score_scale(scale, hd), status};
#define YALM_XT(HD, T) \
  return launch_exact_tc<HD, T>(q, kv_step, k_cache, v_cache, rows, pool_k, pool_v, prows, a, out, n_tokens, n_seqs, \
                                max_q_len, stream)
  if (dtype == DT_F16) {
    if (hd == 64) YALM_XT(64, __half);
    YALM_XT(128, __half);
  }
  if (hd == 64) YALM_XT(64, __nv_bfloat16);
  YALM_XT(128, __nv_bfloat16);
#undef YALM_XT
}
