// What follows a q/k(/v) product whose queries and keys are normed over the WHOLE projection
// (all heads of a token at once) and rotated on a part of each head:
//  * qk_norm_rope_store: sums the product's split-K slices (plus a bias per feature of the row, if
//    the projections have one), norms q and k (each over its whole
//    row, with a weight per feature), rotates the first `dims` features of every head -- pairs
//    (i, i + dims/2) or neighbours (2i, 2i+1) -- by pos * freq[i] with cos and sin times `mult`,
//    and writes q, this step's keys and values and the cache rows in the storage type.  The
//    values are the v rows of the product, or, when it has none, the keys as projected
//    (before norm and rotation).  With head_eps >= 0 every head of q and k is, AFTER its rotation,
//    divided by its own root mean square over head_size features (a norm without a weight);
//  * pool_blocks: the mean key and the mean value of every block of `pool` positions that
//    this step completes, from the rows as the cache holds them, into a second cache that has
//    one row per block.
// Norms, angles and means are 32-bit.
#include "api.h"
#include "common.cuh"

namespace yalm {

// grid (token, part): every block of a token sums the whole row (the norms need it), and writes
// its own part of the outputs; one part when there are many tokens.  The product's row is [q: H heads | k: G heads | v: G heads (if any)],
// every head hd wide (rows beyond a head's true size are zero).  n_q / n_k: the true number of
// features of q and k (what the mean of squares divides by).
template <typename T>
__global__ void qk_norm_rope_store_kernel(
    const float* __restrict__ qkv, int n_partials, long long partial_stride,
    const float* __restrict__ bias, const float* __restrict__ q_norm, const float* __restrict__ k_norm, float n_q, float n_k, float eps,
    const float* __restrict__ freq, int dims, int neighbours, float mult, float head_eps, float head_size,
    const int* __restrict__ token_seq, const int* __restrict__ q_start,
    const int* __restrict__ seq_slot, const int* __restrict__ slot_pos, T* __restrict__ q_out,
    T* __restrict__ kv_step, T* __restrict__ k_cache, T* __restrict__ v_cache, int H, int G, int hd,
    int has_v, int capacity, int write_cache, const int* __restrict__ page_table, int pps, int n_pages) {
  pdl_launch_dependents();
  extern __shared__ float row_s[];                       // the summed row, then dims / 2 (cos, sin) pairs
  __shared__ float scratch[33];
  const int t = blockIdx.x;
  const int b = token_seq[t];
  const int slot = seq_slot[b];
  const int qs = q_start[b], q_end = q_start[b + 1];
  const int past = slot_pos[slot];
  const int pos = past + (t - qs);
  const bool keep = write_cache && pos >= past + (q_end - qs) - capacity;
  pdl_wait();
  const int nq = H * hd, nk = G * hd;
  const int row = nq + nk + (has_v ? nk : 0);
  const float* src = qkv + (size_t)t * row;
  // the token's cosines and sines, once for all heads (the angle in 32 bits)
  float2* cs = reinterpret_cast<float2*>(row_s + ((row + 1) & ~1));
  for (int i = threadIdx.x; i < (dims >> 1); i += blockDim.x) {
    const float ang = (float)pos * freq[i];
    cs[i] = make_float2(cosf(ang) * mult, sinf(ang) * mult);
  }
  float ssq = 0.f, ssk = 0.f;
  for (int i = threadIdx.x; i < row; i += blockDim.x) {
    const float v = sum_slices(src + i, n_partials, partial_stride) + (bias != nullptr ? bias[i] : 0.f);
    row_s[i] = v;
    if (i < nq) ssq += v * v;
    else if (i < nq + nk) ssk += v * v;
  }
  float rq = 1.f, rk = 1.f;
  if (q_norm != nullptr) rq = 1.0f / sqrtf(block_sum(ssq, scratch) / n_q + eps);
  if (k_norm != nullptr) rk = 1.0f / sqrtf(block_sum(ssk, scratch) / n_k + eps);
  __syncthreads();
  const int half = dims >> 1;
  // a norm per head after the rotation: the rotated row replaces the summed one first
  float* head_r = reinterpret_cast<float*>(cs + half);              // [H + G]
  if (head_eps >= 0.f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    for (int head = warp; head < H + G; head += n_warps) {
      float* v = row_s + (size_t)head * hd;
      float ss = 0.f;
      if (neighbours) {
        for (int p = lane; p < half; p += 32) {
          const float a = v[2 * p], b2 = v[2 * p + 1];
          const float lo = rotate_lo(a, b2, cs[p].x, cs[p].y), hi = rotate_hi(a, b2, cs[p].x, cs[p].y);
          v[2 * p] = lo; v[2 * p + 1] = hi;
          ss += lo * lo + hi * hi;
        }
      } else {
        for (int p = lane; p < half; p += 32) {
          const float a = v[p], b2 = v[p + half];
          const float lo = rotate_lo(a, b2, cs[p].x, cs[p].y), hi = rotate_hi(a, b2, cs[p].x, cs[p].y);
          v[p] = lo; v[p + half] = hi;
          ss += lo * lo + hi * hi;
        }
      }
      for (int e = dims + lane; e < hd; e += 32) ss += v[e] * v[e];
      ss = warp_sum(ss);
      if (lane == 0) head_r[head] = 1.0f / sqrtf(ss / head_size + head_eps);
    }
    __syncthreads();
  }
  // this block's part of the outputs
  const int per_part = (nq + nk + gridDim.y - 1) / gridDim.y;
  const int i_lo = blockIdx.y * per_part, i_hi = min(nq + nk, i_lo + per_part);
  const int v_per = (nk + gridDim.y - 1) / gridDim.y;
  const int v_lo = blockIdx.y * v_per, v_hi = min(nk, v_lo + v_per);
  // q and k: norm, then rotate with the partner's normed value
  for (int i = i_lo + threadIdx.x; i < i_hi; i += blockDim.x) {
    const bool is_q = i < nq;
    const int j = is_q ? i : i - nq;                     // index inside q or k
    const int head = j / hd, e = j % hd;
    const float* w = is_q ? q_norm : k_norm;
    const float r = is_q ? rq : rk;
    float me = row_s[i] * (w != nullptr ? r * w[j] : 1.f);
    if (head_eps >= 0.f) {
      me *= head_r[is_q ? head : H + head];
    } else if (e < dims) {
      int pi, pair;                                       // partner's feature, pair number
      bool first;
      if (neighbours) { pi = e ^ 1; pair = e >> 1; first = !(e & 1); }
      else { first = e < half; pi = first ? e + half : e - half; pair = first ? e : e - half; }
      const int ip = i - e + pi;
      const int jp = j - e + pi;
      const float other = row_s[ip] * (w != nullptr ? r * w[jp] : 1.f);
      const float c = cs[pair].x, s = cs[pair].y;
      me = first ? rotate_lo(me, other, c, s) : rotate_hi(other, me, c, s);
    }
    const T val = from_float<T>(me);
    if (is_q) {
      q_out[(size_t)t * nq + j] = val;
    } else {
      kv_step[((size_t)t * 2 * G + head) * hd + e] = val;
      if (keep)
        k_cache[kv_row_offset(page_table, pps, n_pages, slot, head, G, capacity, pos % capacity, hd) + e] = val;
    }
  }
  // values: the v rows, or the keys as they were projected
  const float* vs = row_s + nq + (has_v ? nk : 0);
  for (int j = v_lo + threadIdx.x; j < v_hi; j += blockDim.x) {
    const int head = j / hd, e = j % hd;
    const T val = from_float<T>(vs[j]);
    kv_step[((size_t)t * 2 * G + G + head) * hd + e] = val;
    if (keep)
      v_cache[kv_row_offset(page_table, pps, n_pages, slot, head, G, capacity, pos % capacity, hd) + e] = val;
  }
}

// The same for rows that 16-byte accesses reach (head size a multiple of 4, rotated features of 4 in
// neighbouring pairs and of 8 in halves): a warp per head, a lane four features and, in halves, their
// four partners, so that a lane rotates what it has loaded itself, a norm per head is one warp sum,
// and both whole-row norms are one exchange between the warps.  Bound by its bytes and by how many
// tokens' loads are in flight: loads of all heads go out before the token's cosines are formed.
// grid (token, part) as above; ONE: the product is one slice.
// (2,280 tokens of 16 + 4 + 4 heads of 128 with a norm per head: 24 us against 65 for the kernel above, which
// keeps the other sizes.)
template <typename T>
__device__ __forceinline__ void qks_put(T* __restrict__ p, const float* v) {
  if constexpr (sizeof(T) == 2) *reinterpret_cast<uint2*>(p) = make_uint2(pack2<T>(v[0], v[1]), pack2<T>(v[2], v[3]));
  else *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
constexpr int QKS_WARPS = 8;

template <typename T, bool ONE>
__global__ void __launch_bounds__(QKS_WARPS * 32) qk_norm_rope_store_vec_kernel(
    const float* __restrict__ qkv, int n_partials, long long partial_stride,
    const float* __restrict__ bias, const float* __restrict__ q_norm, const float* __restrict__ k_norm, float n_q, float n_k, float eps,
    const float* __restrict__ freq, int dims, int neighbours, float mult, float head_eps, float head_size,
    const int* __restrict__ token_seq, const int* __restrict__ q_start,
    const int* __restrict__ seq_slot, const int* __restrict__ slot_pos, T* __restrict__ q_out,
    T* __restrict__ kv_step, T* __restrict__ k_cache, T* __restrict__ v_cache, int H, int G, int hd,
    int has_v, int capacity, int write_cache, const int* __restrict__ page_table, int pps, int n_pages) {
  pdl_launch_dependents();
  extern __shared__ __align__(16) float row_s[];         // the summed row, then dims / 2 (cos, sin) pairs
  __shared__ float2 warp_ss[QKS_WARPS];
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = token_seq[t];
  const int slot = seq_slot[b];
  const int qs = q_start[b], q_end = q_start[b + 1];
  const int past = slot_pos[slot];
  const int pos = past + (t - qs);
  const bool keep = write_cache && pos >= past + (q_end - qs) - capacity;
  const int cache_row = pos % capacity;
  const int units = H + (has_v ? 2 : 1) * G, row = units * hd, half = dims >> 1;
  float2* cs = reinterpret_cast<float2*>(row_s + row);
  const bool norms = q_norm != nullptr || k_norm != nullptr;
  // this block's heads (all of the row's are read where whole-row norms are formed)
  const int per_part = (units + gridDim.y - 1) / gridDim.y;
  const int u_lo = blockIdx.y * per_part, u_hi = min(units, u_lo + per_part);
  const int r_lo = norms ? 0 : u_lo, r_hi = norms ? units : u_hi;
  pdl_wait();
  const float* src = qkv + (size_t)t * row;
  float ssq = 0.f, ssk = 0.f;
#pragma unroll 4
  for (int u = r_lo + warp; u < r_hi; u += QKS_WARPS) {
    float ss = 0.f;
    for (int e = lane * 4; e < hd; e += 128) {
      const int i = u * hd + e;
      float4 v;
      if constexpr (ONE) {
        v = *reinterpret_cast<const float4*>(src + i);
      } else {
        v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < n_partials; s0 += 4) {
          float4 x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            x[j] = s0 + j < n_partials ? *reinterpret_cast<const float4*>(src + (size_t)(s0 + j) * partial_stride + i)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 4; ++j) { v.x += x[j].x; v.y += x[j].y; v.z += x[j].z; v.w += x[j].w; }
        }
      }
      if (bias != nullptr) {
        const float4 w = *reinterpret_cast<const float4*>(bias + i);
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
      }
      *reinterpret_cast<float4*>(row_s + i) = v;
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    if (u < H) ssq += ss;
    else if (u < H + G) ssk += ss;
  }
  for (int i = threadIdx.x; i < half; i += QKS_WARPS * 32) {
    const float ang = (float)pos * freq[i];
    cs[i] = make_float2(cosf(ang) * mult, sinf(ang) * mult);
  }
  float rq = 1.f, rk = 1.f;
  if (norms) {
    ssq = warp_sum(ssq);
    ssk = warp_sum(ssk);
    if (lane == 0) warp_ss[warp] = make_float2(ssq, ssk);
  }
  __syncthreads();
  if (norms) {
    ssq = ssk = 0.f;
#pragma unroll
    for (int i = 0; i < QKS_WARPS; ++i) { ssq += warp_ss[i].x; ssk += warp_ss[i].y; }
    if (q_norm != nullptr) rq = 1.0f / sqrtf(ssq / n_q + eps);
    if (k_norm != nullptr) rk = 1.0f / sqrtf(ssk / n_k + eps);
  }
  for (int u = u_lo + warp; u < u_hi; u += QKS_WARPS) {
    const bool is_q = u < H, is_v = u >= H + G;
    const int head = is_q ? u : is_v ? u - H - G : u - H;
    const float* x = row_s + u * hd;
    const float* w = is_v ? nullptr : is_q ? q_norm : k_norm;
    if (w != nullptr) w += head * hd;
    const float r = is_q ? rq : rk;
    T* out = is_q ? q_out + ((size_t)t * H + head) * hd : kv_step + ((size_t)t * 2 * G + (is_v ? G : 0) + head) * hd;
    const size_t cached = !is_q && keep ? kv_row_offset(page_table, pps, n_pages, slot, head, G, capacity, cache_row, hd) : 0;
    if (is_v || (!is_q && !has_v)) {                       // values: the v rows, or the keys as they were projected
      T* vo = kv_step + ((size_t)t * 2 * G + G + head) * hd;
      for (int e = lane * 4; e < hd; e += 128) {
        const float4 v = *reinterpret_cast<const float4*>(x + e);
        const float y[4] = {v.x, v.y, v.z, v.w};
        qks_put(vo + e, y);
        if (keep) qks_put(v_cache + cached + e, y);
      }
      if (is_v) continue;
    }
    // a lane's items: four features and, where halves turn, their partners `half` further on
    const int pairs = neighbours ? 0 : half / 4, items = neighbours ? hd / 4 : pairs + (hd - dims) / 4;
    auto load = [&](int i, float* y) {
      const float4 v = *reinterpret_cast<const float4*>(x + i);
      y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
      if (w != nullptr) {
        const float4 g = *reinterpret_cast<const float4*>(w + i);
        y[0] *= r * g.x; y[1] *= r * g.y; y[2] *= r * g.z; y[3] *= r * g.w;
      }
    };
    auto turned = [&](int it, int& i0, float* y, float* z) {
      if (neighbours) {
        i0 = it * 4;
        load(i0, y);
        if (i0 < dims) {
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const float2 c = cs[(i0 + j) >> 1];
            const float lo = rotate_lo(y[j], y[j + 1], c.x, c.y);
            y[j + 1] = rotate_hi(y[j], y[j + 1], c.x, c.y);
            y[j] = lo;
          }
        }
      } else if (it < pairs) {
        i0 = it * 4;
        load(i0, y);
        load(half + i0, z);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 c = cs[i0 + j];
          const float lo = rotate_lo(y[j], z[j], c.x, c.y);
          z[j] = rotate_hi(y[j], z[j], c.x, c.y);
          y[j] = lo;
        }
      } else {
        i0 = dims + (it - pairs) * 4;
        load(i0, y);
      }
    };
    float scale = 1.f;
    if (head_eps >= 0.f) {
      float ss = 0.f;
      for (int it = lane; it < items; it += 32) {
        int i0;
        float y[4], z[4] = {0.f, 0.f, 0.f, 0.f};
        turned(it, i0, y, z);
#pragma unroll
        for (int j = 0; j < 4; ++j) ss += y[j] * y[j] + z[j] * z[j];
      }
      scale = 1.0f / sqrtf(warp_sum(ss) / head_size + head_eps);
    }
    for (int it = lane; it < items; it += 32) {
      int i0;
      float y[4], z[4];
      turned(it, i0, y, z);
      if (head_eps >= 0.f) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { y[j] *= scale; z[j] *= scale; }
      }
      qks_put(out + i0, y);
      if (!is_q && keep) qks_put(k_cache + cached + i0, y);
      if (it < pairs) {
        qks_put(out + half + i0, z);
        if (!is_q && keep) qks_put(k_cache + cached + half + i0, z);
      }
    }
  }
}

// grid (blocks a sequence may complete in this step, G, sequences); one thread per feature, or (VEC) eight
// features per thread and the block's positions dealt out among POOL_GROUPS threads, whose sums are added in
// shared memory (32 blocks of 64 positions of 4 heads of 128: 21 us with a thread walking 64 rows, 4 so).
// Block number blk of a sequence (positions blk * pool .. blk * pool + pool - 1) is complete
// after this step if its last position is one of the step's.  A position of this step is read
// from kv_step, an earlier one from the ring (the ring holds at least the last pool - 1
// positions before the step; the step's late ring write, if any, has not happened yet).
constexpr int POOL_GROUPS = 8;
template <typename T, bool VEC>
__global__ void pool_blocks_kernel(const T* __restrict__ kv_step, const T* __restrict__ k_cache,
                                   const T* __restrict__ v_cache, const int* __restrict__ q_start,
                                   const int* __restrict__ seq_slot, const int* __restrict__ slot_pos,
                                   T* __restrict__ pool_k, T* __restrict__ pool_v, int G, int hd,
                                   int capacity, int pool, const int* __restrict__ page_table, int pps,
                                   int n_pages, int pool_capacity, const int* __restrict__ pool_table,
                                   int pool_pps, int pool_pages, int* __restrict__ status) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.z, g = blockIdx.y;
  const int slot = seq_slot[b];
  const int qs = q_start[b], ql = q_start[b + 1] - qs;
  const int past = slot_pos[slot];
  const int blk = past / pool + blockIdx.x;
  if ((blk + 1) * pool > past + ql) return;               // not complete yet
  if (blk >= pool_capacity) {
    if (threadIdx.x == 0) atomicOr(status, ERR_CONTEXT_RANGE);
    return;
  }
  const size_t out = kv_row_offset(pool_table, pool_pps, pool_pages, slot, g, G, pool_capacity, blk, hd);
  const float inv = 1.0f / (float)pool;
  if constexpr (VEC) {
    extern __shared__ __align__(16) float pool_s[];       // [POOL_GROUPS][2][hd]
    const int n8 = hd / 8, e = (threadIdx.x % n8) * 8, grp = threadIdx.x / n8;
    float sk[8] = {0.f}, sv[8] = {0.f};
    auto add = [](uint4 u, float* acc) {
      const T* x = reinterpret_cast<const T*>(&u);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += to_float(x[i]);
    };
    for (int j0 = grp; j0 < pool; j0 += 4 * POOL_GROUPS) {
      uint4 k[4], v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {                        // four rows of each in flight
        const int j = j0 + q * POOL_GROUPS, pos = blk * pool + j;
        k[q] = v[q] = make_uint4(0u, 0u, 0u, 0u);          // (zeros of either type)
        if (j >= pool) continue;
        const T *kp, *vp;
        if (pos >= past) {
          kp = kv_step + ((size_t)(qs + pos - past) * 2 * G + g) * hd;
          vp = kp + (size_t)G * hd;
        } else {
          const size_t off = kv_row_offset(page_table, pps, n_pages, slot, g, G, capacity, pos % capacity, hd);
          kp = k_cache + off;
          vp = v_cache + off;
        }
        k[q] = *reinterpret_cast<const uint4*>(kp + e);
        v[q] = *reinterpret_cast<const uint4*>(vp + e);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) { add(k[q], sk); add(v[q], sv); }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      pool_s[(grp * 2) * hd + e + i] = sk[i];
      pool_s[(grp * 2 + 1) * hd + e + i] = sv[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * hd; i += blockDim.x) {
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < POOL_GROUPS; ++q) sum += pool_s[q * 2 * hd + i];
      if (i < hd) pool_k[out + i] = from_float<T>(sum * inv);
      else pool_v[out + i - hd] = from_float<T>(sum * inv);
    }
  } else {
  for (int e = threadIdx.x; e < hd; e += blockDim.x) {
    float sk = 0.f, sv = 0.f;
    for (int j = 0; j < pool; ++j) {
      const int pos = blk * pool + j;
      if (pos >= past) {
        const T* kp = kv_step + ((size_t)(qs + pos - past) * 2 * G + g) * hd + e;
        sk += to_float(kp[0]);
        sv += to_float(kp[(size_t)G * hd]);
      } else {
        const size_t off = kv_row_offset(page_table, pps, n_pages, slot, g, G, capacity, pos % capacity, hd) + e;
        sk += to_float(k_cache[off]);
        sv += to_float(v_cache[off]);
      }
    }
    pool_k[out + e] = from_float<T>(sk * inv);
    pool_v[out + e] = from_float<T>(sv * inv);
  }
  }
}

}  // namespace yalm

using namespace yalm;

extern "C" int yalm_qk_norm_rope_store(const float* qkv, int n_partials, long long partial_stride,
                                       const float* bias, const float* q_norm, const float* k_norm, int n_q, int n_k,
                                       float eps, const float* freq, int dims, int neighbours,
                                       float mult, float head_eps, int head_size, const int* token_seq, const int* q_start,
                                       const int* seq_slot, const int* slot_pos, void* q_out,
                                       void* kv_step, void* k_cache, void* v_cache, int dtype,
                                       int n_tokens, int H, int G, int hd, int has_v, int capacity,
                                       int write_cache, const int* page_table, int pages_per_slot,
                                       int n_pages, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (hd <= 0 || dims < 0 || dims > hd || (dims & 1) || H <= 0 || G <= 0 || n_q <= 0 || n_k <= 0) return -2;
  const int row = (H + (has_v ? 2 : 1) * G) * hd;
  const size_t smem = (size_t)(((row + 1) & ~1) + dims + H + G) * sizeof(float);
  if (smem > 200 * 1024) return -2;
  if (head_eps >= 0.f && (head_size <= 0 || head_size > hd || q_norm != nullptr || k_norm != nullptr)) return -3;
  const int threads = row >= 2048 ? 512 : (row >= 512 ? 256 : 128);
  // a few tokens (a decode step): several blocks per token, each with a part of the outputs
  int parts = 1;
  if (n_tokens < 74) {
    parts = 148 / n_tokens;
    if (parts > 8) parts = 8;
    if (parts > row / 256) parts = row / 256 > 0 ? row / 256 : 1;
  }
  const uintptr_t bases = (uintptr_t)qkv | (uintptr_t)bias | (uintptr_t)q_norm | (uintptr_t)k_norm | (uintptr_t)q_out |
                          (uintptr_t)kv_step | (uintptr_t)k_cache | (uintptr_t)v_cache;
  // (a launch without the attribute below has 48 KB of shared memory for the kernel's own variables too)
  const bool vec = hd % 4 == 0 && dims % (neighbours ? 4 : 8) == 0 && (partial_stride & 3) == 0 && (bases & 15) == 0 &&
                   (size_t)(row + dims) * sizeof(float) <= 48 * 1024 - QKS_WARPS * sizeof(float2);
#define YALM_QKS(T)                                                                                   \
  do {                                                                                                \
    if (vec) {                                                                                        \
      launch_pdl(n_partials == 1 ? qk_norm_rope_store_vec_kernel<T, true> : qk_norm_rope_store_vec_kernel<T, false>, \
                 dim3(n_tokens, parts), dim3(QKS_WARPS * 32), (row + dims) * sizeof(float), stream, qkv, n_partials, \
                 partial_stride, bias, q_norm, k_norm, (float)n_q, (float)n_k, eps, freq, dims, neighbours, mult, \
                 head_eps, (float)head_size, token_seq, q_start, seq_slot, slot_pos, (T*)q_out, (T*)kv_step, \
                 (T*)k_cache, (T*)v_cache, H, G, hd, has_v, capacity, write_cache, page_table, pages_per_slot, n_pages); \
      break;                                                                                          \
    }                                                                                                 \
    static size_t attr = 48 * 1024 - 33 * sizeof(float);                                              \
    if (smem > attr) {                                                                                \
      cudaError_t e = cudaFuncSetAttribute(qk_norm_rope_store_kernel<T>,                              \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
      if (e != cudaSuccess) return (int)e;                                                            \
      attr = smem;                                                                                    \
    }                                                                                                 \
    launch_pdl(qk_norm_rope_store_kernel<T>, dim3(n_tokens, parts), dim3(threads), smem, stream, qkv, \
               n_partials, partial_stride, bias, q_norm, k_norm, (float)n_q, (float)n_k, eps, freq, dims,   \
               neighbours, mult, head_eps, (float)head_size, token_seq, q_start, seq_slot, slot_pos, (T*)q_out, (T*)kv_step,      \
               (T*)k_cache, (T*)v_cache, H, G, hd, has_v, capacity, write_cache, page_table,          \
               pages_per_slot, n_pages);                                                              \
  } while (0)
  if (dtype == DT_F32) YALM_QKS(float);
  else if (dtype == DT_BF16) YALM_QKS(__nv_bfloat16);
  else if (dtype == DT_F16) YALM_QKS(__half);
  else return -3;
#undef YALM_QKS
  YALM_LAUNCH_CHECK();
  return 0;
}

extern "C" int yalm_pool_blocks(const void* kv_step, const void* k_cache, const void* v_cache,
                                const int* q_start, const int* seq_slot, const int* slot_pos,
                                void* pool_k, void* pool_v, int dtype, int n_seqs, int max_q_len, int G,
                                int hd, int capacity, int pool, const int* page_table,
                                int pages_per_slot, int n_pages, int pool_capacity,
                                const int* pool_table, int pool_pps, int pool_pages, int* status,
                                cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (pool <= 0 || hd <= 0 || G <= 0 || capacity < pool - 1 || n_seqs > 65535 || G > 65535) return -2;
  const dim3 grid(max_q_len / pool + 1, G, n_seqs), block(hd >= 128 ? 128 : (hd >= 64 ? 64 : 32));
  const bool vec = dtype != DT_F32 && hd % 8 == 0 && hd <= 256 &&
                   ((((uintptr_t)kv_step) | ((uintptr_t)k_cache) | ((uintptr_t)v_cache)) & 15) == 0;
  const dim3 vblock(hd / 8 * POOL_GROUPS);
  const size_t vsmem = (size_t)POOL_GROUPS * 2 * hd * sizeof(float);
#define YALM_POOL_ARGS(T)                                                                            \
  stream, (const T*)kv_step, (const T*)k_cache, (const T*)v_cache, q_start, seq_slot, slot_pos, (T*)pool_k, (T*)pool_v, \
      G, hd, capacity, pool, page_table, pages_per_slot, n_pages, pool_capacity, pool_table, pool_pps, pool_pages, status
#define YALM_POOL(T)                                                                                 \
  do {                                                                                               \
    if (vec) launch_pdl(pool_blocks_kernel<T, sizeof(T) == 2>, grid, vblock, vsmem, YALM_POOL_ARGS(T)); \
    else launch_pdl(pool_blocks_kernel<T, false>, grid, block, 0, YALM_POOL_ARGS(T));                \
  } while (0)
  if (dtype == DT_F32) YALM_POOL(float);
  else if (dtype == DT_BF16) YALM_POOL(__nv_bfloat16);
  else if (dtype == DT_F16) YALM_POOL(__half);
  else return -3;
#undef YALM_POOL
#undef YALM_POOL_ARGS
  YALM_LAUNCH_CHECK();
  return 0;
}
