// The gated delta rule with a decay per key channel, per head with key size dk and value size dv:
//   S <- diag(g_t) S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
// S [dk, dv] per head and sequence in 32-bit floats, carried from step to step.  Query/key heads may
// be fewer than value heads: head h reads q/k head h / (H / G).  Everything here is 32-bit.
//
//  * delta_prep: q and k of every token and q/k head become unit vectors (x / sqrt(sum x^2 + 1e-6)),
//    q times 1/sqrt(dk); beta = sigmoid(.); and the two low-rank projections' first halves go out in
//    the storage type as the input of their second halves;
//  * delta_decay: the decay per head and key channel, kept as g - 1 = expm1(-exp(A_h) softplus(z + dt))
//    (a decay close to 1 has few bits of its own left in g; S + (g - 1) S keeps them), and the output
//    gate sigmoid(.) per head and value channel;
//  * delta_scan: the recurrence.  As in the other scans of this library a block owns 16 value
//    columns of one (sequence, head) -- the columns of S are independent of one another -- and the
//    step's tokens come through a three-stage cp.async ring.  Unlike a plain linear recurrence the write
//    needs k.S first, so every token costs one all-reduce before its update; the outputs' sums are
//    formed for 16 tokens at once.  Key sizes up to 128 run with eight lanes per two columns
//    (delta_scan8_kernel), larger ones with a warp per two columns (delta_scan_kernel);
//  * delta_step: a step of one token per sequence, key sizes up to 128: the state streamed once.
//
// The activated row of a token, float32: [q: G dk | k: G dk | v: H dv | beta: H padded to 4 | g - 1: H dk].
#include "api.h"
#include "common.cuh"
#include "scan.cuh"

namespace yalm {

constexpr int DR_CPW = 2;
constexpr int DR_COLS = 8 * DR_CPW;
constexpr int DR_TOK = 16;
constexpr int DR_STAGES = 3;

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// grid (tokens); a warp per q/k head for the unit vectors, then the block's threads for the rest.
// proj: slices [.][tokens][proj_row] with beta at col_b (H), the low-rank inputs at col_low (n_low)
template <typename T>
__global__ void delta_prep_kernel(float* __restrict__ act, int row, const float* __restrict__ proj,
                                  int n_partials, long long partial_stride, int proj_row, int col_b,
                                  int col_low, int n_low, T* __restrict__ low, int H, int G, int dk, int dv) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  float* a = act + (size_t)t * row;
  const float q_scale = 1.0f / sqrtf((float)dk);
  for (int head = warp; head < 2 * G; head += n_warps) {
    float* v = a + (size_t)head * dk;                       // q heads, then k heads
    float ss = 0.f;
    for (int i = lane; i < dk; i += 32) ss += v[i] * v[i];
    ss = warp_sum(ss);
    const float r = (1.0f / sqrtf(ss + 1e-6f)) * (head < G ? q_scale : 1.0f);
    for (int i = lane; i < dk; i += 32) v[i] *= r;
  }
  const float* p = proj + (size_t)t * proj_row;
  const int beta0 = 2 * G * dk + H * dv;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float z = sum_slices(p + col_b + i, n_partials, partial_stride);
    a[beta0 + i] = 1.0f / (1.0f + expf(-z));
  }
  for (int i = threadIdx.x; i < n_low; i += blockDim.x)
    low[(size_t)t * n_low + i] = from_float<T>(sum_slices(p + col_low + i, n_partials, partial_stride));
}

// grid (tokens, parts); z: slices [.][tokens][H dk + H dv] = (decay logits | gate logits)
__global__ void delta_decay_kernel(float* __restrict__ act, int row, int decay0, const float* __restrict__ z,
                                   int n_partials, long long partial_stride, const float* __restrict__ dt_bias,
                                   const float* __restrict__ a_log, float* __restrict__ gate, int H, int dk,
                                   int dv) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int n_k = H * dk, n_v = H * dv;
  const float* zr = z + (size_t)t * (n_k + n_v);
  const int e_end = min(n_k + n_v, (int)(blockIdx.y + 1) * 1024);
  for (int e = blockIdx.y * 1024 + threadIdx.x; e < e_end; e += blockDim.x) {
    const float v = n_partials == 1 ? zr[e] : sum_slices(zr + e, n_partials, partial_stride);
    if (e < n_k) act[(size_t)t * row + decay0 + e] = expm1f(-expf(a_log[e / dk]) * softplus_f(v + dt_bias[e]));
    else gate[(size_t)t * n_v + (e - n_k)] = 1.0f / (1.0f + expf(-v));
  }
}

template <int BYTES>
__device__ __forceinline__ void dr_cp_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void dr_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void dr_cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A lane's RPT neighbouring rows of a staged vector, as one 8- or 16-byte access per two or four rows:
// single-float loads at a stride of RPT floats would meet RPT-fold bank conflicts.
template <int RPT>
__device__ __forceinline__ void lane_rows(const float* __restrict__ p, float* out) {
  if constexpr (RPT % 4 == 0) {
#pragma unroll
    for (int r = 0; r < RPT; r += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + r);
      out[r] = v.x; out[r + 1] = v.y; out[r + 2] = v.z; out[r + 3] = v.w;
    }
  } else if constexpr (RPT == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    out[0] = v.x; out[1] = v.y;
  } else {
#pragma unroll
    for (int r = 0; r < RPT; ++r) out[r] = p[r];
  }
}

// VEC: floats per copy (4 when every run starts on a 16-byte boundary, else 1)
template <int RPT, int VEC>
__global__ void __launch_bounds__(256)
delta_scan_kernel(const float* __restrict__ act, int row, const int* __restrict__ q_start,
                  const int* __restrict__ seq_slot, float* __restrict__ state, float* __restrict__ out,
                  int H, int G, int dk, int dv) {
  pdl_launch_dependents();
  constexpr int DKP = 32 * RPT;                       // rows, padded
  constexpr int PER_TOK = 3 * DKP + DR_COLS + 4;      // q, k, g, this block's v columns, beta (+ padding)
  extern __shared__ __align__(16) float stage[];      // [DR_STAGES][DR_TOK][PER_TOK]
  const int b = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * DR_COLS;
  const int hq = h / (H / G);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = c0 + w * DR_CPW;
  const int slot = seq_slot[b];
  const int t0 = q_start[b], t1 = q_start[b + 1];
  const int hp = (H + 3) & ~3;
  // rows beyond dk: q = k = 0 for ever (never copied over), so their state stays zero
  if (dk < DKP) {
    for (int i = threadIdx.x; i < DR_STAGES * DR_TOK * PER_TOK; i += blockDim.x) stage[i] = 0.f;
    __syncthreads();
  }
  // what this thread copies of every token: up to four runs of VEC floats, and thread 0 the beta
  const int per = 3 * dk + DR_COLS;
  int src_off[4], dst_off[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int e = (threadIdx.x + k * 256) * VEC;
    src_off[k] = dst_off[k] = -1;
    if (e < dk) { src_off[k] = hq * dk + e; dst_off[k] = e; }
    else if (e < 2 * dk) { src_off[k] = G * dk + hq * dk + (e - dk); dst_off[k] = DKP + (e - dk); }
    else if (e < 3 * dk) { src_off[k] = 2 * G * dk + H * dv + hp + h * dk + (e - 2 * dk); dst_off[k] = 2 * DKP + (e - 2 * dk); }
    else if (e < per && c0 + (e - 3 * dk) < dv) {
      src_off[k] = 2 * G * dk + h * dv + c0 + (e - 3 * dk);
      dst_off[k] = 3 * DKP + (e - 3 * dk);
    }
  }
  const int beta_off = 2 * G * dk + H * dv + h;
  pdl_wait();
  float S[RPT][DR_CPW];
  float* st = state + (((size_t)slot * H + h) * dk) * dv + col;
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < DR_CPW; ++c) {
      const int i = lane * RPT + r;
      S[r][c] = (col + c < dv && i < dk) ? st[(size_t)i * dv + c] : 0.f;
    }
  const int n_groups = (t1 - t0 + DR_TOK - 1) / DR_TOK;
  auto issue = [&](int g) {
    if (g < n_groups) {
      const int base = t0 + g * DR_TOK;
      const int nt = min(DR_TOK, t1 - base);
      float* dst = stage + (size_t)(g % DR_STAGES) * DR_TOK * PER_TOK;
      const float* src = act + (size_t)base * row;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (src_off[k] >= 0)
          for (int tt = 0; tt < nt; ++tt)
            dr_cp_async<4 * VEC>(dst + tt * PER_TOK + dst_off[k], src + (size_t)tt * row + src_off[k]);
      if (threadIdx.x < nt)
        dr_cp_async<4>(dst + threadIdx.x * PER_TOK + 3 * DKP + DR_COLS, src + (size_t)threadIdx.x * row + beta_off);
    }
    dr_cp_commit();
  };
  issue(0);
  issue(1);
  for (int g = 0; g < n_groups; ++g) {
    dr_cp_wait<DR_STAGES - 2>();
    __syncthreads();                                   // stage g has landed; stage g - 1 is no longer read
    issue(g + 2);
    const int base = t0 + g * DR_TOK;
    const int nt = min(DR_TOK, t1 - base);
    const float* sg = stage + (size_t)(g % DR_STAGES) * DR_TOK * PER_TOK;
    float o[DR_TOK][DR_CPW];
    auto token = [&](int tt) {
      const float* qq = sg + tt * PER_TOK + lane * RPT;
      const float* kk = qq + DKP;
      const float* gg = qq + 2 * DKP;
      const float beta = sg[tt * PER_TOK + 3 * DKP + DR_COLS];
      float vj[DR_CPW], kd[DR_CPW], kr[RPT], qr[RPT], gr[RPT];
      lane_rows<RPT>(qq, qr);
      lane_rows<RPT>(kk, kr);
      lane_rows<RPT>(gg, gr);
#pragma unroll
      for (int c = 0; c < DR_CPW; ++c) { vj[c] = sg[tt * PER_TOK + 3 * DKP + w * DR_CPW + c]; kd[c] = 0.f; }
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const float gi = gr[r];
#pragma unroll
        for (int c = 0; c < DR_CPW; ++c) {
          S[r][c] = fmaf(gi, S[r][c], S[r][c]);
          kd[c] = fmaf(kr[r], S[r][c], kd[c]);
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < DR_CPW; ++c) kd[c] += __shfl_xor_sync(0xffffffffu, kd[c], off);
      float u[DR_CPW];
#pragma unroll
      for (int c = 0; c < DR_CPW; ++c) u[c] = beta * (vj[c] - kd[c]);
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < DR_CPW; ++c) {
          S[r][c] = fmaf(kr[r], u[c], S[r][c]);
          o[tt][c] = fmaf(S[r][c], qr[r], o[tt][c]);
        }
    };
#pragma unroll
    for (int tt = 0; tt < DR_TOK; ++tt)
#pragma unroll
      for (int c = 0; c < DR_CPW; ++c) o[tt][c] = 0.f;
    if (nt == DR_TOK) {                                // a full group: no test between the tokens, so that a
#pragma unroll                                         // token's rows are loaded while the one before is reduced
      for (int tt = 0; tt < DR_TOK; ++tt) token(tt);
    } else {
#pragma unroll
      for (int tt = 0; tt < DR_TOK; ++tt)
        if (tt < nt) token(tt);
    }
    // the 32 lanes' partial sums of the group's 32 outputs: in every round a lane hands half of its
    // values to its partner and adds the partner's other half to its own
    static_assert(DR_TOK * DR_CPW == 32, "one output per lane");
    float* ov = &o[0][0];
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
      const bool upper = (lane & half) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float send = upper ? ov[i] : ov[i + half];
        const float keep = upper ? ov[i + half] : ov[i];
        ov[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
      }
    }
    {
      const int tt = lane / DR_CPW, c = lane % DR_CPW;
      if (tt < nt && col + c < dv) out[((size_t)(base + tt) * H + h) * dv + col + c] = ov[0];
    }
  }
  dr_cp_wait<0>();
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int c = 0; c < DR_CPW; ++c) {
      const int i = lane * RPT + r;
      if (col + c < dv && i < dk) st[(size_t)i * dv + c] = S[r][c];
    }
}

// The same recurrence with EIGHT lanes per two value columns (key sizes up to 128): a warp owns eight columns, a
// lane RPL = 4, 8 or 16 rows of two of them, two rows per packed instruction.  The all-reduce of k.S that every
// token's write waits for takes three exchange rounds, and a token's k, q and decay, which every lane group
// reads for itself, are read once for two columns: with one column per group these reads (24 KB per token of
// a block, at 128 bytes a clock) were half of a token's time.  A block of two warps owns 16 columns, so the grid
// is that of the kernel above.  (16 heads of 128 x 128, three prompts of 2,150 tokens in all: 323 us with one
// column per group, 279 so.)
constexpr int D8_WARPS = 2;
constexpr int D8_COLS = 8 * D8_WARPS;

// a run of floats of nt <= DR_TOK tokens: a whole stage's copies go out without a test between them
template <int BYTES>
__device__ __forceinline__ void dr_copy_tokens(float* dst, int dst_pitch, const float* src, int src_pitch, int nt) {
  if (nt == DR_TOK) {
#pragma unroll
    for (int tt = 0; tt < DR_TOK; ++tt) dr_cp_async<BYTES>(dst + tt * dst_pitch, src + (size_t)tt * src_pitch);
  } else {
    for (int tt = 0; tt < nt; ++tt) dr_cp_async<BYTES>(dst + tt * dst_pitch, src + (size_t)tt * src_pitch);
  }
}

template <int RPL, int VEC>
__global__ void __launch_bounds__(32 * D8_WARPS)
delta_scan8_kernel(const float* __restrict__ act, int row, const int* __restrict__ q_start,
                   const int* __restrict__ seq_slot, float* __restrict__ state, float* __restrict__ out,
                   int H, int G, int dk, int dv) {
  pdl_launch_dependents();
  constexpr int DKP = 8 * RPL;                        // rows, padded
  constexpr int PER_TOK = 3 * DKP + D8_COLS + 4;      // q, k, g - 1, this block's v columns, beta (+ padding)
  constexpr int NT = 32 * D8_WARPS;
  constexpr int KC = (3 * DKP + D8_COLS + NT * VEC - 1) / (NT * VEC);   // runs of VEC floats a thread copies per token
  extern __shared__ __align__(16) float stage[];      // [DR_STAGES][DR_TOK][PER_TOK]
  const int b = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * D8_COLS;
  const int hq = h / (H / G);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int cg = lane >> 3, sub = lane & 7;
  const int col = c0 + w * 8 + cg * 2;                // this lane's columns: col, col + 1
  const int slot = seq_slot[b];
  const int t0 = q_start[b], t1 = q_start[b + 1];
  const int hp = (H + 3) & ~3;
  if (dk < DKP) {                                     // rows beyond dk: q = k = 0 for ever, their state stays zero
    for (int i = threadIdx.x; i < DR_STAGES * DR_TOK * PER_TOK; i += NT) stage[i] = 0.f;
    __syncthreads();
  }
  const int per = 3 * dk + D8_COLS;
  int src_off[KC], dst_off[KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    const int e = (threadIdx.x + k * NT) * VEC;
    src_off[k] = dst_off[k] = -1;
    if (e < dk) { src_off[k] = hq * dk + e; dst_off[k] = e; }
    else if (e < 2 * dk) { src_off[k] = G * dk + hq * dk + (e - dk); dst_off[k] = DKP + (e - dk); }
    else if (e < 3 * dk) { src_off[k] = 2 * G * dk + H * dv + hp + h * dk + (e - 2 * dk); dst_off[k] = 2 * DKP + (e - 2 * dk); }
    else if (e < per && c0 + (e - 3 * dk) < dv) {
      src_off[k] = 2 * G * dk + h * dv + c0 + (e - 3 * dk);
      dst_off[k] = 3 * DKP + (e - 3 * dk);
    }
  }
  const int beta_off = 2 * G * dk + H * dv + h;
  pdl_wait();
  f2 S[RPL / 2][2];                                   // pair r: rows 4 (sub + 8 (r / 2)) + 2 (r % 2) and the next; per column
  float* st = state + (((size_t)slot * H + h) * dk) * dv + col;
#pragma unroll
  for (int r = 0; r < RPL / 2; ++r) {
    const int i = 4 * (sub + 8 * (r >> 1)) + 2 * (r & 1);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float lo = (col + c < dv && i < dk) ? st[(size_t)i * dv + c] : 0.f;
      const float hi = (col + c < dv && i + 1 < dk) ? st[(size_t)(i + 1) * dv + c] : 0.f;
      S[r][c] = pack_f2(lo, hi);
    }
  }
  const int n_groups = (t1 - t0 + DR_TOK - 1) / DR_TOK;
  auto issue = [&](int g) {
    if (g < n_groups) {
      const int base = t0 + g * DR_TOK;
      const int nt = min(DR_TOK, t1 - base);
      float* dst = stage + (size_t)(g % DR_STAGES) * DR_TOK * PER_TOK;
      const float* src = act + (size_t)base * row;
#pragma unroll
      for (int k = 0; k < KC; ++k)
        if (src_off[k] >= 0) dr_copy_tokens<4 * VEC>(dst + dst_off[k], PER_TOK, src + src_off[k], row, nt);
      if (threadIdx.x < nt)
        dr_cp_async<4>(dst + threadIdx.x * PER_TOK + 3 * DKP + D8_COLS, src + (size_t)threadIdx.x * row + beta_off);
    }
    dr_cp_commit();
  };
  issue(0);
  issue(1);
  for (int g = 0; g < n_groups; ++g) {
    dr_cp_wait<DR_STAGES - 2>();
    __syncthreads();                                   // stage g has landed; stage g - 1 is no longer read
    issue(g + 2);
    const int base = t0 + g * DR_TOK;
    const int nt = min(DR_TOK, t1 - base);
    const float* sg = stage + (size_t)(g % DR_STAGES) * DR_TOK * PER_TOK;
    float o[DR_TOK][2];
    auto token = [&](int tt) {
      // a lane's rows are every eighth group of four: the eight lanes of a group then read 128
      // neighbouring bytes at a time (RPL rows in a row per lane would meet four-fold bank conflicts)
      const float* qq = sg + tt * PER_TOK + 4 * sub;
      f2 qr[RPL / 2], kr[RPL / 2], gr[RPL / 2];
#pragma unroll
      for (int j = 0; j < RPL / 4; ++j) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(qq + 32 * j);
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(qq + DKP + 32 * j);
        const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(qq + 2 * DKP + 32 * j);
        qr[2 * j] = x.x; qr[2 * j + 1] = x.y;
        kr[2 * j] = y.x; kr[2 * j + 1] = y.y;
        gr[2 * j] = z.x; gr[2 * j + 1] = z.y;
      }
      const float beta = sg[tt * PER_TOK + 3 * DKP + D8_COLS];
      const float2 v = *reinterpret_cast<const float2*>(sg + tt * PER_TOK + 3 * DKP + w * 8 + cg * 2);
      f2 kd[2][2];
#pragma unroll
      for (int r = 0; r < RPL / 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[r][c] = fma_f2(gr[r], S[r][c], S[r][c]);
          kd[c][r & 1] = r < 2 ? mul_f2(kr[r], S[r][c]) : fma_f2(kr[r], S[r][c], kd[c][r & 1]);
        }
      float d0 = sum_f2(kd[0][0], kd[0][1]), d1 = sum_f2(kd[1][0], kd[1][1]);
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) {
        d0 += __shfl_xor_sync(0xffffffffu, d0, off);
        d1 += __shfl_xor_sync(0xffffffffu, d1, off);
      }
      const float u0 = beta * (v.x - d0), u1 = beta * (v.y - d1);
      const f2 u[2] = {pack_f2(u0, u0), pack_f2(u1, u1)};
      f2 od[2][2];
#pragma unroll
      for (int r = 0; r < RPL / 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[r][c] = fma_f2(kr[r], u[c], S[r][c]);
          od[c][r & 1] = r < 2 ? mul_f2(S[r][c], qr[r]) : fma_f2(S[r][c], qr[r], od[c][r & 1]);
        }
      o[tt][0] = sum_f2(od[0][0], od[0][1]);
      o[tt][1] = sum_f2(od[1][0], od[1][1]);
    };
    if (nt == DR_TOK) {                                // a full group: no test between the tokens, so that a
#pragma unroll                                         // token's rows are loaded while the one before is reduced
      for (int tt = 0; tt < DR_TOK; ++tt) token(tt);
    } else {
#pragma unroll
      for (int tt = 0; tt < DR_TOK; ++tt) {
        o[tt][0] = o[tt][1] = 0.f;
        if (tt < nt) token(tt);
      }
    }
    // the eight lanes' partial sums of the two columns' 32 outputs, value number 2 tt + c: in every round a lane
    // hands half of its values to its partner and adds the partner's other half to its own; four whole sums
    // are left per lane, tokens 2 sub and 2 sub + 1
    static_assert(DR_TOK == 16, "four outputs per lane");
    float* ov = &o[0][0];
#pragma unroll
    for (int half = 4, n = 16; half >= 1; half >>= 1, n >>= 1) {
      const bool upper = (sub & half) != 0;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const float send = upper ? ov[i] : ov[i + n];
        const float keep = upper ? ov[i + n] : ov[i];
        ov[i] = keep + __shfl_xor_sync(0xffffffffu, send, half);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tt = 2 * sub + (i >> 1), c = i & 1;
      if (tt < nt && col + c < dv) out[((size_t)(base + tt) * H + h) * dv + col + c] = ov[i];
    }
  }
  dr_cp_wait<0>();
#pragma unroll
  for (int r = 0; r < RPL / 2; ++r) {
    const int i = 4 * (sub + 8 * (r >> 1)) + 2 * (r & 1);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float lo, hi;
      unpack_f2(S[r][c], lo, hi);
      if (col + c < dv && i < dk) st[(size_t)i * dv + c] = lo;
      if (col + c < dv && i + 1 < dk) st[(size_t)(i + 1) * dv + c] = hi;
    }
  }
}

// A step of one token per sequence: bound by the state's bytes, read and written once.  A block takes 4 CQ
// value columns of one (sequence, head) and holds their state in registers between the two passes that the
// write needs (k.S first): a thread four neighbouring columns of every (256 / CQ)-th row, ROWS of them, so
// that all its 16-byte loads are in flight at once.  (The scan's lanes read 4 or 8 bytes of a row each.  64
// sequences of 16 heads of 128 x 128, 134 MB of state in and out: a whole decode step of two Samulorn layers
// 417 us with the scan, 352 with this.)
template <int ROWS, int CQ>
__global__ void __launch_bounds__(256, ROWS == 16 ? 2 : ROWS == 8 ? 3 : 5)
delta_step_kernel(const float* __restrict__ act, int row, const int* __restrict__ q_start,
                  const int* __restrict__ seq_slot, float* __restrict__ state, float* __restrict__ out, int H, int G,
                  int dk, int dv) {
  pdl_launch_dependents();
  constexpr int RG = 256 / CQ;
  __shared__ float qs[RG * ROWS], ks[RG * ROWS], gs[RG * ROWS];
  __shared__ __align__(16) float part[RG][4 * CQ];
  __shared__ __align__(16) float u_s[4 * CQ];
  const int b = blockIdx.z, h = blockIdx.y, hq = h / (H / G), hp = (H + 3) & ~3;
  const int cq = threadIdx.x % CQ, rg = threadIdx.x / CQ;
  const int c0 = blockIdx.x * 4 * CQ, col = c0 + cq * 4;
  const int slot = seq_slot[b], t0 = q_start[b], t1 = q_start[b + 1];
  const bool on = col < dv;
  float* st = state + ((size_t)slot * H + h) * dk * dv + col;
  pdl_wait();
  float4 S[ROWS];
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    const int r = rg + j * RG;
    S[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on && r < dk) S[j] = *reinterpret_cast<const float4*>(st + (size_t)r * dv);
  }
  // one token; none or several where a caller's step has as many tokens as sequences but does not deal them out evenly
#pragma unroll 1
  for (int t = t0; t < t1; ++t) {
    const float* src = act + (size_t)t * row;
    for (int i = threadIdx.x; i < RG * ROWS; i += 256) {
      qs[i] = i < dk ? src[hq * dk + i] : 0.f;
      ks[i] = i < dk ? src[G * dk + hq * dk + i] : 0.f;
      gs[i] = i < dk ? src[2 * G * dk + H * dv + hp + h * dk + i] : 0.f;
    }
    __syncthreads();
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const float g = gs[rg + j * RG], k = ks[rg + j * RG];
      S[j].x = fmaf(g, S[j].x, S[j].x); S[j].y = fmaf(g, S[j].y, S[j].y);
      S[j].z = fmaf(g, S[j].z, S[j].z); S[j].w = fmaf(g, S[j].w, S[j].w);
      d.x = fmaf(k, S[j].x, d.x); d.y = fmaf(k, S[j].y, d.y);
      d.z = fmaf(k, S[j].z, d.z); d.w = fmaf(k, S[j].w, d.w);
    }
    *reinterpret_cast<float4*>(&part[rg][4 * cq]) = d;
    __syncthreads();
    if (threadIdx.x < 4 * CQ) {
      const int c = c0 + threadIdx.x;
      float sum = 0.f;
#pragma unroll
      for (int g = 0; g < RG; ++g) sum += part[g][threadIdx.x];
      u_s[threadIdx.x] = c < dv ? src[2 * G * dk + H * dv + h] * (src[2 * G * dk + h * dv + c] - sum) : 0.f;
    }
    __syncthreads();
    const float4 u = *reinterpret_cast<const float4*>(&u_s[4 * cq]);
    d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const int r = rg + j * RG;
      const float k = ks[r], q = qs[r];
      S[j].x = fmaf(k, u.x, S[j].x); S[j].y = fmaf(k, u.y, S[j].y);
      S[j].z = fmaf(k, u.z, S[j].z); S[j].w = fmaf(k, u.w, S[j].w);
      d.x = fmaf(S[j].x, q, d.x); d.y = fmaf(S[j].y, q, d.y);
      d.z = fmaf(S[j].z, q, d.z); d.w = fmaf(S[j].w, q, d.w);
      if (on && r < dk) *reinterpret_cast<float4*>(st + (size_t)r * dv) = S[j];
    }
    *reinterpret_cast<float4*>(&part[rg][4 * cq]) = d;
    __syncthreads();
    if (threadIdx.x < 4 * CQ) {
      const int c = c0 + threadIdx.x;
      float sum = 0.f;
#pragma unroll
      for (int g = 0; g < RG; ++g) sum += part[g][threadIdx.x];
      if (c < dv) out[((size_t)t * H + h) * dv + c] = sum;
    }
  }
}

}  // namespace yalm

using namespace yalm;

// The length of a token's activated row (see the head of this file)
extern "C" int yalm_delta_row(int H, int G, int dk, int dv) {
  return 2 * G * dk + H * dv + ((H + 3) & ~3) + H * dk;
}

// act: float32 [tokens][yalm_delta_row], whose first 2 G dk + H dv columns hold q | k | v after their
// convolution and activation.  proj: slices [.][tokens][proj_row] of the mixer's first product, with
// the beta logits at column col_b and the n_low low-rank values at col_low; low [tokens][n_low] in
// low_dtype receives those.
extern "C" int yalm_delta_prep(float* act, const float* proj, int n_partials, long long partial_stride,
                               int proj_row, int col_b, int col_low, int n_low, void* low, int low_dtype,
                               int n_tokens, int H, int G, int dk, int dv, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0 || n_low < 0) return -2;
  const int row = yalm_delta_row(H, G, dk, dv);
  const dim3 grid(n_tokens), block(256);
#define YALM_DP(T)                                                                                     \
  launch_pdl(delta_prep_kernel<T>, grid, block, 0, stream, act, row, proj, n_partials, partial_stride, \
             proj_row, col_b, col_low, n_low, (T*)low, H, G, dk, dv)
  if (low_dtype == DT_F32) YALM_DP(float);
  else if (low_dtype == DT_BF16) YALM_DP(__nv_bfloat16);
  else if (low_dtype == DT_F16) YALM_DP(__half);
  else return -3;
#undef YALM_DP
  YALM_LAUNCH_CHECK();
  return 0;
}

// z: slices [.][tokens][H dk + H dv] (decay logits | gate logits); dt_bias [H dk]; a_log [H];
// gate float32 [tokens][H dv] receives sigmoid(gate logits); then the scan: state float32
// [slots][H][dk][dv], out float32 [tokens][H dv].  dk up to 256.
extern "C" int yalm_delta_scan(float* act, const float* z, int n_partials, long long partial_stride,
                               const float* dt_bias, const float* a_log, float* gate, const int* q_start,
                               const int* seq_slot, float* state, float* out, int n_tokens, int n_seqs,
                               int H, int G, int dk, int dv, cudaStream_t stream) {
  if (n_tokens <= 0 || n_seqs <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0 || dk > 256 || n_seqs > 65535 || H > 65535) return -2;
  const int row = yalm_delta_row(H, G, dk, dv);
  const int decay0 = row - H * dk;
  const int parts = (H * dk + H * dv + 1023) / 1024;
  if (parts > 65535) return -4;
  launch_pdl(delta_decay_kernel, dim3(n_tokens, parts), dim3(256), 0, stream, act, row, decay0, z, n_partials,
             partial_stride, dt_bias, a_log, gate, H, dk, dv);
  YALM_LAUNCH_CHECK();
  const bool vec = dk % 4 == 0 && dv % 4 == 0 && (((uintptr_t)act) & 15) == 0;
  // one token per sequence, whole 16-byte accesses
  if (n_tokens == n_seqs && dk <= 128 && vec && (((uintptr_t)state) & 15) == 0) {
#define YALM_DSTEP(R, CQ)                                                                                    \
  launch_pdl(delta_step_kernel<R, CQ>, dim3((dv + 4 * CQ - 1) / (4 * CQ), H, n_seqs), dim3(256), 0, stream,  \
             (const float*)act, row, q_start, seq_slot, state, out, H, G, dk, dv)
    if (dv <= 64) {
      if (dk <= 64) YALM_DSTEP(4, 16);
      else YALM_DSTEP(8, 16);
    } else {
      if (dk <= 64) YALM_DSTEP(8, 32);
      else YALM_DSTEP(16, 32);
    }
#undef YALM_DSTEP
    YALM_LAUNCH_CHECK();
    return 0;
  }
  if (dk <= 128) {
    // eight lanes per two columns
    const dim3 grid8((dv + D8_COLS - 1) / D8_COLS, H, n_seqs), block8(32 * D8_WARPS);
#define YALM_D8(R)                                                                                   \
  do {                                                                                               \
    const size_t smem = (size_t)DR_STAGES * DR_TOK * (3 * 8 * R + D8_COLS + 4) * sizeof(float);      \
    static bool set = false;                                                                         \
    if (!set && smem > 48 * 1024) {                                                                  \
      cudaError_t e = cudaFuncSetAttribute(delta_scan8_kernel<R, 4>,                                 \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
      if (e == cudaSuccess)                                                                          \
        e = cudaFuncSetAttribute(delta_scan8_kernel<R, 1>,                                           \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);            \
      if (e != cudaSuccess) return (int)e;                                                           \
      set = true;                                                                                    \
    }                                                                                                \
    if (vec)                                                                                         \
      launch_pdl(delta_scan8_kernel<R, 4>, grid8, block8, smem, stream, (const float*)act, row,      \
                 q_start, seq_slot, state, out, H, G, dk, dv);                                       \
    else                                                                                             \
      launch_pdl(delta_scan8_kernel<R, 1>, grid8, block8, smem, stream, (const float*)act, row,      \
                 q_start, seq_slot, state, out, H, G, dk, dv);                                       \
  } while (0)
    if (dk <= 32) YALM_D8(4);
    else if (dk <= 64) YALM_D8(8);
    else YALM_D8(16);
#undef YALM_D8
    YALM_LAUNCH_CHECK();
    return 0;
  }
  const dim3 grid((dv + DR_COLS - 1) / DR_COLS, H, n_seqs), block(256);
  const int rpt = (dk + 31) / 32;
#define YALM_DS(R)                                                                                  \
  do {                                                                                              \
    const size_t smem = (size_t)DR_STAGES * DR_TOK * (3 * 32 * R + DR_COLS + 4) * sizeof(float);    \
    static bool set = false;                                                                        \
    if (!set && smem > 48 * 1024) {                                                                 \
      cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<R, 4>,                                 \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e == cudaSuccess)                                                                         \
        e = cudaFuncSetAttribute(delta_scan_kernel<R, 1>,                                           \
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);           \
      if (e != cudaSuccess) return (int)e;                                                          \
      set = true;                                                                                   \
    }                                                                                               \
    if (vec)                                                                                        \
      launch_pdl(delta_scan_kernel<R, 4>, grid, block, smem, stream, (const float*)act, row, q_start, \
                 seq_slot, state, out, H, G, dk, dv);                                               \
    else                                                                                            \
      launch_pdl(delta_scan_kernel<R, 1>, grid, block, smem, stream, (const float*)act, row, q_start, \
                 seq_slot, state, out, H, G, dk, dv);                                               \
  } while (0)
  if (rpt <= 1) YALM_DS(1);
  else if (rpt <= 2) YALM_DS(2);
  else if (rpt <= 4) YALM_DS(4);
  else YALM_DS(8);
#undef YALM_DS
  YALM_LAUNCH_CHECK();
  return 0;
}
