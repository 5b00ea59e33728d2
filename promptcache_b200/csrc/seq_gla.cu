// Gated linear attention over the slot pool.
//
// Per head, with a decay per key channel alpha_t = exp(ld_t) in (0, 1):
//     S_t = diag(alpha_t) S_{t-1} + k_t v_t^T          (S: dim x vdim; the decay scales the rows, which belong to key channels)
//     o_t = S_t^T q_t
// followed by o_t / rms(o_t) per head, one norm weight vector for all heads, and the gate silu(g_t).  S lives in 32-bit floats
// in the slot pool and is carried from step to step; a sequence whose slot holds no tokens yet starts from zero.  Decays,
// their logarithms and the state are 32-bit in both compute types; q, k, v and g come from the projections in the compute type.
//
// pcs_gla_decay  one block per token: z = A2 a + b per channel from the low-rank input a (32-bit sums), ld = logsigmoid(z) / tau.
// pcs_gla_scan   the token-by-token recurrence, one block per (sequence, head, slice of value columns): state in registers
//                (dim <= 256, 16-byte aligned projections) or in shared memory, then the per-head output norm with the gate.
#include "seq_common.cuh"
#include "seq_mma.cuh"

namespace pcs {

// From a channel's pre-activation z to its log decay: logsigmoid(z) / tau, or -rate * softplus(z) with one rate per rate_dim
// neighbouring channels; optionally the decay itself.
struct DecayForm {
  float inv_tau;
  const float* rate;
  int rate_dim, expo;
  __device__ __forceinline__ float operator()(float z, int c) const {
    const float l = rate ? -rate[c / rate_dim] * softplusf_(z) : logsigmoidf_(z) * inv_tau;
    return expo ? expf(l) : l;
  }
};

template <typename T>
__global__ void __launch_bounds__(256) gla_decay_kernel(const T* __restrict__ a, long long a_stride, const T* __restrict__ a2,
                                                        const float* __restrict__ a2_b, float* __restrict__ ld, int n_channels, int rank,
                                                        const DecayForm form) {
  extern __shared__ float as[];  // the token's low-rank input
  const long long t = blockIdx.x;
  for (int r = threadIdx.x; r < rank; r += blockDim.x) as[r] = ldf(a + t * a_stride + r);
  __syncthreads();
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < n_channels; c += gridDim.y * blockDim.x) {
    const T* w = a2 + static_cast<long long>(c) * rank;
    float z = 0.f;
    for (int r = 0; r < rank; ++r) z = fmaf(ldf(w + r), as[r], z);
    z += a2_b ? a2_b[c] : 0.f;
    ld[t * n_channels + c] = form(z, c);
  }
}

// Many tokens: block = 128 channels x 32 tokens, a thread owns 4 channels of 4 tokens.  The low rank is walked in pieces of kDecayR: the block's
// rows of A2 and its tokens' low-rank inputs sit in shared memory, rank first, so a step is two 16-byte reads for 16 multiply-adds.
// The sum runs over r in increasing order as in the kernel above: both give the same bits.
constexpr int kDecayTokens = 32, kDecayChannels = 128, kDecayR = 32;
template <typename T>
__global__ void __launch_bounds__(256) gla_decay_tile_kernel(const T* __restrict__ a, long long a_stride, const T* __restrict__ a2,
                                                             const float* __restrict__ a2_b, float* __restrict__ ld, int n_tokens, int n_channels,
                                                             int rank, const DecayForm form) {
  __shared__ __align__(16) float w[kDecayR][kDecayChannels + 4];
  __shared__ __align__(16) float as[kDecayR][kDecayTokens + 4];
  const int c0 = blockIdx.x * kDecayChannels, t0 = blockIdx.y * kDecayTokens, tid = threadIdx.x;
  const int cq = (tid & 31) * 4, tq = (tid >> 5) * 4;
  float acc[4][4];   // [token][channel]
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  for (int r0 = 0; r0 < rank; r0 += kDecayR) {
    const int rn = min(kDecayR, rank - r0);
    for (int e = tid; e < kDecayChannels * kDecayR; e += 256) {
      const int c = e / kDecayR, r = e - c * kDecayR;
      w[r][c] = (r < rn && c0 + c < n_channels) ? ldf(a2 + static_cast<long long>(c0 + c) * rank + r0 + r) : 0.f;
    }
    for (int e = tid; e < kDecayTokens * kDecayR; e += 256) {
      const int t = e / kDecayR, r = e - t * kDecayR;
      as[r][t] = (r < rn && t0 + t < n_tokens) ? ldf(a + static_cast<long long>(t0 + t) * a_stride + r0 + r) : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int r = 0; r < rn; ++r) {
      const float4 wv = *reinterpret_cast<const float4*>(&w[r][cq]), av = *reinterpret_cast<const float4*>(&as[r][tq]);
      const float at[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = fmaf(wv.x, at[i], acc[i][0]);
        acc[i][1] = fmaf(wv.y, at[i], acc[i][1]);
        acc[i][2] = fmaf(wv.z, at[i], acc[i][2]);
        acc[i][3] = fmaf(wv.w, at[i], acc[i][3]);
      }
    }
    __syncthreads();
  }
  float bias[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) bias[j] = (a2_b && c0 + cq + j < n_channels) ? a2_b[c0 + cq + j] : 0.f;
  const bool vec = (n_channels & 3) == 0 && (reinterpret_cast<uintptr_t>(ld) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (t0 + tq + i >= n_tokens) break;
    float* o = ld + static_cast<long long>(t0 + tq + i) * n_channels + c0 + cq;
    if (vec && c0 + cq < n_channels) {
      *reinterpret_cast<float4*>(o) = make_float4(form(acc[i][0] + bias[0], c0 + cq), form(acc[i][1] + bias[1], c0 + cq + 1), form(acc[i][2] + bias[2], c0 + cq + 2),
                                                  form(acc[i][3] + bias[3], c0 + cq + 3));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c0 + cq + j < n_channels) o[j] = form(acc[i][j] + bias[j], c0 + cq + j);
    }
  }
}

// Grid (sequence, head, slice of value columns): the columns of S evolve independently given the decays, k and q.  Thread
// (r, c) owns rows r, r + R, ... of column c of the slice; threads past VS * R only take part in loads.
template <typename T>
__global__ void __launch_bounds__(1024) gla_scan_kernel(const pcs_gla_params p, int VS, int R) {
  extern __shared__ float sm[];
  const int D = p.dim, V = p.vdim, H = p.heads;
  const int v0 = blockIdx.z * VS, vs = min(VS, V - v0);
  float* S = sm;               // [D][VS]
  float* ks = S + D * VS;      // [D]
  float* qs = ks + D;          // [D]
  float* as = qs + D;          // [D] decay
  float* vsm = as + D;         // [VS]
  float* part = vsm + VS;      // [R][VS]
  const int b = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, nthr = blockDim.x;
  const int slot = p.seq_slot[b], pos0 = p.seq_pos0[b], len = p.seq_len[b], off = p.seq_off[b];
  if (len <= 0) return;
  float* Sg = p.s_pool + (static_cast<long long>(slot) * H + head) * D * V;
  const bool fresh = pos0 == 0;
  for (int e = tid; e < D * vs; e += nthr) {
    const int d = e / vs, c = e - d * vs;
    S[d * VS + c] = fresh ? 0.f : Sg[d * V + v0 + c];
  }
  const int c = tid % VS, r = tid / VS;
  const bool active = r < R && c < vs;
  __syncthreads();
  for (int i = 0; i < len; ++i) {
    const long long t = off + i;
    const T* row = static_cast<const T*>(p.proj) + t * p.row_stride;
    const float* ldr = p.ld + t * (static_cast<long long>(H) * D) + head * D;
    for (int d = tid; d < D; d += nthr) {
      ks[d] = ldf(row + p.k_off + head * D + d);
      qs[d] = ldf(row + p.q_off + head * D + d) * p.q_scale;
      as[d] = expf(ldr[d]);
    }
    for (int e = tid; e < vs; e += nthr) vsm[e] = ldf(row + p.v_off + head * V + v0 + e);
    __syncthreads();
    if (active) {
      const float vv = vsm[c];
      float num = 0.f;
      for (int d = r; d < D; d += R) {
        const float sv = fmaf(as[d], S[d * VS + c], ks[d] * vv);
        S[d * VS + c] = sv;
        num = fmaf(sv, qs[d], num);
      }
      part[r * VS + c] = num;
    }
    __syncthreads();
    if (tid < vs) {
      float o = 0.f;
      for (int rr = 0; rr < R; ++rr) o += part[rr * VS + tid];
      p.o_raw[t * (static_cast<long long>(H) * V) + head * V + v0 + tid] = o;
    }
    __syncthreads();  // ks / qs / as / vsm / part are rewritten by the next token
  }
  for (int e = tid; e < D * vs; e += nthr) {
    const int d = e / vs, cc = e - d * vs;
    Sg[d * V + v0 + cc] = S[d * VS + cc];
  }
}

constexpr int kGlaRing = 24;   // shared-memory slots of tokens whose k / q / v / decays are in flight or waiting
constexpr int kGlaAhead = 16;  // tokens requested ahead of the arithmetic
constexpr int kGlaGroup = 4;   // tokens computed between two block barriers

template <int N>
__device__ __forceinline__ void ldv(const float* p, float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = p[i];
}
template <int N>
__device__ __forceinline__ void ldv(const __nv_bfloat16* p, float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = __bfloat162float(p[i]);
}

// The same recurrence with the state in REGISTERS.  A warp owns 8 value columns; lane l owns the DR = ceil(dim / 32) rows
// l*DR .. l*DR + DR - 1 of them, so a thread keeps a DR x 8 patch of S.  Per token a thread does 2 * DR * 8 fused
// multiply-adds from 3 * DR + 8 shared-memory values; the 8 column sums over the 32 lanes are one reduce-scatter butterfly.
// k, q, v (compute type) and the log decays (32-bit) of the next tokens arrive through a ring of shared-memory slots filled by
// cp.async, kGlaAhead tokens ahead of the arithmetic; kGlaGroup tokens are computed between two block barriers.  The order of
// every sum is fixed by DR alone: a token's result does not depend on how the sequence is cut into steps or on the batch.
template <typename T, int DR>
__global__ void __launch_bounds__(512) gla_scan_reg_kernel(const pcs_gla_params p, int W) {
  extern __shared__ __align__(16) unsigned char ring[];
  constexpr int ES = static_cast<int>(sizeof(T)), PER = 16 / ES;
  const int D = p.dim, V = p.vdim, H = p.heads;
  const int slot_bytes = (2 * D + 8 * W) * ES + D * 4;  // k[D] q[D] v[8W] (compute type), ld[D] (32-bit)
  const int b = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * 8 * W;
  const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int slot = p.seq_slot[b], pos0 = p.seq_pos0[b], len = p.seq_len[b], off = p.seq_off[b];
  if (len <= 0) return;
  const int c0 = v0 + warp * 8, d0 = lane * DR;
  const int ncol = max(0, min(8, V - c0));
  const T* proj = static_cast<const T*>(p.proj);
  const int ck = D / PER, cv = 8 * W / PER, cl = D / 4;
  const int n_pieces = 2 * ck + cv + cl;
  auto issue = [&](int i) {  // token i of this entry into slot i % kGlaRing
    const long long t = off + i;
    unsigned char* s = ring + (i % kGlaRing) * slot_bytes;
    const T* row = proj + t * p.row_stride;
    for (int e = tid; e < n_pieces; e += nthr) {
      if (e < ck) cp_async16(s + e * 16, row + p.k_off + head * D + e * PER);
      else if (e < 2 * ck) cp_async16(s + D * ES + (e - ck) * 16, row + p.q_off + head * D + (e - ck) * PER);
      else if (e < 2 * ck + cv) {
        const int c = e - 2 * ck, col = v0 + c * PER;
        if (col < V) cp_async16(s + 2 * D * ES + c * 16, row + p.v_off + head * V + col);
        else *reinterpret_cast<uint4*>(s + 2 * D * ES + c * 16) = make_uint4(0u, 0u, 0u, 0u);
      } else {
        const int c = e - 2 * ck - cv;
        cp_async16(s + (2 * D + 8 * W) * ES + c * 16, p.ld + t * (static_cast<long long>(H) * D) + head * D + c * 4);
      }
    }
  };
  for (int i = 0; i < kGlaAhead; ++i) {
    if (i < len) issue(i);
    cp_async_commit();
  }
  float* Sg = p.s_pool + (static_cast<long long>(slot) * H + head) * D * V;
  const bool fresh = pos0 == 0;
  float S[DR][8];
#pragma unroll
  for (int r = 0; r < DR; ++r) {
    const int d = d0 + r;
#pragma unroll
    for (int c = 0; c < 8; ++c) S[r][c] = (!fresh && d < D && c < ncol) ? Sg[static_cast<long long>(d) * V + c0 + c] : 0.f;
  }
  for (int i0 = 0; i0 < len; i0 += kGlaGroup) {
    cp_async_wait<kGlaAhead - kGlaGroup>();  // this thread's copies of tokens i0 .. i0 + 3 have landed ...
    __syncthreads();                         // ... and everybody's; the slots of the previous groups have been read by all warps
#pragma unroll
    for (int u = 0; u < kGlaGroup; ++u) {
      if (i0 + kGlaAhead + u < len) issue(i0 + kGlaAhead + u);
      cp_async_commit();
    }
#pragma unroll
    for (int u = 0; u < kGlaGroup; ++u) {
      const int i = i0 + u;
      if (i >= len) break;
      const long long t = off + i;
      const unsigned char* cur = ring + (i % kGlaRing) * slot_bytes;
      const T* kb = reinterpret_cast<const T*>(cur);
      const T* qb = kb + D;
      const T* vb = qb + D;
      const float* lb = reinterpret_cast<const float*>(cur + (2 * D + 8 * W) * ES);
      float kk[DR], qq[DR], aa[DR], vv[8];
#pragma unroll
      for (int r = 0; r < DR; ++r) {
        const bool ok = d0 + r < D;
        kk[r] = ok ? ldf(kb + d0 + r) : 0.f;
        qq[r] = ok ? ldf(qb + d0 + r) * p.q_scale : 0.f;
        aa[r] = ok ? expf(lb[d0 + r]) : 0.f;
      }
      ldv<8>(vb + warp * 8, vv);
      float num[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float acc = 0.f;
#pragma unroll
        for (int r = 0; r < DR; ++r) {
          S[r][c] = fmaf(aa[r], S[r][c], kk[r] * vv[c]);
          acc = fmaf(S[r][c], qq[r], acc);
        }
        num[c] = acc;
      }
      // reduce-scatter over the lanes: afterwards lane l holds the sum of column ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 + ((l >> 2) & 1)
      float x4[4], x2[2], x1;
      {
        const bool up = lane & 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float recv = __shfl_xor_sync(0xffffffffu, up ? num[j] : num[j + 4], 16);
          x4[j] = (up ? num[j + 4] : num[j]) + recv;
        }
      }
      {
        const bool up = lane & 8;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float recv = __shfl_xor_sync(0xffffffffu, up ? x4[j] : x4[j + 2], 8);
          x2[j] = (up ? x4[j + 2] : x4[j]) + recv;
        }
      }
      {
        const bool up = lane & 4;
        const float recv = __shfl_xor_sync(0xffffffffu, up ? x2[0] : x2[1], 4);
        x1 = (up ? x2[1] : x2[0]) + recv;
      }
      x1 += __shfl_xor_sync(0xffffffffu, x1, 2);
      x1 += __shfl_xor_sync(0xffffffffu, x1, 1);
      const int col = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
      if ((lane & 3) == 0 && col < ncol) p.o_raw[t * (static_cast<long long>(H) * V) + head * V + c0 + col] = x1;
    }
  }
#pragma unroll
  for (int r = 0; r < DR; ++r) {
    const int d = d0 + r;
    if (d < D) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < ncol) Sg[static_cast<long long>(d) * V + c0 + c] = S[r][c];
    }
  }
}

// out[t, head, :] = o / rms(o) * norm_w * silu(g): one block of kOutThreads per (token, head); a thread's columns, their gates and
// norm weights are requested together before the reduction.
constexpr int kOutThreads = 128, kOutCols = 4;   // up to kOutThreads * kOutCols columns stay in registers
template <typename T>
__device__ __forceinline__ void gla_head_out(const float* __restrict__ o, const T* __restrict__ g, const T* __restrict__ nw, T* __restrict__ out, int V,
                                             float eps, float* red) {
  float ov[kOutCols], gv[kOutCols], wv[kOutCols];
  float ss = 0.f;
#pragma unroll
  for (int u = 0; u < kOutCols; ++u) {
    const int c = threadIdx.x + u * kOutThreads;
    ov[u] = c < V ? o[c] : 0.f;
    gv[u] = c < V ? ldf(g + c) : 0.f;
    wv[u] = c < V ? ldf(nw + c) : 0.f;
  }
#pragma unroll
  for (int u = 0; u < kOutCols; ++u) ss = fmaf(ov[u], ov[u], ss);
  for (int c = threadIdx.x + kOutCols * kOutThreads; c < V; c += kOutThreads) ss = fmaf(o[c], o[c], ss);
  ss = block_sum(ss, red);
  const float inv = 1.f / sqrtf(ss / static_cast<float>(V) + eps);
#pragma unroll
  for (int u = 0; u < kOutCols; ++u) {
    const int c = threadIdx.x + u * kOutThreads;
    if (c < V) stf(out + c, ov[u] * inv * wv[u] * (gv[u] * sigmoidf_(gv[u])));
  }
  for (int c = threadIdx.x + kOutCols * kOutThreads; c < V; c += kOutThreads) {
    const float x = ldf(g + c);
    stf(out + c, o[c] * inv * ldf(nw + c) * (x * sigmoidf_(x)));
  }
}

template <typename T>
__global__ void __launch_bounds__(kOutThreads) gla_out_kernel(const pcs_gla_params p) {
  __shared__ float red[33];
  const int V = p.vdim, H = p.heads, head = blockIdx.y;
  const long long t = blockIdx.x;
  gla_head_out<T>(p.o_raw + t * (static_cast<long long>(H) * V) + head * V, static_cast<const T*>(p.proj) + t * p.row_stride + p.g_off + head * V,
                  static_cast<const T*>(p.norm_w), static_cast<T*>(p.out) + t * (static_cast<long long>(H) * V) + head * V, V, p.eps, red);
}

// ---- the chunkwise form (prompts) -------------------------------------------------------------------------------------
// One block per (chunk, head).  q, k and the running sums of the log decays of the chunk sit in shared memory as 32-bit rows
// of DP numbers: dim + 1 where the pairs' loop reads single numbers (a row per token: threads that walk the tokens at a fixed channel touch different
// banks), dim + 4 where it reads 16-byte pieces (eight neighbouring rows in different banks).  The scores
// inside the chunk are formed pair by pair with the exact factor exp(B_i[d] - B_s[d]) <= 1 per channel, so no decay, however
// strong, overflows a factor; everything that crosses chunks is left to matrix products on exp(B_i) and exp(B_e - B_i) <= 1.
constexpr int kPrepThreads = 1024;
template <typename T>
__global__ void __launch_bounds__(kPrepThreads) gla_chunk_prep_kernel(const pcs_gla_chunk_params p, const int DP) {
  extern __shared__ float sm[];
  const int D = p.dim, V = p.vdim, H = p.heads, C = p.chunk;
  const bool rows4 = DP == D + 4;   // rows of whole 16-byte pieces
  float* qs = sm;              // [C][DP]
  float* ks = qs + C * DP;     // [C][DP]
  float* Bs = ks + C * DP;     // [C][DP]
  const int cn = blockIdx.x, head = blockIdx.y, tid = threadIdx.x;
  const int first = p.chunk_first[cn], n = p.chunk_len[cn];
  const T* proj = static_cast<const T*>(p.proj);
  // rows in pieces of four channels, a warp per row, where the sizes allow it (bfloat16 runs)
  const int warp = tid >> 5, lane = tid & 31;
  auto al = [](const void* q, int b) { return (reinterpret_cast<uintptr_t>(q) & (b - 1)) == 0; };
  const bool quads = sizeof(T) == 2 && rows4 && V % 4 == 0 && p.q_off % 4 == 0 && p.k_off % 4 == 0 && p.v_off % 4 == 0 && p.row_stride % 4 == 0 && al(p.proj, 8) &&
                     al(p.ld, 16) && al(p.qd, 16) && al(p.kd, 16) && al(p.vf, 16);
  auto ld4 = [](const T* x) {
    const uint2 u = *reinterpret_cast<const uint2*>(x);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
  };
  if (quads) {
    for (int i = warp; i < C; i += kPrepThreads / 32) {
      const T* row = proj + static_cast<long long>(first + i) * p.row_stride;
      for (int d = lane * 4; d < D; d += 128) {
        float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), kv = qv, lv = qv;
        if (i < n) {
          qv = ld4(row + p.q_off + head * D + d);
          kv = ld4(row + p.k_off + head * D + d);
          lv = *reinterpret_cast<const float4*>(p.ld + static_cast<long long>(first + i) * (H * D) + head * D + d);
        }
        *reinterpret_cast<float4*>(qs + i * DP + d) = make_float4(qv.x * p.q_scale, qv.y * p.q_scale, qv.z * p.q_scale, qv.w * p.q_scale);
        *reinterpret_cast<float4*>(ks + i * DP + d) = kv;
        *reinterpret_cast<float4*>(Bs + i * DP + d) = lv;
      }
    }
  } else
  for (int e = tid; e < C * D; e += kPrepThreads) {
    const int i = e / D, d = e - i * D;
    float qv = 0.f, kv = 0.f, lv = 0.f;
    if (i < n) {
      const T* row = proj + static_cast<long long>(first + i) * p.row_stride;
      qv = ldf(row + p.q_off + head * D + d) * p.q_scale;
      kv = ldf(row + p.k_off + head * D + d);
      lv = p.ld[static_cast<long long>(first + i) * (H * D) + head * D + d];
    }
    qs[i * DP + d] = qv;
    ks[i * DP + d] = kv;
    Bs[i * DP + d] = lv;
  }
  __syncthreads();
  for (int d = tid; d < D; d += kPrepThreads) {  // running sums over the chunk's tokens, per channel (rows past the chunk add nothing)
    float acc = 0.f;
    for (int i = 0; i < C; ++i) {
      acc += Bs[i * DP + d];
      Bs[i * DP + d] = acc;
    }
  }
  __syncthreads();
  const long long base = static_cast<long long>(cn) * H + head;
  float* qd = p.qd + base * C * D;
  float* kd = p.kd + base * C * D;
  const float* Be = Bs + (C - 1) * DP;
  if (quads) {
    for (int i = warp; i < C; i += kPrepThreads / 32)
      for (int d = lane * 4; d < D; d += 128) {
        const float4 b = *reinterpret_cast<const float4*>(Bs + i * DP + d), be = *reinterpret_cast<const float4*>(Be + d);
        const float4 q = *reinterpret_cast<const float4*>(qs + i * DP + d), k = *reinterpret_cast<const float4*>(ks + i * DP + d);
        *reinterpret_cast<float4*>(qd + i * D + d) = make_float4(q.x * expf(b.x), q.y * expf(b.y), q.z * expf(b.z), q.w * expf(b.w));
        *reinterpret_cast<float4*>(kd + i * D + d) = make_float4(k.x * expf(be.x - b.x), k.y * expf(be.y - b.y), k.z * expf(be.z - b.z), k.w * expf(be.w - b.w));
      }
  } else
  for (int e = tid; e < C * D; e += kPrepThreads) {
    const int i = e / D, d = e - i * D;
    const float bi = Bs[i * DP + d];
    qd[e] = qs[i * DP + d] * expf(bi);
    kd[e] = ks[i * DP + d] * expf(Be[d] - bi);
  }
  for (int d = tid; d < D; d += kPrepThreads) p.g[base * D + d] = expf(Be[d]);
  float* vf = p.vf + base * C * V;
  if (quads) {
    for (int i = warp; i < C; i += kPrepThreads / 32)
      for (int c = lane * 4; c < V; c += 128)
        *reinterpret_cast<float4*>(vf + i * V + c) = i < n ? ld4(proj + static_cast<long long>(first + i) * p.row_stride + p.v_off + head * V + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  } else
  for (int e = tid; e < C * V; e += kPrepThreads) {
    const int i = e / V, c = e - i * V;
    vf[e] = i < n ? ldf(proj + static_cast<long long>(first + i) * p.row_stride + p.v_off + head * V + c) : 0.f;
  }
  // scores inside the chunk.  Query rows i and C - 1 - i together have C + 1 visible keys, so the pairs are walked as C / 2 rows of
  // C + 1 places with every lane busy; lanes of a warp mostly walk the keys of one query (k and B rows in different banks, q and
  // B_i broadcast).  Pairs above the diagonal, and rows past the chunk's end, are zero.
  float* a = p.a + base * C * C;
  for (int e = tid; e < C * C; e += kPrepThreads) a[e] = 0.f;
  // bfloat16 projections: the pair factors go through the base-2 exponential unit (relative error 2^-22, far below the operands'
  // rounding), with the running sums rescaled once; float32 runs keep the library exponential
  constexpr bool kFast = sizeof(T) == 2;
  __syncthreads();
  if (kFast) {
    for (int e = tid; e < C * D; e += kPrepThreads) {
      const int i = e / D, d = e - i * D;
      Bs[i * DP + d] *= 1.4426950408889634f;
    }
  }
  __syncthreads();
  const int half = (C + 1) / 2, places = half * (C + 1);
  auto pair_at = [&](int e, int& i, int& s_) {
    const int r = e / (C + 1), j = e - r * (C + 1);
    if (j <= r) { i = r; s_ = j; } else { i = C - 1 - r; s_ = j - r - 1; }
    return i < n && s_ <= i && !(i == r && j > r);   // (an odd chunk's middle row is taken once)
  };
  // bfloat16 runs: whole rounds of one pair per thread, and the pairs that are left one per warp (64 tokens: 2080 pairs are two rounds and 32 pairs)
  const int whole = kFast ? places / kPrepThreads * kPrepThreads : places;
  for (int e = whole + warp; e < places; e += kPrepThreads / 32) {
    int i, s_;
    if (!pair_at(e, i, s_)) continue;
    float x = 0.f;
    for (int d = lane; d < D; d += 32) x = fmaf(qs[i * DP + d] * ks[s_ * DP + d], ex2(Bs[i * DP + d] - Bs[s_ * DP + d]), x);
    x = warp_sum(x);
    if (lane == 0) a[i * C + s_] = x;
  }
  for (int e = tid; e < whole; e += kPrepThreads) {
    int i, s_;
    if (!pair_at(e, i, s_)) continue;
    const float* qi = qs + i * DP;
    const float* bi = Bs + i * DP;
    const float* kk = ks + s_ * DP;
    const float* bs = Bs + s_ * DP;
    float a0 = 0.f, a1 = 0.f;
    int d = 0;
    if (kFast && rows4) {   // four channels per read: the loop is bound by shared memory (with the loads in pieces and the pairs in whole rounds: 86 -> 56 us at 136 chunks of 256 channels)
#pragma unroll 2
      for (; d < D; d += 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(qi + d), k4 = *reinterpret_cast<const float4*>(kk + d);
        const float4 b4 = *reinterpret_cast<const float4*>(bi + d), c4 = *reinterpret_cast<const float4*>(bs + d);
        a0 = fmaf(q4.x * k4.x, ex2(b4.x - c4.x), a0);
        a1 = fmaf(q4.y * k4.y, ex2(b4.y - c4.y), a1);
        a0 = fmaf(q4.z * k4.z, ex2(b4.z - c4.z), a0);
        a1 = fmaf(q4.w * k4.w, ex2(b4.w - c4.w), a1);
      }
    }
    for (; d + 1 < D; d += 2) {
      a0 = fmaf(qi[d] * kk[d], kFast ? ex2(bi[d] - bs[d]) : expf(bi[d] - bs[d]), a0);
      a1 = fmaf(qi[d + 1] * kk[d + 1], kFast ? ex2(bi[d + 1] - bs[d + 1]) : expf(bi[d + 1] - bs[d + 1]), a1);
    }
    if (d < D) a0 = fmaf(qi[d] * kk[d], kFast ? ex2(bi[d] - bs[d]) : expf(bi[d] - bs[d]), a0);
    a[i * C + s_] = a0 + a1;
  }
}

// The same for bfloat16 runs of 64 tokens in 16-byte pieces.  The exact factor of every pair costs an exponential per channel (532 k a block; they and the four rows they read bounded the
// kernel above, 67 of its 102 k cycles): here only pairs inside blocks of 16 tokens do.  For tokens of different blocks the factor is a product of at most three numbers <= 1, from the key to the end
// of its block, over the blocks between, and from the start of the query's block, so these pairs are plain dot products of rows scaled once.
// Running sums are kept inside the blocks (Bs), with the blocks' sums beside them.  Figures: 132 blocks of 64 x 256, 55 us above,
// 26 here: 41 by the blocks, 29 once a row's pieces are requested together and nobody wants the copies of the values, 26 with two by two pairs inside the blocks
// (one at a time read four rows per pair, and shared memory was what they waited for).
// Error against float64 (rms, decays of logsigmoid(z + 1) / 16), exact exponentials / here: pairs of different blocks 2.34e-7 / 2.20e-7 at 256 channels, 1.60e-7 / 1.36e-7 at 64, inside 2.06e-7 / 0.95e-7
// (shorter running sums); with decays fifty times weaker a product of several rounded factors shows, 2.07e-7 / 2.22e-7 across, 1.96e-7 / 0.93e-7 inside.
constexpr int kP64 = 64, kP64Block = 16;
__global__ void __launch_bounds__(kPrepThreads) gla_chunk_prep64_kernel(const pcs_gla_chunk_params p) {
  extern __shared__ __align__(16) float sm[];
  const int D = p.dim, V = p.vdim, H = p.heads, DP = D + 4, per = D / 4;
  float* qs = sm;               // [64][DP]: q; later scaled from its block's start
  float* ks = qs + kP64 * DP;   // [64][DP]: k; later scaled to its block's end
  float* Bs = ks + kP64 * DP;   // [64][DP]: running sums inside the blocks
  float* T = Bs + kP64 * DP;    // [4][D] the blocks' sums; later, in rows 1 and 2, their exponentials
  const int cn = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = p.chunk_first[cn], n = p.chunk_len[cn];
  const __nv_bfloat16* proj = static_cast<const __nv_bfloat16*>(p.proj);
  constexpr float kLog2e = 1.4426950408889634f;
  auto ld4 = [](const __nv_bfloat16* x) {
    const uint2 u = *reinterpret_cast<const uint2*>(x);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
  };
  const long long base = static_cast<long long>(cn) * H + head;
  float* a = p.a + base * kP64 * kP64;
  {   // two rows per warp, all of their pieces under way at once
    constexpr int kIt = 2;   // (dim <= 256)
    uint2 q2[2][kIt], k2[2][kIt];
    float4 l4[2][kIt];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int i = warp + 32 * u, d = lane * 4 + 128 * it;
        q2[u][it] = k2[u][it] = make_uint2(0u, 0u);
        l4[u][it] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n && d < D) {
          const __nv_bfloat16* row = proj + static_cast<long long>(first + i) * p.row_stride + head * D + d;
          q2[u][it] = *reinterpret_cast<const uint2*>(row + p.q_off);
          k2[u][it] = *reinterpret_cast<const uint2*>(row + p.k_off);
          l4[u][it] = *reinterpret_cast<const float4*>(p.ld + static_cast<long long>(first + i) * (H * D) + head * D + d);
        }
      }
    auto wide = [](const uint2& u) { return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u)); };
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int it = 0; it < kIt; ++it) {
        const int i = warp + 32 * u, d = lane * 4 + 128 * it;
        if (d < D) {
          const float4 q = wide(q2[u][it]);
          *reinterpret_cast<float4*>(qs + i * DP + d) = make_float4(q.x * p.q_scale, q.y * p.q_scale, q.z * p.q_scale, q.w * p.q_scale);
          *reinterpret_cast<float4*>(ks + i * DP + d) = wide(k2[u][it]);
          *reinterpret_cast<float4*>(Bs + i * DP + d) = l4[u][it];
        }
      }
  }
  if (p.vf) {   // (NULL: the caller reads the values themselves)
    float* vf = p.vf + base * kP64 * V;
    for (int i = warp; i < kP64; i += kPrepThreads / 32)
      for (int c = lane * 4; c < V; c += 128)
        *reinterpret_cast<float4*>(vf + i * V + c) = i < n ? ld4(proj + static_cast<long long>(first + i) * p.row_stride + p.v_off + head * V + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int e = tid; e < kP64 * kP64; e += kPrepThreads)
    if ((e & 63) > (e >> 6)) a[e] = 0.f;   // above the diagonal
  __syncthreads();
  for (int e = tid; e < 4 * D; e += kPrepThreads) {   // (block, channel)
    const int blk = e / D, d = e - blk * D;
    float* b = Bs + blk * kP64Block * DP + d;
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < kP64Block; ++i) {
      acc += b[i * DP];
      b[i * DP] = acc;
    }
    T[e] = acc;
  }
  __syncthreads();
  // Pairs inside the blocks: tiles of two rows by two keys, 36 of a block's 64 hold a pair (i, s <= i).  A warp takes two tiles, sixteen lanes each, which split the channels.
  for (int w = warp; w < 72; w += kPrepThreads / 32) {
    const int t4 = w * 2 + (lane >> 4), blk = t4 / 36, tr = t4 - blk * 36;
    int ti = static_cast<int>((sqrtf(8.f * tr + 1.f) - 1.f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= tr) ++ti;
    while (ti * (ti + 1) / 2 > tr) --ti;
    const int i = blk * kP64Block + 2 * ti, s_ = blk * kP64Block + 2 * (tr - ti * (ti + 1) / 2);
    float v[4] = {0.f, 0.f, 0.f, 0.f};   // [row][key]
    for (int d = (lane & 15) * 4; d < D; d += 64) {
      float bs[2][4], kk[2][4];
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        ldx(Bs + (s_ + y) * DP + d, bs[y]);
        ldx(ks + (s_ + y) * DP + d, kk[y]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float bi[4], qi[4];
        ldx(Bs + (i + u) * DP + d, bi);
        ldx(qs + (i + u) * DP + d, qi);
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int c = 0; c < 4; ++c) v[2 * u + y] = fmaf(qi[c] * kk[y][c], ex2((bi[c] - bs[y][c]) * kLog2e), v[2 * u + y]);   // (in a tile on the diagonal one pair looks ahead, and is dropped)
      }
    }
    // halves change places until a lane holds a quarter of one sum
#pragma unroll
    for (int h = 2; h >= 1; h >>= 1) {
      const int m = 4 * h;
      const bool up = lane & m;
#pragma unroll
      for (int x = 0; x < h; ++x) {
        const float send = up ? v[x] : v[x + h], keep = up ? v[x + h] : v[x];
        v[x] = keep + __shfl_xor_sync(0xffffffffu, send, m);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    const int iu = i + (lane >> 3 & 1), sy = s_ + (lane >> 2 & 1);
    if (!(lane & 3) && sy <= iu) a[iu * kP64 + sy] = v[0];
  }
  __syncthreads();
  // what leaves the chunk, and the rows scaled within their blocks
  float* qd = p.qd + base * kP64 * D;
  float* kd = p.kd + base * kP64 * D;
  for (int i = warp; i < kP64; i += kPrepThreads / 32) {
    const int blk = i / kP64Block;
    for (int d = lane * 4; d < D; d += 128) {
      float t[4][4], b[4], q[4], k[4], x[4], y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) ldx(T + j * D + d, t[j]);
      ldx(Bs + i * DP + d, b);
      ldx(qs + i * DP + d, q);
      ldx(ks + i * DP + d, k);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float before = blk == 0 ? 0.f : blk == 1 ? t[0][c] : blk == 2 ? t[0][c] + t[1][c] : (t[0][c] + t[1][c]) + t[2][c];
        const float after = blk == 3 ? 0.f : blk == 2 ? t[3][c] : blk == 1 ? t[2][c] + t[3][c] : t[1][c] + (t[2][c] + t[3][c]);
        const float left = (blk == 0 ? t[0][c] : blk == 1 ? t[1][c] : blk == 2 ? t[2][c] : t[3][c]) - b[c];
        x[c] = q[c] * expf(before + b[c]);
        y[c] = k[c] * expf(left + after);
        q[c] *= ex2(b[c] * kLog2e);
        k[c] *= ex2(left * kLog2e);
      }
      stx(qd + i * D + d, x);
      stx(kd + i * D + d, y);
      stx(qs + i * DP + d, q);
      stx(ks + i * DP + d, k);
    }
  }
  for (int d = tid; d < D; d += kPrepThreads) p.g[base * D + d] = expf((T[d] + T[D + d]) + (T[2 * D + d] + T[3 * D + d]));
  __syncthreads();
  for (int e = tid; e < 2 * D; e += kPrepThreads) T[D + e] = ex2(T[D + e] * kLog2e);
  __syncthreads();
  // pairs across blocks: six (I, J) pairs of 16 x 16, 2 x 2 pairs by two threads of a warp that split the channels (eight neighbouring lanes as above)
  if (tid < 6 * 128) {
    const int pr = tid >> 7, q4 = (tid >> 4 & 7) * 8 + (tid & 7);
    const int I = pr == 0 ? 1 : pr < 3 ? 2 : 3, J = pr == 0 ? 0 : pr < 3 ? pr - 1 : pr - 3;
    const int i = I * kP64Block + (q4 >> 3), s_ = J * kP64Block + (q4 & 7);   // rows i, i + 8 and keys s, s + 8
    const bool over1 = J == 0 && I > 1, over2 = J < 2 && I == 3;               // block 1 lies between, block 2
    float x[2][2] = {};
    for (int j = tid >> 3 & 1; j < per; j += 2) {
      const int d = 4 * j;
      float qa[4], qb[4], ka[4], kb[4];
      ldx(qs + i * DP + d, qa);
      ldx(qs + (i + 8) * DP + d, qb);
      ldx(ks + s_ * DP + d, ka);
      ldx(ks + (s_ + 8) * DP + d, kb);
      if (over1 || over2) {
        float f[4] = {1.f, 1.f, 1.f, 1.f}, t[4];
        if (over1) ldx(T + D + d, f);
        if (over2) {
          ldx(T + 2 * D + d, t);
#pragma unroll
          for (int c = 0; c < 4; ++c) f[c] *= t[c];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) { ka[c] *= f[c]; kb[c] *= f[c]; }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        x[0][0] = fmaf(qa[c], ka[c], x[0][0]);
        x[0][1] = fmaf(qa[c], kb[c], x[0][1]);
        x[1][0] = fmaf(qb[c], ka[c], x[1][0]);
        x[1][1] = fmaf(qb[c], kb[c], x[1][1]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < 2; ++v) x[u][v] += __shfl_xor_sync(0xffffffffu, x[u][v], 8);
    const int u = tid >> 3 & 1;   // each of the two writes a row
    a[(i + 8 * u) * kP64 + s_] = u ? x[1][0] : x[0][0];
    a[(i + 8 * u) * kP64 + s_ + 8] = u ? x[1][1] : x[0][1];
  }
}

// A chunk's own sum of k v^T, decayed to its end: u[c, h] = kd[c, h]^T v (bfloat16 runs, chunks of 64).  kd is 32-bit and enters the tensor cores as three
// bfloat16 parts (all 24 bits of it), v is bfloat16 already, the sums are 32-bit: as exact as the library's 32-bit product this stands for, which runs on the
// multiply-add units (59 us at 34 chunks x 4 heads of 256 x 512; this: 38 us).  Block = (chunk, head, 128 value columns), a warp = 32 channels x 64 columns
// per turn; kd stays 32-bit in shared memory and is taken apart in registers (rows D + 4 numbers apart: a fragment's eight channels x four token pairs lie in
// different banks).
constexpr int kSumsThreads = 256, kSumsCols = 128, kSumsChunk = 64, kSumsRow = kSumsCols + 8;
__global__ void __launch_bounds__(kSumsThreads, 2) gla_chunk_sums_kernel(const pcs_gla_chunk_params p) {
  extern __shared__ __align__(16) float sm[];
  const int D = p.dim, V = p.vdim, H = p.heads, LK = D + 4;
  float* Ks = sm;                                                                  // [64][D + 4]
  __nv_bfloat16* Vs = reinterpret_cast<__nv_bfloat16*>(Ks + kSumsChunk * LK);      // [64][136]
  const int cn = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * kSumsCols, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3;
  const long long base = static_cast<long long>(cn) * H + head;
  const int first = p.chunk_first[cn], n = p.chunk_len[cn], pieces = D / 4;
  const float* kd = p.kd + base * kSumsChunk * D;
  for (int e = tid; e < kSumsChunk * pieces; e += kSumsThreads) {
    const int r = e / pieces, c = (e - r * pieces) * 4;
    cp_async16(Ks + r * LK + c, kd + r * D + c);
  }
  const __nv_bfloat16* rows = static_cast<const __nv_bfloat16*>(p.proj) + static_cast<long long>(first) * p.row_stride + p.v_off + head * V + v0;
#pragma unroll
  for (int u = 0; u < kSumsChunk * kSumsCols / 8 / kSumsThreads; ++u) {
    const int e = tid + u * kSumsThreads, r = e / (kSumsCols / 8), c = e % (kSumsCols / 8) * 8;
    if (r < n && v0 + c < V) cp_async16(Vs + r * kSumsRow + c, rows + r * p.row_stride + c);
    else *reinterpret_cast<uint4*>(Vs + r * kSumsRow + c) = make_uint4(0u, 0u, 0u, 0u);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const uint32_t v_base = static_cast<uint32_t>(__cvta_generic_to_shared(Vs)) + ((lane & 15) * kSumsRow + (lane >> 4) * 8) * 2;
  float* U = p.u + base * D * V;
  // a pair of neighbouring tokens at one channel as three packed parts
  auto parts = [](float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack_bf16(x0, x1);
    x0 -= __uint_as_float(h << 16);
    x1 -= __uint_as_float(h & 0xffff0000u);
    m = split_pair(x0, x1, l);
  };
  for (int w = warp; w < (D + 31) / 32 * 2; w += kSumsThreads / 32) {
    const int d0 = (w >> 1) * 32, c0 = (w & 1) * 64;
    if (v0 + c0 >= V) continue;
    float acc[2][8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < kSumsChunk / 16; ++ks) {
      uint32_t f[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) ldsm_x4_t(v_base + (ks * 16 * kSumsRow + c0 + u * 16) * 2, f[u][0], f[u][1], f[u][2], f[u][3]);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float step[8][4];   // sums of sixteen tokens join in rounded additions: the tensor core's own running sum cuts bits off (1.35e-7 -> 1.5e-7 of a state)
#pragma unroll
        for (int j = 0; j < 8; ++j) step[j][0] = step[j][1] = step[j][2] = step[j][3] = 0.f;
        uint32_t a[3][4];   // [part][fragment register]: channels grp, grp + 8; tokens 2 qd.., 2 qd + 8..
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int d = d0 + i * 16 + grp + (q & 1) * 8, s = ks * 16 + 2 * qd + (q >> 1) * 8;
          const float* k = Ks + s * LK + min(d, D - 1);
          parts(k[0], k[LK], a[0][q], a[1][q], a[2][q]);
        }
#pragma unroll
        for (int x = 2; x >= 0; --x)   // the smallest part first
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            mma_bf16(step[2 * u], a[x][0], a[x][1], a[x][2], a[x][3], f[u][0], f[u][1]);
            mma_bf16(step[2 * u + 1], a[x][0], a[x][1], a[x][2], a[x][3], f[u][2], f[u][3]);
          }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[i][j][q] += step[j][q];
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int d = d0 + i * 16 + grp, col = v0 + c0 + j * 8 + qd * 2;
        if (col >= V) continue;
        if (d < D) *reinterpret_cast<float2*>(U + static_cast<long long>(d) * V + col) = make_float2(acc[i][j][0], acc[i][j][1]);
        if (d + 8 < D) *reinterpret_cast<float2*>(U + static_cast<long long>(d + 8) * V + col) = make_float2(acc[i][j][2], acc[i][j][3]);
      }
  }
}

// The sums and the scan in one kernel: block = 64 state rows x 64 columns of one (entry, head), the chunks in order.  Per chunk the state it starts from goes to u,
// S <- g S + kd^T v for the tile, the product as in gla_chunk_sums_kernel; the chunks' own sums never pass through memory, kd and v are read again by every tile (24 KB a chunk, from L2).
// Four warps, one per scheduler, hold 16 rows x 64 columns each in registers, so that every number of kd is taken apart once per block; four others keep the loads three chunks ahead.
// 33 chunks of 4 heads of 256 x 512: 41 us (sums 38, scan 30); the wrapper's rule says for which walks (a step takes 1.25 to 1.33 us whatever the number of blocks, so few tiles over long walks
// stay with the sums of all chunks side by side).
constexpr int kStMul = 128, kStThreads = 2 * kStMul, kStStages = 4, kStKRow = 68, kStVRow = 72;
constexpr int kStStage = kSumsChunk * (kStKRow * 4 + kStVRow * 2) + 64 * 4;   // bytes: kd, v, the rows' decays
__global__ void __launch_bounds__(kStThreads, 2) gla_chunk_states_kernel(const pcs_gla_chunk_params p) {
  extern __shared__ __align__(16) unsigned char st_smem[];
  const int D = p.dim, V = p.vdim, H = p.heads, b = blockIdx.z, head = blockIdx.y, vtiles = (V + 63) / 64;
  const int d0 = static_cast<int>(blockIdx.x) / vtiles * 64, v0 = static_cast<int>(blockIdx.x) % vtiles * 64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3;
  const int nc = p.seq_chunks[b], c0 = p.seq_chunk0[b];
  if (nc <= 0) return;
  if (tid >= kStMul) {
    const int ht = tid - kStMul, kr = ht >> 4, kc = (ht & 15) * 4, vr = ht >> 3, vc = (ht & 7) * 8;   // pieces of every eighth row of kd, of every sixteenth of v
    const bool k_in = d0 + kc < D, v_in = v0 + vc < V;
    const long long rs = p.row_stride, step_k = static_cast<long long>(H) * kSumsChunk * D;
    const float* ks = p.kd + (static_cast<long long>(c0) * H + head) * kSumsChunk * D + kr * D + d0 + kc;
    const float* gs = p.g + (static_cast<long long>(c0) * H + head) * D + d0 + ht * 4;
    const __nv_bfloat16* vs = static_cast<const __nv_bfloat16*>(p.proj) + p.v_off + head * V + v0 + vc;
    int loaded = 0;
    auto load = [&]() {
      if (loaded < nc) {
        unsigned char* st = st_smem + loaded % kStStages * kStStage;
        float* kd = reinterpret_cast<float*>(st) + kr * kStKRow + kc;
        __nv_bfloat16* vd = reinterpret_cast<__nv_bfloat16*>(st + kSumsChunk * kStKRow * 4) + vr * kStVRow + vc;
        const int n = p.chunk_len[c0 + loaded];
        const __nv_bfloat16* src = vs + (static_cast<long long>(p.chunk_first[c0 + loaded]) + vr) * rs;
#pragma unroll
        for (int u = 0; u < kSumsChunk / 8; ++u) {
          if (k_in) cp_async16(kd + 8 * u * kStKRow, ks + 8 * u * D);
          else *reinterpret_cast<float4*>(kd + 8 * u * kStKRow) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kSumsChunk / 16; ++u) {
          if (v_in && vr + 16 * u < n) cp_async16(vd + 16 * u * kStVRow, src + 16 * u * rs);
          else *reinterpret_cast<uint4*>(vd + 16 * u * kStVRow) = make_uint4(0u, 0u, 0u, 0u);
        }
        if (ht < 16 && d0 + 4 * ht < D) cp_async16(st + kStStage - 256 + ht * 16, gs);
        ks += step_k;
        gs += static_cast<long long>(H) * D;
        ++loaded;
      }
      cp_async_commit();
    };
#pragma unroll 1
    for (int c = 0; c < kStStages - 1; ++c) load();
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
      cp_async_wait<kStStages - 2>();
      __syncthreads();   // chunk c has landed; what chunk c - 1 lay in is free
      load();
    }
    return;
  }
  // this lane's state: rows dr and dr + 8, columns vc + 8 j and the next
  const int dl = warp * 16 + grp, dr = d0 + dl, vc = v0 + 2 * qd;
  float* Sg = p.s_pool + (static_cast<long long>(p.seq_slot[b]) * H + head) * D * V;
  const bool fresh = p.seq_pos0[b] == 0;
  float s[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      s[j][2 * i] = s[j][2 * i + 1] = 0.f;
      if (!fresh && dr + 8 * i < D && vc + 8 * j < V) {
        const float2 x = *reinterpret_cast<const float2*>(Sg + static_cast<long long>(dr + 8 * i) * V + vc + 8 * j);
        s[j][2 * i] = x.x;
        s[j][2 * i + 1] = x.y;
      }
    }
  float* U = p.u + (static_cast<long long>(c0) * H + head) * D * V + static_cast<long long>(dr) * V + vc;
  const long long step_u = static_cast<long long>(H) * D * V;
  const uint32_t v_base = static_cast<uint32_t>(__cvta_generic_to_shared(st_smem)) + kSumsChunk * kStKRow * 4 + ((lane & 15) * kStVRow + (lane >> 4) * 8) * 2;
  auto parts = [](float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack_bf16(x0, x1);
    x0 -= __uint_as_float(h << 16);
    x1 -= __uint_as_float(h & 0xffff0000u);
    m = split_pair(x0, x1, l);
  };
#pragma unroll 1
  for (int c = 0, st = 0; c < nc; ++c, U += step_u) {
    __syncthreads();   // chunk c stands
    const unsigned char* stage = st_smem + st * kStStage;
    const float* ks = reinterpret_cast<const float*>(stage) + 2 * qd * kStKRow + dl;
    const float* gs = reinterpret_cast<const float*>(stage + kStStage - 256) + dl;
    const uint32_t vb = v_base + st * kStStage;
    // the state this chunk starts from
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (dr + 8 * i < D && vc + 8 * j < V) *reinterpret_cast<float2*>(U + 8 * i * V + 8 * j) = make_float2(s[j][2 * i], s[j][2 * i + 1]);
    const float g0 = gs[0], g1 = gs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { s[j][0] *= g0; s[j][1] *= g0; s[j][2] *= g1; s[j][3] *= g1; }
#pragma unroll
    for (int k16 = 0; k16 < kSumsChunk / 16; ++k16) {
      uint32_t a[3][4];   // [part][fragment register]: rows grp, grp + 8; tokens 2 qd.., 2 qd + 8..
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float* k = ks + (k16 * 16 + (q >> 1) * 8) * kStKRow + (q & 1) * 8;
        parts(k[0], k[kStKRow], a[0][q], a[1][q], a[2][q]);
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t f[2][4];
        float step[4][4];   // sums of sixteen tokens join in rounded additions
#pragma unroll
        for (int u = 0; u < 2; ++u) ldsm_x4_t(vb + (k16 * 16 * kStVRow + (half * 2 + u) * 16) * 2, f[u][0], f[u][1], f[u][2], f[u][3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) step[j][0] = step[j][1] = step[j][2] = step[j][3] = 0.f;
#pragma unroll
        for (int x = 2; x >= 0; --x)   // the smallest part first
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            mma_bf16(step[2 * u], a[x][0], a[x][1], a[x][2], a[x][3], f[u][0], f[u][1]);
            mma_bf16(step[2 * u + 1], a[x][0], a[x][1], a[x][2], a[x][3], f[u][2], f[u][3]);
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) s[4 * half + j][q] += step[j][q];
      }
    }
    st = st + 1 == kStStages ? 0 : st + 1;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (dr + 8 * i < D && vc + 8 * j < V) *reinterpret_cast<float2*>(Sg + static_cast<long long>(dr + 8 * i) * V + vc + 8 * j) = make_float2(s[j][2 * i], s[j][2 * i + 1]);
}

// One thread per VW neighbouring value columns of one state row: the entry's chunks in order.  The sums and decays of eight
// chunks are requested before the dependent chain S <- g S + u runs over them, so eight loads per thread are in flight.
template <int VW>
__global__ void __launch_bounds__(256) gla_chunk_scan_kernel(const pcs_gla_chunk_params p) {
  const int D = p.dim, V = p.vdim, H = p.heads;
  const int b = blockIdx.z, head = blockIdx.y;
  const int nchunks = p.seq_chunks[b];
  if (nchunks <= 0) return;
  const long long e = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * VW;
  if (e >= static_cast<long long>(D) * V) return;
  const int d = static_cast<int>(e / V);
  const int slot = p.seq_slot[b], c0 = p.seq_chunk0[b];
  float* Sg = p.s_pool + (static_cast<long long>(slot) * H + head) * D * V + e;
  float S[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) S[j] = p.seq_pos0[b] == 0 ? 0.f : Sg[j];
  const long long cstride = static_cast<long long>(H) * D * V;
  float* u0 = p.u + (static_cast<long long>(c0) * H + head) * D * V + e;
  const float* g0 = p.g + (static_cast<long long>(c0) * H + head) * D + d;
  constexpr int U = 8;
  for (int c = 0; c < nchunks; c += U) {
    float un[U][VW], gn[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (c + k < nchunks) {
        gn[k] = g0[static_cast<long long>(c + k) * H * D];
        if (VW == 4) {
          const float4 v = *reinterpret_cast<const float4*>(u0 + (c + k) * cstride);
          un[k][0] = v.x; un[k][1 % VW] = v.y; un[k][2 % VW] = v.z; un[k][3 % VW] = v.w;
        } else {
          un[k][0] = u0[(c + k) * cstride];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (c + k < nchunks) {
        float* u = u0 + (c + k) * cstride;
        if (VW == 4) *reinterpret_cast<float4*>(u) = make_float4(S[0], S[1 % VW], S[2 % VW], S[3 % VW]);
        else u[0] = S[0];
#pragma unroll
        for (int j = 0; j < VW; ++j) S[j] = fmaf(gn[k], S[j], un[k][j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < VW; ++j) Sg[j] = S[j];
}

template <typename T>
__global__ void __launch_bounds__(kOutThreads) gla_chunk_out_kernel(const pcs_gla_chunk_params p) {
  __shared__ float red[33];
  const int V = p.vdim, H = p.heads, C = p.chunk, head = blockIdx.y;
  const long long t = blockIdx.x;
  const int row = p.tok_row[t];
  gla_head_out<T>(p.o + ((static_cast<long long>(row / C) * H + head) * C + row % C) * V, static_cast<const T*>(p.proj) + t * p.row_stride + p.g_off + head * V,
                  static_cast<const T*>(p.norm_w), static_cast<T*>(p.out) + t * (static_cast<long long>(H) * V) + head * V, V, p.eps, red);
}

}  // namespace pcs

PCS_API int pcs_gla_chunk_prep(const pcs_gla_chunk_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_chunk_prep: null params");
  if (p->n_chunks == 0) return PCS_OK;
  PCS_REQUIRE(p->proj && p->ld && p->chunk_first && p->chunk_len && p->qd && p->kd && p->g && p->a, "pcs_gla_chunk_prep: null tensor");
  PCS_REQUIRE(p->heads > 0 && p->heads <= 65535 && p->dim > 0 && p->vdim > 0 && p->chunk > 0, "pcs_gla_chunk_prep: bad sizes");
  // (32-bit runs read single numbers: rows of dim + 4 would put four neighbouring rows into one bank)
  constexpr size_t kLimit = 220 * 1024;
  auto bytes = [&](int row) { return static_cast<size_t>(3) * p->chunk * row * sizeof(float); };
  const int row = p->dtype == PCS_BF16 && p->dim % 4 == 0 && bytes(p->dim + 4) <= kLimit ? p->dim + 4 : p->dim + 1;
  const size_t smem = bytes(row);
  PCS_REQUIRE(smem <= kLimit, "pcs_gla_chunk_prep: a chunk of %d tokens x %d channels exceeds shared memory", p->chunk, p->dim);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto al = [](const void* q, int b) { return (reinterpret_cast<uintptr_t>(q) & (b - 1)) == 0; };
  const size_t smem64 = (static_cast<size_t>(3) * pcs::kP64 * (p->dim + 4) + 4 * p->dim) * sizeof(float);
  if (p->dtype == PCS_BF16 && p->chunk == pcs::kP64 && p->dim % 4 == 0 && p->vdim % 4 == 0 && p->q_off % 4 == 0 && p->k_off % 4 == 0 && p->v_off % 4 == 0 && p->row_stride % 4 == 0 &&
      p->dim <= 256 && al(p->proj, 8) && al(p->ld, 16) && al(p->qd, 16) && al(p->kd, 16) && al(p->vf, 16) && smem64 <= kLimit) {
    PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_chunk_prep64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kLimit)));
    pcs::gla_chunk_prep64_kernel<<<dim3(p->n_chunks, p->heads), pcs::kPrepThreads, smem64, st>>>(*p);
    PCS_CHECK_CUDA(cudaGetLastError());
    pcs::count_launch();
    return PCS_OK;
  }
  PCS_REQUIRE(p->vf, "pcs_gla_chunk_prep: null tensor");
  if (smem > 48 * 1024)
    PCS_DISPATCH(p->dtype, PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_chunk_prep_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kLimit))));
  PCS_DISPATCH(p->dtype, pcs::gla_chunk_prep_kernel<T><<<dim3(p->n_chunks, p->heads), pcs::kPrepThreads, smem, st>>>(*p, row));
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

// PCS_ERR_UNSUPPORTED: other types, chunks or sizes (the caller forms the product itself)
PCS_API int pcs_gla_chunk_sums(const pcs_gla_chunk_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_chunk_sums: null params");
  if (p->n_chunks == 0) return PCS_OK;
  PCS_REQUIRE(p->proj && p->kd && p->u && p->chunk_first && p->chunk_len && p->heads > 0 && p->heads <= 65535 && p->dim > 0 && p->vdim > 0, "pcs_gla_chunk_sums: bad arguments");
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (p->dtype != PCS_BF16 || p->chunk != pcs::kSumsChunk || p->dim % 16 != 0 || p->dim > 256 || p->vdim % 8 != 0 || p->v_off % 8 != 0 || p->row_stride % 8 != 0 ||
      !al16(p->proj) || !al16(p->kd) || !al16(p->u))
    return pcs::set_error(PCS_ERR_UNSUPPORTED, "pcs_gla_chunk_sums: serves bfloat16 in 16-byte pieces, chunks of %d, dim a multiple of 16 up to 256", pcs::kSumsChunk);
  auto smem = [](int D) { return static_cast<size_t>(pcs::kSumsChunk) * (D + 4) * sizeof(float) + static_cast<size_t>(pcs::kSumsChunk) * pcs::kSumsRow * 2; };
  PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_chunk_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem(256))));
  pcs::gla_chunk_sums_kernel<<<dim3(p->n_chunks, p->heads, (p->vdim + pcs::kSumsCols - 1) / pcs::kSumsCols), pcs::kSumsThreads, smem(p->dim),
                               static_cast<cudaStream_t>(stream)>>>(*p);
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

// What pcs_gla_chunk_sums serves, with vdim a multiple of 8 and 16-byte aligned pools; PCS_ERR_UNSUPPORTED otherwise
PCS_API int pcs_gla_chunk_states(const pcs_gla_chunk_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_chunk_states: null params");
  if (p->n_seqs == 0 || p->n_chunks == 0) return PCS_OK;
  PCS_REQUIRE(p->proj && p->kd && p->u && p->g && p->s_pool && p->chunk_first && p->chunk_len && p->seq_slot && p->seq_pos0 && p->seq_chunk0 && p->seq_chunks &&
              p->heads > 0 && p->heads <= 65535 && p->n_seqs <= 65535 && p->dim > 0 && p->vdim > 0, "pcs_gla_chunk_states: bad arguments");
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (p->dtype != PCS_BF16 || p->chunk != pcs::kSumsChunk || p->dim % 16 != 0 || p->dim > 256 || p->vdim % 8 != 0 || p->v_off % 8 != 0 || p->row_stride % 8 != 0 ||
      !al16(p->proj) || !al16(p->kd) || !al16(p->u) || !al16(p->g) || !al16(p->s_pool))
    return pcs::set_error(PCS_ERR_UNSUPPORTED, "pcs_gla_chunk_states: serves bfloat16 in 16-byte pieces, chunks of %d, dim a multiple of 16 up to 256", pcs::kSumsChunk);
  constexpr int smem = pcs::kStStages * pcs::kStStage;
  PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_chunk_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  pcs::gla_chunk_states_kernel<<<dim3(((p->dim + 63) / 64) * ((p->vdim + 63) / 64), p->heads, p->n_seqs), pcs::kStThreads, smem, static_cast<cudaStream_t>(stream)>>>(*p);
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

PCS_API int pcs_gla_chunk_scan(const pcs_gla_chunk_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_chunk_scan: null params");
  if (p->n_seqs == 0 || p->n_chunks == 0) return PCS_OK;
  PCS_REQUIRE(p->u && p->g && p->s_pool && p->seq_slot && p->seq_pos0 && p->seq_chunk0 && p->seq_chunks, "pcs_gla_chunk_scan: null tensor");
  PCS_REQUIRE(p->heads > 0 && p->heads <= 65535 && p->n_seqs <= 65535 && p->dim > 0 && p->vdim > 0, "pcs_gla_chunk_scan: bad sizes");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long elems = static_cast<long long>(p->dim) * p->vdim;
  if (p->vdim % 4 == 0 && ((reinterpret_cast<uintptr_t>(p->u) | reinterpret_cast<uintptr_t>(p->s_pool)) & 15) == 0)
    pcs::gla_chunk_scan_kernel<4><<<dim3(static_cast<unsigned>((elems / 4 + 255) / 256), p->heads, p->n_seqs), 256, 0, st>>>(*p);
  else
    pcs::gla_chunk_scan_kernel<1><<<dim3(static_cast<unsigned>((elems + 255) / 256), p->heads, p->n_seqs), 256, 0, st>>>(*p);
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

PCS_API int pcs_gla_chunk_out(const pcs_gla_chunk_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_chunk_out: null params");
  if (p->n_tokens == 0) return PCS_OK;
  PCS_REQUIRE(p->proj && p->o && p->tok_row && p->norm_w && p->out && p->chunk > 0 && p->heads > 0 && p->vdim > 0, "pcs_gla_chunk_out: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PCS_DISPATCH(p->dtype, pcs::gla_chunk_out_kernel<T><<<dim3(p->n_tokens, p->heads), pcs::kOutThreads, 0, st>>>(*p));
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

PCS_API int pcs_gla_decay(const void* a, int64_t a_stride, const void* a2, const float* a2_b, float* ld, int n_tokens, int n_channels, int rank,
                          float tau, const float* rate, int rate_dim, int expo, int dtype, void* stream) {
  if (n_tokens == 0) return PCS_OK;
  PCS_REQUIRE(a && a2 && ld && n_channels > 0 && rank > 0 && rank <= 8192 && (rate ? rate_dim > 0 : tau > 0.f), "pcs_gla_decay: bad arguments");
  const pcs::DecayForm form{rate ? 0.f : 1.f / tau, rate, rate_dim, expo};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (n_tokens >= 2 * pcs::kDecayTokens) {
    dim3 grid((n_channels + pcs::kDecayChannels - 1) / pcs::kDecayChannels, (n_tokens + pcs::kDecayTokens - 1) / pcs::kDecayTokens);
    PCS_DISPATCH(dtype, pcs::gla_decay_tile_kernel<T><<<grid, 256, 0, st>>>(static_cast<const T*>(a), a_stride, static_cast<const T*>(a2), a2_b, ld, n_tokens, n_channels,
                                                                           rank, form));
  } else
  PCS_DISPATCH(dtype, pcs::gla_decay_kernel<T><<<dim3(n_tokens, (n_channels + 255) / 256 > 64 ? 64 : (n_channels + 255) / 256), 256, rank * sizeof(float), st>>>(static_cast<const T*>(a), a_stride, static_cast<const T*>(a2),
                                                                                           a2_b, ld, n_channels, rank, form));
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch();
  return PCS_OK;
}

PCS_API int pcs_gla_scan(const pcs_gla_params* p, void* stream) {
  PCS_REQUIRE(p, "pcs_gla_scan: null params");
  if (p->n_seqs == 0 || p->n_tokens == 0) return PCS_OK;
  PCS_REQUIRE(p->proj && p->ld && p->norm_w && p->out && p->s_pool && p->seq_slot && p->seq_pos0 && p->seq_len && p->seq_off && p->o_raw,
              "pcs_gla_scan: null tensor");
  PCS_REQUIRE(p->heads > 0 && p->heads <= 65535 && p->dim > 0 && p->vdim > 0 && p->n_tokens > 0, "pcs_gla_scan: bad sizes");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int es = p->dtype == PCS_BF16 ? 2 : 4, per = 16 / es;
  const bool aligned = p->dim % per == 0 && p->dim % 4 == 0 && p->vdim % per == 0 && p->q_off % per == 0 && p->k_off % per == 0 && p->v_off % per == 0 &&
                       p->row_stride % per == 0 && reinterpret_cast<uintptr_t>(p->proj) % 16 == 0 && reinterpret_cast<uintptr_t>(p->ld) % 16 == 0;
  if (p->impl != 1 && p->dim <= 256 && aligned) {
    // register-resident state: warps per block halve until the launch has two blocks per SM (or 2 warps are left)
    int W = 16;
    while (W > 1 && 8 * (W / 2) >= p->vdim) W /= 2;
    auto blocks = [&](int w) { return static_cast<long long>(p->n_seqs) * p->heads * ((p->vdim + 8 * w - 1) / (8 * w)); };
    while (W > 2 && blocks(W) < 2 * 148) W /= 2;
    if (W < 2) W = 2;
    const int DR = p->dim <= 32 ? 1 : p->dim <= 64 ? 2 : p->dim <= 128 ? 4 : 8;
    const size_t smem = static_cast<size_t>(pcs::kGlaRing) * ((2 * p->dim + 8 * W) * es + p->dim * 4);
    if (smem > 48 * 1024) {
#define PCS_GLA_ATTR(DRV) PCS_DISPATCH(p->dtype, PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_scan_reg_kernel<T, DRV>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024)))
      if (DR == 1) PCS_GLA_ATTR(1);
      else if (DR == 2) PCS_GLA_ATTR(2);
      else if (DR == 4) PCS_GLA_ATTR(4);
      else PCS_GLA_ATTR(8);
#undef PCS_GLA_ATTR
    }
    dim3 grid(p->n_seqs, p->heads, (p->vdim + 8 * W - 1) / (8 * W));
#define PCS_GLA_REG(DRV) PCS_DISPATCH(p->dtype, (pcs::gla_scan_reg_kernel<T, DRV><<<grid, 32 * W, smem, st>>>(*p, W)))
    if (DR == 1) PCS_GLA_REG(1);
    else if (DR == 2) PCS_GLA_REG(2);
    else if (DR == 4) PCS_GLA_REG(4);
    else PCS_GLA_REG(8);
#undef PCS_GLA_REG
    PCS_CHECK_CUDA(cudaGetLastError());
  } else {
    // slice width: at most 128 columns, and small enough that the slice of S fits shared memory
    int VS = p->vdim < 128 ? p->vdim : 128;
    while (VS > 8 && static_cast<size_t>(p->dim) * VS * sizeof(float) > 160 * 1024) VS /= 2;
    int R = 512 / VS;
    if (R < 1) R = 1;
    if (R > p->dim) R = p->dim;
    const int slices = (p->vdim + VS - 1) / VS;
    const int threads = ((VS * R + 31) / 32) * 32;
    const size_t smem = (static_cast<size_t>(p->dim) * VS + 3 * p->dim + VS + static_cast<size_t>(R) * VS) * sizeof(float);
    PCS_REQUIRE(smem <= 220 * 1024, "pcs_gla_scan: a state of %d rows exceeds shared memory", p->dim);
    if (smem > 48 * 1024)
      PCS_DISPATCH(p->dtype, PCS_CHECK_CUDA(cudaFuncSetAttribute(pcs::gla_scan_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)));
    dim3 grid(p->n_seqs, p->heads, slices);
    PCS_DISPATCH(p->dtype, pcs::gla_scan_kernel<T><<<grid, threads, smem, st>>>(*p, VS, R));
    PCS_CHECK_CUDA(cudaGetLastError());
  }
  PCS_DISPATCH(p->dtype, pcs::gla_out_kernel<T><<<dim3(p->n_tokens, p->heads), pcs::kOutThreads, 0, st>>>(*p));
  PCS_CHECK_CUDA(cudaGetLastError());
  pcs::count_launch(2);
  return PCS_OK;
}
