// What the attention kernels over the slot pool share: the keys a query sees, and where its result goes.
#pragma once
#include "seq_common.cuh"

namespace pcs {

// (slot, K/V head) planes of a pool for its tensor maps: they end where the pool ends, if the caller says where that is
inline unsigned long long pool_planes(const pcs_attn_params& p) {
  return p.n_slots > 0 ? static_cast<unsigned long long>(p.n_slots) * p.n_kv_heads : 1ull << 30;
}

// A launch over a step's own dense K/V (`pool_slot`) with rows of 96 and 64 numbers once ended with an illegal memory access.  What raised it is not known: the sizes, strides and slots it
// got are in range, and so is every index that the kernel forms from them.  Such pools with rows that a tensor map's boxes of 64 columns do not divide are served by the mma.sync kernel, which
// reads by plain loads, until it is known (and which forms a row again whose result is not finite there, as the tcgen05 kernels do).
inline bool dense_rows_off_boxes(const pcs_attn_params& p) { return p.pool_slot && (p.dim % 64 != 0 || p.vdim % 64 != 0); }

// the launch chooses the kernel (1 and 2 name one)
inline bool automatic(const pcs_attn_params& p) { return p.impl == 0 || p.impl == 3 || p.impl == 4 || p.impl == 7; }

constexpr int kAttnMaxSplits = 64;  // partial results of one (token, head) that attn_combine_kernel merges

// The keys a query at position `pos` sees, as one dense index range: with a window, the kept first keys [0, n_first) and
// then the window [lo, pos]; without one (or when the two touch), all of [0, pos].  With chunks, the keys of the query's own chunk.
struct VisibleKeys {
  int n_first, lo, count;
  __device__ __forceinline__ VisibleKeys(int pos, int window, int keep_first, int chunk) {
    lo = window > 0 ? max(0, pos - window + 1) : (chunk > 0 ? pos / chunk * chunk : 0);
    n_first = chunk > 0 ? 0 : min(max(keep_first, 0), lo);
    count = n_first + (pos + 1 - lo);
  }
  __device__ __forceinline__ int key(int v) const { return v < n_first ? v : lo + (v - n_first); }
};

// The key tiles of BN keys that the new tokens [a, e) of an entry walk: [0, nf) and [lo, hi)
template <int BN>
struct Walk {
  int nf, lo, n;   // n: tiles in all
  __host__ __device__ __forceinline__ Walk(const pcs_attn_params& p, int pos0, int len, int a, int e) {
    const int first = pos0 + a, keep = p.window > 0 ? min(max(p.keep_first, 0), pos0 + len) : 0;
    lo = p.window > 0 ? max(0, first - p.window + 1) / BN : p.chunk > 0 ? first / p.chunk * p.chunk / BN : 0;
    nf = (keep + BN - 1) / BN;
    if (nf >= lo) nf = lo = 0;
    n = nf + (pos0 + e + BN - 1) / BN - lo;
  }
  __host__ __device__ __forceinline__ int tile(int it) const { return it < nf ? it : lo + it - nf; }
};

// The entries of a launch as the host knows them: each by itself, or all like the longest one
struct Entries {
  const int32_t *pos0, *len;
  int n, any_pos0, any_len;
  Entries(const pcs_attn_params& p, const int32_t* host_pos0, const int32_t* host_len)
      : pos0(host_len ? host_pos0 : nullptr), len(host_pos0 ? host_len : nullptr), n(p.n_seqs), any_pos0(0), any_len(p.max_len) {
    const int keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap;
    any_pos0 = keys > p.max_len ? keys - p.max_len : 0;
  }
  int pos_of(int b) const { return pos0 ? pos0[b] : any_pos0; }
  int len_of(int b) const { return len ? len[b] : any_len; }
};

// where head h of token t is written, and what its normalised result is multiplied by: the constant and the head's gate
template <typename T>
__device__ __forceinline__ T* out_row(const pcs_attn_params& p, int t, int h) {
  return static_cast<T*>(p.out) + static_cast<long long>(t) * (p.out_stride > 0 ? p.out_stride : static_cast<long long>(p.n_heads) * p.vdim) + h * p.vdim;
}
template <typename T>
__device__ __forceinline__ float out_factor(const pcs_attn_params& p, int t, int h) {
  float f = p.out_scale != 0.f ? p.out_scale : 1.f;
  if (p.head_gate) f *= sigmoidf_(ldf(static_cast<const T*>(p.head_gate) + static_cast<long long>(t) * p.head_gate_stride + h));
  return f;
}

// Columns [c0, c0 + n) of the result of head h of token t (entry b, position pos), by one warp with multiply-adds over the visible keys alone; n <= 128,
// rows in 16-byte pieces.  A matrix product over tiles of keys multiplies hidden keys by a weight of 0, and 0 * inf is not 0: a query whose result is not
// finite there is formed again here, so that rows it does not see cannot reach it.
template <typename T>
__device__ __forceinline__ void attn_row_again(const pcs_attn_params& p, int b, int h, int t, int pos, int c0, int n) {
  constexpr int N = Vec<T>::n;
  const int lane = threadIdx.x & 31, D = p.dim, slot = p.pool_slot ? p.pool_slot[b] : p.seq_slot[b];
  const long long VS = p.v_row_stride > 0 ? p.v_row_stride : p.vdim, plane = (static_cast<long long>(slot) * p.n_kv_heads + h / (p.n_heads / p.n_kv_heads)) * p.cap;
  const T* q = static_cast<const T*>(p.q) + (static_cast<long long>(t) * p.n_heads + h) * D;
  const T* K = static_cast<const T*>(p.k_pool) + plane * D;
  const T* Vp = static_cast<const T*>(p.v_pool) + plane * VS + c0;
  const float scale = p.scale * (p.head_scale ? p.head_scale[h] : 1.f), r1 = p.bias_r1 ? p.bias_r1[h] : 0.f, r2 = p.bias_r1 ? p.bias_r2[h] : 0.f;
  const float* tab = p.bias_table ? p.bias_table + static_cast<long long>(h) * p.bias_len : nullptr;
  const VisibleKeys vis(pos, p.window, p.keep_first, p.chunk);
  float m = p.sink ? (p.sink_logit ? p.sink_logit[h] : 0.f) : -INFINITY, l = p.sink ? 1.f : 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int j0 = 0; j0 < vis.count; j0 += 32) {
    const int nt = min(32, vis.count - j0);
    float s = -INFINITY;
    if (lane < nt) {
      const int j = vis.key(j0 + lane);
      float a = 0.f;
      for (int d = 0; d < D; d += N) {
        float x[N], y[N];
        ld16(q + d, x);
        ld16(K + static_cast<long long>(j) * D + d, y);
#pragma unroll
        for (int e = 0; e < N; ++e) a = fmaf(x[e], y[e], a);
      }
      s = a * scale;
      if (p.softcap > 0.f) s = p.softcap * tanhf(s / p.softcap);
      if (p.bias_r1) s -= r1 * log1pf(r2 * static_cast<float>(pos - j));
      if (tab) s += tab[min(pos - j, p.bias_len - 1)];
    }
    const float mn = fmaxf(m, warp_max(s)), f = m == -INFINITY ? 0.f : expf(m - mn);
    const float w = lane < nt ? expf(s - (mn == -INFINITY ? 0.f : mn)) : 0.f;
    m = mn;
    l = l * f + warp_sum(w);
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] *= f;
    for (int i = 0; i < nt; ++i) {
      const float wi = __shfl_sync(0xffffffffu, w, i);
      const T* v = Vp + static_cast<long long>(vis.key(j0 + i)) * VS;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (lane + 32 * u < n) acc[u] = fmaf(wi, ldf(v + lane + 32 * u), acc[u]);
    }
  }
  const float inv = (l > 0.f ? 1.f / l : 0.f) * out_factor<T>(p, t, h);
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (lane + 32 * u < n) stf(out_row<T>(p, t, h) + c0 + lane + 32 * u, acc[u] * inv);
}

// The same as a call (in line, it made a walk of 6144 keys of the tcgen05 kernels 1 % slower; the 32-bit kernel is 1.5 % slower with a call)
template <typename T>
__device__ __noinline__ void attn_row_again_call(const pcs_attn_params& p, int b, int h, int t, int pos, int c0, int n) { attn_row_again<T>(p, b, h, t, pos, c0, n); }

}  // namespace pcs
