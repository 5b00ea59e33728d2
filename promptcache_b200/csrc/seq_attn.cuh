// What the attention kernels over the slot pool share: the keys a query sees, and where its result goes.
#pragma once
#include "seq_common.cuh"

namespace pcs {

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

}  // namespace pcs
