// Attention of a few tokens over many stored keys (decoding): the heads of a group share every row they read.
//
// Bound by the K / V rows themselves.  One block = (token, up to eight heads of one K/V head, split of the keys), 4 warps that never wait for each other
// inside the walk.  A warp takes four row loads at a time (a row in 16-byte pieces over 8, 16 or 32 neighbouring lanes, so every load instruction reads whole
// rows), and keeps for all its heads:
//   scores     every lane multiplies its piece of the row with its piece of each head's query (32-bit, in registers); the partial sums of several
//              rows and heads are reduced together, halving their number at each shuffle, so that a lane ends with one (row, head)
//   softmax    online, per warp and head, on those lanes; scale / cap / bias / masks once per score
//   values     V rows are requested before the scores are formed; every lane adds its piece to one 32-bit accumulator per head
// The warps meet once, at the end.  Two to eight splits of a token are one cluster and merge through distributed shared memory; more go through the
// workspace to attn_combine_kernel.
//
// 16 sequences at 2 - 4 thousand keys, 16 heads over 4 K/V heads of 128, bfloat16 (B200): 112 -> 37 us (2.7 TB/s of distinct bytes; attn_decode_kernel, one
// block per head, reads every row four times through L2 and adds a merge launch of 4 us).  16 heads of their own: 16 sequences at 2048 keys 83 -> 54 us.  Eight row loads at a time need 233 registers, two blocks per SM and a second wave: 53 us.
#include "seq_attn.cuh"
#include "seq_tc5.cuh"

namespace pcs {

namespace {

constexpr int kWarps = 4, kThreads = kWarps * 32, kLoads = 4;
constexpr int kMaxCluster = 8;

constexpr int ilog2(int v) { return v <= 1 ? 0 : 1 + ilog2(v / 2); }

template <typename T, int LK, int LV, int GP>
struct DecodeCfg {
  static constexpr int N = Vec<T>::n;                                  // elements of a 16-byte piece
  static constexpr int RK = 32 / LK, RV = 32 / LV;                     // rows of one load instruction
  static constexpr int KT = kLoads * RK;                               // keys of a warp's tile
  static constexpr int VL = KT / RV;                                   // V loads of a tile
  static constexpr int NG = LK / GP < 1 ? 1 : (LK / GP < kLoads ? LK / GP : kLoads);  // K loads whose sums are reduced together
  static constexpr int NVAL = NG * GP;                                 // their (row, head) sums, at most LK of them
  static constexpr int DUP = LK / NVAL;                                // lanes that end with the same sum
  static constexpr int VMAX = LV * N;                                  // value columns
  // weights of the warps' tiles; after the walk the warps' accumulators [warp][row group][head][column] and (m, l) [warp][head]
  static constexpr int kWeights = kWarps * KT * GP;
  static constexpr int kPart = kWarps * RV * GP * VMAX;
  static constexpr int kFloats = (kWeights > kPart ? kWeights : kPart) + 2 * kWarps * GP;
  // the cluster's partial results [split][head][column], then (m, l) [split][head]
  static constexpr int kMerge = kMaxCluster * GP * (VMAX + 2);
};

template <typename T, int LK, int LV, int GP>
__global__ void __launch_bounds__(kThreads) attn_group_decode_kernel(const pcs_attn_params p, const int n_blocks_per_group, const int cluster) {
  using C = DecodeCfg<T, LK, LV, GP>;
  constexpr int N = C::N;
  extern __shared__ __align__(16) float sm[];
  float* weights = sm;
  float* ml = sm + (C::kWeights > C::kPart ? C::kWeights : C::kPart);  // [warp][head][m, l]
  float* merge = ml + 2 * kWarps * GP;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (cluster) cluster_arrive();   // a block's shared memory may be written once it has started: the wait stands before the merge
  // grid (splits, groups, tokens)
  const int sp = blockIdx.x, S = gridDim.x, t = blockIdx.z;
  const int G = p.n_heads / p.n_kv_heads, g = blockIdx.y / n_blocks_per_group, hb = g * G + (blockIdx.y - g * n_blocks_per_group) * GP;
  const int heads = min(GP, (g + 1) * G - hb);   // live heads of this block
  const int b = p.tok_seq[t], pos = p.tok_pos[t], slot = p.pool_slot ? p.pool_slot[b] : p.seq_slot[b];
  const int D = p.dim, V = p.vdim;
  const long long VS = p.v_row_stride > 0 ? p.v_row_stride : V;
  const T* K = static_cast<const T*>(p.k_pool) + (static_cast<long long>(slot) * p.n_kv_heads + g) * p.cap * D;
  const T* Vp = static_cast<const T*>(p.v_pool) + (static_cast<long long>(slot) * p.n_kv_heads + g) * p.cap * VS;
  const VisibleKeys vis(pos, p.window, p.keep_first, p.chunk);
  const int tiles = (vis.count + C::KT - 1) / C::KT;
  const int tile0 = static_cast<int>(static_cast<long long>(sp) * tiles / S), tile1 = static_cast<int>(static_cast<long long>(sp + 1) * tiles / S);

  const int ck = (lane % LK) * N, rk = lane / LK, cv = (lane % LV) * N, rv = lane / LV;   // this lane's columns and row of a load
  const bool col_k = ck < D, col_v = cv < V;
  // the (row, head) sum this lane ends with
  const int val = (lane % LK) / C::DUP, own_h = val % GP, own_i = val / GP;
  const bool first_of_dups = (lane % LK) % C::DUP == 0;
  const int h = hb + min(own_h, heads - 1);
  const float scale = p.scale * (p.head_scale ? p.head_scale[h] : 1.f);
  const float r1 = p.bias_r1 ? p.bias_r1[h] : 0.f, r2 = p.bias_r1 ? p.bias_r2[h] : 0.f;
  const float* tab = p.bias_table ? p.bias_table + static_cast<long long>(h) * p.bias_len : nullptr;
  const bool sink_here = p.sink && sp == 0 && warp == 0;
  float m = sink_here ? (p.sink_logit ? p.sink_logit[h] : 0.f) : -INFINITY;   // the same on every lane of a head
  float l = (sink_here && first_of_dups && own_i == 0 && rk == 0) ? 1.f : 0.f; // this lane's share

  float q[GP][N], acc[GP][N];
#pragma unroll
  for (int i = 0; i < GP; ++i) {
#pragma unroll
    for (int e = 0; e < N; ++e) q[i][e] = acc[i][e] = 0.f;
    if (i < heads && col_k) ld16(static_cast<const T*>(p.q) + (static_cast<long long>(t) * p.n_heads + hb + i) * D + ck, q[i]);
  }
  float* w_tile = weights + warp * C::KT * GP;

  uint4 kr[kLoads];
  auto load_k = [&](int tile) {
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int j = tile * C::KT + i * C::RK + rk;
      kr[i] = make_uint4(0u, 0u, 0u, 0u);
      if (tile < tile1 && col_k && j < vis.count) kr[i] = *reinterpret_cast<const uint4*>(K + static_cast<long long>(vis.key(j)) * D + ck);
    }
  };
  load_k(tile0 + warp);
  for (int tile = tile0 + warp; tile < tile1; tile += kWarps) {
    uint4 vr[C::VL];
#pragma unroll
    for (int i = 0; i < C::VL; ++i) {
      const int j = tile * C::KT + i * C::RV + rv;
      vr[i] = make_uint4(0u, 0u, 0u, 0u);
      if (col_v && j < vis.count) vr[i] = *reinterpret_cast<const uint4*>(Vp + static_cast<long long>(vis.key(j)) * VS + cv);
    }
    // ---- scores ----
    float s[kLoads / C::NG];
#pragma unroll
    for (int grp = 0; grp < kLoads / C::NG; ++grp) {
      float x[C::NVAL];
#pragma unroll
      for (int i = 0; i < C::NG; ++i) {
        float k[N];
        ld16(reinterpret_cast<const T*>(&kr[grp * C::NG + i]), k);
#pragma unroll
        for (int hh = 0; hh < GP; ++hh) {
          float a = q[hh][0] * k[0];
#pragma unroll
          for (int e = 1; e < N; ++e) a = fmaf(q[hh][e], k[e], a);
          x[i * GP + hh] = a;
        }
      }
      int n = C::NVAL;
#pragma unroll
      for (int o = LK / 2; o >= 1; o >>= 1) {
        if (n > 1) {
          n >>= 1;
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int i = 0; i < C::NVAL / 2; ++i)
            if (i < n) {
              const float give = up ? x[i] : x[i + n], keep = up ? x[i + n] : x[i];
              x[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        } else {
          x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
        }
      }
      s[grp] = x[0];
    }
    load_k(tile + kWarps);
    // ---- this lane's scores: scale, cap, bias, mask ----
    float mx = -INFINITY;
#pragma unroll
    for (int grp = 0; grp < kLoads / C::NG; ++grp) {
      const int j = tile * C::KT + (grp * C::NG + own_i) * C::RK + rk;
      float z = s[grp] * scale;
      if (p.softcap > 0.f) z = p.softcap * tanhf(z / p.softcap);
      if (p.bias_r1 || tab) {
        const int d = pos - vis.key(min(j, vis.count - 1));
        if (p.bias_r1) z -= r1 * log1pf(r2 * static_cast<float>(d));
        if (tab) z += tab[min(d, p.bias_len - 1)];
      }
      s[grp] = j < vis.count ? z : -INFINITY;
      mx = fmaxf(mx, s[grp]);
    }
    // the head's maximum: over every lane bit that does not choose the head
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
      if (o < C::DUP || o >= C::DUP * GP) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float m_new = fmaxf(m, mx);   // minus infinity while the bias table hides every key so far (a tile has as few as four)
    if (__any_sync(0xffffffffu, m_new != m)) {
      const float f = m == -INFINITY ? 0.f : expf(m - m_new);
      l *= f;
      m = m_new;
#pragma unroll
      for (int hh = 0; hh < GP; ++hh) {
        const float fh = __shfl_sync(0xffffffffu, f, hh * C::DUP);
#pragma unroll
        for (int e = 0; e < N; ++e) acc[hh][e] *= fh;
      }
    }
    const float sub = m == -INFINITY ? 0.f : m;   // hidden scores then give exp(-inf) = 0
    __syncwarp();   // the previous tile's weights have been read
#pragma unroll
    for (int grp = 0; grp < kLoads / C::NG; ++grp) {
      const float w = expf(s[grp] - sub);
      if (first_of_dups) {
        l += w;
        w_tile[((grp * C::NG + own_i) * C::RK + rk) * GP + own_h] = w;
      }
    }
    __syncwarp();
    // ---- values ----
#pragma unroll
    for (int i = 0; i < C::VL; ++i) {
      float v[N];
      ld16(reinterpret_cast<const T*>(&vr[i]), v);
      const float* w = w_tile + (i * C::RV + rv) * GP;
#pragma unroll
      for (int hh = 0; hh < GP; ++hh) {
        const float wh = w[hh];
#pragma unroll
        for (int e = 0; e < N; ++e) acc[hh][e] = fmaf(wh, v[e], acc[hh][e]);
      }
    }
  }
  // ---- the warps' results ----
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
    if (o < C::DUP || o >= C::DUP * GP) l += __shfl_xor_sync(0xffffffffu, l, o);
  __syncthreads();   // every warp is done with its weights
  if (lane < LK && first_of_dups && own_i == 0) {
    ml[(warp * GP + own_h) * 2] = m;
    ml[(warp * GP + own_h) * 2 + 1] = l;
  }
  float* part = sm;
#pragma unroll
  for (int hh = 0; hh < GP; ++hh) {
    float* d = part + ((warp * C::RV + rv) * GP + hh) * C::VMAX + cv;
    if constexpr (N == 8) stx(d, acc[hh]); else stx(d, acc[hh]);
  }
  __syncthreads();
  // per head, once: the warps' factors (in the place of their maxima), the common maximum, the sum, and what a finished result is multiplied by.  (Formed
  // again for every column, the end of a block of eight heads of 256 columns took 9 us in a cluster.)
  float* common = ml + 1;   // [3][head], in the places of the first three warps' sums
  if (tid < GP) {
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, ml[(w * GP + tid) * 2]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      float* x = ml + (w * GP + tid) * 2;
      const float f = x[0] == -INFINITY ? 0.f : expf(x[0] - M);
      L = fmaf(x[1], f, L);
      x[0] = f;
    }
    common[tid * 2] = M;
    common[(GP + tid) * 2] = L;
    if (tid < heads) common[(2 * GP + tid) * 2] = (L > 0.f ? 1.f / L : 0.f) * out_factor<T>(p, t, hb + tid);
  }
  __syncthreads();
  auto block_sum_of = [&](int hh, int c) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      float x = 0.f;
#pragma unroll
      for (int r = 0; r < C::RV; ++r) x += part[((w * C::RV + r) * GP + hh) * C::VMAX + c];
      a = fmaf(x, ml[(w * GP + hh) * 2], a);
    }
    return a;
  };
  if (!cluster) {
    for (int i = tid; i < heads * C::VMAX; i += kThreads) {
      const int hh = i / C::VMAX, c = i - hh * C::VMAX;
      if (c >= V) continue;
      const float a = block_sum_of(hh, c);
      if (S == 1) {
        stf(out_row<T>(p, t, hb + hh) + c, a * common[(2 * GP + hh) * 2]);
      } else {
        float* ws = p.workspace + ((static_cast<long long>(t) * p.n_heads + hb + hh) * S + sp) * (V + 2);
        if (c == 0) { ws[0] = common[hh * 2]; ws[1] = common[(GP + hh) * 2]; }
        ws[2 + c] = a;
      }
    }
    return;
  }
  // a cluster's splits: block q writes every S-th group of eight columns; everybody sends it the sums of them
  float* mm = merge + kMaxCluster * GP * C::VMAX;
  __syncwarp();
  cluster_wait();
  for (int i = tid; i < heads * C::VMAX; i += kThreads) {
    const int hh = i / C::VMAX, c = i - hh * C::VMAX;
    if (c >= V) continue;
    st_cluster(cluster_addr(merge + (sp * GP + hh) * C::VMAX + c, (c / 8) % S), block_sum_of(hh, c));
    if (c < S) st_cluster(cluster_addr(mm + (sp * GP + hh) * 2, c), common[hh * 2], common[(GP + hh) * 2]);
  }
  __syncwarp();
  cluster_barrier();
  if (tid < heads) {   // the splits' factors, in the place of their maxima
    float mt = -INFINITY, lt = 0.f;
    for (int r = 0; r < S; ++r) mt = fmaxf(mt, mm[(r * GP + tid) * 2]);
    for (int r = 0; r < S; ++r) {
      float* x = mm + (r * GP + tid) * 2;
      const float f = x[0] == -INFINITY ? 0.f : expf(x[0] - mt);
      lt = fmaf(x[1], f, lt);
      x[0] = f;
    }
    mm[tid * 2 + 1] = (lt > 0.f ? 1.f / lt : 0.f) * out_factor<T>(p, t, hb + tid);
  }
  __syncthreads();
  const int mine = (C::VMAX / 8 - sp + S - 1) / S * 8;   // this block's columns of a head
  for (int i = tid; i < heads * mine; i += kThreads) {
    const int hh = i / mine, j = i - hh * mine, c = ((j >> 3) * S + sp) * 8 + (j & 7);
    if (c >= V) continue;
    float a = 0.f;
    for (int r = 0; r < S; ++r) a = fmaf(merge[(r * GP + hh) * C::VMAX + c], mm[(r * GP + hh) * 2], a);
    stf(out_row<T>(p, t, hb + hh) + c, a * mm[hh * 2 + 1]);
  }
}

// *splits in: the most splits worth having (by the keys); out: the partial results left in the workspace, or 1
template <typename T, int LK, int LV, int GP>
int launch(const pcs_attn_params& p, int* splits_io, int per_group, cudaStream_t st) {
  using C = DecodeCfg<T, LK, LV, GP>;
  auto kernel = attn_group_decode_kernel<T, LK, LV, GP>;
  constexpr size_t full = static_cast<size_t>(C::kFloats + C::kMerge) * sizeof(float);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = full;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  struct Info { int room[kMaxCluster + 1]; };   // clusters of s blocks that run side by side
  static PerDevice<Info> per_device;
  const Info* info;
  if (int rc = per_device.get(&info, [&](Info& x) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(full));
        for (int s = 1; s <= kMaxCluster && err == cudaSuccess; ++s) {
          attr[0].val.clusterDim.x = s;
          cfg.gridDim = dim3(s);
          err = cudaOccupancyMaxActiveClusters(&x.room[s], kernel, &cfg);
        }
        return err;
      }))
    return rc;
  const int* room = info->room;
  // One wave: the largest cluster of which all fit side by side.  Few groups over many keys: more splits than a cluster has, through the workspace and a second
  // launch (6 us with the merge).  max_keys is what the pool holds and the sequence may be short, so neither end may lose much.  Over 50, 300, 1000, 4000, 8000 keys of a
  // pool of 8192, us: one token of 8 heads of 128 in a cluster 7, 8, 10, 19, 29, with 32 splits 13, 15, 15, 17, 19 (a block per head: 15, 17, 17, 17, 21); four tokens
  // 8, 8, 10, 19, 29 and, with 24 splits, 12, 15, 17, 19, 24 (13, 15, 15, 27, 43); eight tokens 8, 8, 10, 23, 38 and 12, 15, 17, 23, 28 (13, 15, 19, 41, 76).  A
  // key of a row over 32 lanes costs twice as much, so splits pay sooner; over 8 lanes half, and clusters win.
  const long long groups = static_cast<long long>(p.n_tokens) * p.n_kv_heads * per_group, all_heads = static_cast<long long>(p.n_tokens) * p.n_heads;
  int splits = *splits_io;
  bool cluster = true;
  const bool few = LK == 32   ? GP < 8 || all_heads <= 48 || p.max_keys > 4096
                   : LK == 16 ? all_heads <= 8 || p.max_keys > 8192 || (p.max_keys > 4096 && (all_heads <= 16 || all_heads >= 64))
                              : p.max_keys > 16384;
  if (few && p.max_keys >= (2 * kMaxCluster + 1) * 128 && groups * kMaxCluster * 2 <= room[1]) {
    const long long want = room[1] / groups;
    int wide = all_heads <= 8 ? 32 : 24;
    if (wide < p.max_keys / 341) wide = p.max_keys / 341;
    if (wide > p.max_keys / 128) wide = p.max_keys / 128;
    if (wide > want) wide = static_cast<int>(want);
    if (wide > kAttnMaxSplits) wide = kAttnMaxSplits;
    // (a workspace that holds only the fewer splits that pcs_attn asks for: a cluster, which needs none)
    if (p.workspace_floats >= static_cast<long long>(p.n_tokens) * p.n_heads * wide * (p.vdim + 2)) {
      cluster = false;
      splits = wide;
    }
  }
  if (cluster) {
    if (splits > kMaxCluster) splits = kMaxCluster;
    while (splits > 1 && room[splits] < groups) --splits;
    if (splits < 1) splits = 1;
    cluster = splits > 1;
  }
  *splits_io = cluster ? 1 : splits;
  cfg.gridDim = dim3(splits, p.n_kv_heads * per_group, p.n_tokens);
  cfg.dynamicSmemBytes = cluster ? full : static_cast<size_t>(C::kFloats) * sizeof(float);
  attr[0].val.clusterDim.x = cluster ? static_cast<unsigned>(splits) : 1u;
  PCS_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, per_group, cluster ? 1 : 0));
  count_launch();
  return PCS_OK;
}

template <typename T, int LK, int LV>
int launch_g(const pcs_attn_params& p, int gp, int* splits, int per_group, cudaStream_t st) {
  if (gp == 1) return launch<T, LK, LV, 1>(p, splits, per_group, st);
  if (gp == 2) return launch<T, LK, LV, 2>(p, splits, per_group, st);
  if (gp == 4) return launch<T, LK, LV, 4>(p, splits, per_group, st);
  return launch<T, LK, LV, 8>(p, splits, per_group, st);
}

template <typename T>
int launch_t(const pcs_attn_params& p, int gp, int* splits, int per_group, cudaStream_t st) {
  constexpr int N = Vec<T>::n;
  const int pk = (p.dim + N - 1) / N, pv = (p.vdim + N - 1) / N;
  if (pk <= 8 && pv <= 8) return launch_g<T, 8, 8>(p, gp, splits, per_group, st);
  if (pk <= 16 && pv <= 16) return launch_g<T, 16, 16>(p, gp, splits, per_group, st);
  if (pv <= 16) return launch_g<T, 32, 16>(p, gp, splits, per_group, st);
  return launch_g<T, 32, 32>(p, gp, splits, per_group, st);
}

}  // namespace

// *splits_out: 0 = not handled; 1 = done; more: that many partial results per (token, head) wait in the workspace.
// The caller has checked that rows are in 16-byte pieces.  Rows of up to four pieces would leave half of a row's eight lanes idle, rows of more than 32 do
// not fit a load: those stay with attn_decode_kernel.
int launch_attn_group_decode(const pcs_attn_params& p, cudaStream_t st, int* splits_out) {
  *splits_out = 0;
  const int N = p.dtype == PCS_BF16 ? 8 : 4, pieces = 32;
  if (p.dim <= 4 * N) return PCS_OK;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (p.dim > pieces * N || p.vdim > pieces * N || !al16(p.q) || !al16(p.k_pool) || !al16(p.v_pool) || p.n_tokens > 65535) return PCS_OK;
  const int G = p.n_heads / p.n_kv_heads, gp = G >= 8 ? 8 : G > 2 ? 4 << (G > 4) : G, per_group = (G + gp - 1) / gp;
  if (static_cast<long long>(p.n_kv_heads) * per_group > 65535) return PCS_OK;
  // Eight heads per block take a block 2 us longer to begin and to end than one head does: over 128 keys at most, and with 24 (token, head) pairs or fewer of narrow
  // bfloat16 rows, a block per head is the faster form (16 heads of 256 over one K/V head, 50 keys: 8.3 against 10.4 us; 20 heads of 128, one token, 300 and
  // 1000 keys of 8192: 14.5 and 14.5 against 16.5 and 17.5), and a split has 48 keys (300 keys of 20 heads of 128: 11.2 instead of 13.3 us; one head per block 12.4).
  if (gp == 8 && (p.max_keys <= 128 || (p.dtype == PCS_BF16 && p.dim <= 128 && p.vdim <= 128 && static_cast<long long>(p.n_tokens) * p.n_heads <= 24))) return PCS_OK;
  const int least = gp == 8 ? 48 : 128;
  int splits = p.max_keys > least ? p.max_keys / least : 1, rc;
  PCS_DISPATCH(p.dtype, rc = launch_t<T>(p, gp, &splits, per_group, st));
  if (rc) return rc;
  *splits_out = splits;
  return PCS_OK;
}

}  // namespace pcs
