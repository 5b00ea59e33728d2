// Attention over the slot pool for prompts in 32-bit (true 32-bit multiply-adds, no tensor cores).
//
// Bound by the 32-bit multiply-add rate.  One block = 32 consecutive new tokens of one sequence and head, 128 threads, keys in tiles of 64.  A thread holds a 4 x 4
// piece of the scores and 4 rows x vdim / 16 columns of the result; both operands of a product are read from shared memory in 16-byte
// pieces along the summed index (rows padded by 16 bytes: eight lanes read eight rows without a bank conflict), 64 multiply-adds per 8 reads, two per
// instruction.  K of the next tile travels (cp.async) while V is multiplied, V while the scores are formed.  Two blocks share an SM; the blocks
// with the most keys come first and every second group of 148 runs backwards, so that a long block is paired with a short one.
// Distance biases are evaluated once per distance and tile; expf, log1pf and tanhf as in the plain kernel.  A row whose result is not finite is formed again
// from the keys it sees alone (attn_row_again).
//
// 8 heads of 128 (B200), against the plain kernel (one block per token and head, every row read again): 1024 tokens 818 -> 103 us (21 TFLOP/s), 2048: 2.92 -> 0.32
// ms, 64 behind 400 stored 76 -> 21 us, 16 behind 4000 473 -> 68 us.  A cluster shares a walk where there are few blocks (choose_splits).
#include "seq_attn.cuh"
#include "seq_mma.cuh"
#include "seq_tc5.cuh"

namespace pcs {

namespace {

constexpr int FM = 32, FN = 64, F_THREADS = 128, FSMs = 148, kMaxSplits = 8;

__device__ __forceinline__ void fma_x2(float2& d, float2 a, float2 b) {
  asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nmov.b64 z, {%0, %1};\nfma.rn.f32x2 z, x, y, z;\nmov.b64 {%0, %1}, z;\n}\n"
      : "+f"(d.x), "+f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

// VP: value columns padded to 64 or 128
template <int VP>
__global__ void __launch_bounds__(F_THREADS) attn_f32_kernel(const __grid_constant__ pcs_attn_params p, const int splits) {
  constexpr int VC = VP / 64;              // 4-column pieces of a thread's result row
  extern __shared__ __align__(16) float sm[];
  const int D = p.dim, V = p.vdim, LD = D + 4;
  float* Qs = sm;                          // [32][LD]
  float* Ks = Qs + FM * LD;                // [64][LD]
  float* Vs = Ks + FN * LD;                // [64][VP]
  float* Ps = Vs + FN * VP;                // [32][68]
  float* Ts = Ps + FM * (FN + 4);          // [96] biases of the tile's distances
  constexpr int LP = FN + 4;
  const int n_tiles = (p.max_len + FM - 1) / FM, per_tile = p.n_seqs * p.n_heads;
  int idx = blockIdx.x / splits;
  const int rank = blockIdx.x - idx * splits;
  if (splits == 1) {
    const int wave = idx / FSMs, first = wave * FSMs, last = min(first + FSMs, static_cast<int>(gridDim.x)) - 1;
    if (wave & 1) idx = first + (last - idx);
  }
  const int qt = idx / per_tile, rem = idx - qt * per_tile, b = rem / p.n_heads, h = rem - b * p.n_heads, q0 = (n_tiles - 1 - qt) * FM;
  const int len = p.seq_len[b];
  if (q0 >= len) return;
  const int pos0 = p.seq_pos0[b], off = p.seq_off[b], slot = p.pool_slot ? p.pool_slot[b] : p.seq_slot[b];
  const int g = h / (p.n_heads / p.n_kv_heads), rows = min(FM, len - q0), first = pos0 + q0;
  const float* K = static_cast<const float*>(p.k_pool) + (static_cast<long long>(slot) * p.n_kv_heads + g) * p.cap * D;
  const float* Vg = static_cast<const float*>(p.v_pool) + (static_cast<long long>(slot) * p.n_kv_heads + g) * p.cap * V;
  const float* Q = static_cast<const float*>(p.q) + (static_cast<long long>(off + q0) * p.n_heads + h) * D;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int total = pos0 + len, n_keys = first + rows;
  const bool windowed = p.window > 0, chunked = p.chunk > 0;
  const int keep = windowed ? min(max(p.keep_first, 0), total) : 0;
  int lo = windowed ? max(0, first - p.window + 1) / FN : chunked ? first / p.chunk * p.chunk / FN : 0, nf = (keep + FN - 1) / FN;
  if (nf >= lo) nf = lo = 0;
  const int n_all = nf + (n_keys + FN - 1) / FN - lo, it0 = rank * n_all / splits, n_it = (rank + 1) * n_all / splits - it0;
  auto tile_of = [&](int it) { return it0 + it < nf ? it0 + it : lo + it0 + it - nf; };
  // rows of a [*, width] matrix into a padded tile; rows from `n` on are zero
  auto stage = [&](float* dst, int ld, const float* src, long long stride, int count, int n, int width) {
    const int ch = width / 4;
    for (int e = tid; e < count * ch; e += F_THREADS) {
      const int r = e / ch, c = (e - r * ch) * 4;
      if (r < n) cp_async16(dst + r * ld + c, src + r * stride + c);
      else *reinterpret_cast<float4*>(dst + r * ld + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  const float scale = p.scale * (p.head_scale ? p.head_scale[h] : 1.f);
  const float r1 = p.bias_r1 ? p.bias_r1[h] : 0.f, r2 = p.bias_r1 ? p.bias_r2[h] : 0.f;
  const float* tab = p.bias_table ? p.bias_table + static_cast<long long>(h) * p.bias_len : nullptr;
  const bool bias = p.bias_r1 || tab;
  float m[4], l[4];
  float2 o[4][VC][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = p.sink && rank == 0 ? (p.sink_logit ? p.sink_logit[h] : 0.f) : -INFINITY;
    l[i] = (p.sink && rank == 0 && tx == 0) ? 1.f : 0.f;   // the share of this thread's columns
#pragma unroll
    for (int c = 0; c < VC; ++c) o[i][c][0] = o[i][c][1] = make_float2(0.f, 0.f);
  }
  for (int e = tid; e < FN * VP; e += F_THREADS) Vs[e] = 0.f;   // columns past vdim stay zero
  __syncthreads();
  stage(Qs, LD, Q, static_cast<long long>(p.n_heads) * D, FM, rows, D);
  if (n_it > 0) {
    const int k0 = tile_of(0) * FN;
    stage(Ks, LD, K + static_cast<long long>(k0) * D, D, FN, total - k0, D);
  }
  cp_async_commit();
  for (int it = 0; it < n_it; ++it) {
    const int k0 = tile_of(it) * FN;
    stage(Vs, VP, Vg + static_cast<long long>(k0) * V, V, FN, total - k0, V);
    cp_async_commit();
    if (bias && tid < FM + FN - 1) {   // entry y: distance first - k0 + y - 63
      const int d = first - k0 + tid - (FN - 1);
      float v = 0.f;
      if (d >= 0) v = tab ? tab[min(d, p.bias_len - 1)] : -r1 * log1pf(r2 * static_cast<float>(d));
      Ts[tid] = v;
    }
    cp_async_wait<1>();
    __syncthreads();   // Q, this K tile and its biases
    // ---- scores of rows ty + 8 i, keys tx + 16 j ----
    float2 a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int d = 0; d < D; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(Qs + (ty + 8 * i) * LD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * LD + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma_x2(a[i][j], make_float2(qv[i].x, qv[i].y), make_float2(kv[j].x, kv[j].y));
          fma_x2(a[i][j], make_float2(qv[i].z, qv[i].w), make_float2(kv[j].z, kv[j].w));
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = ty + 8 * i, pos = first + row;
      const int lo_key = windowed ? max(0, pos - p.window + 1) : chunked ? pos / p.chunk * p.chunk : 0;
      float s[4], mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + tx + 16 * j;
        float z = (a[i][j].x + a[i][j].y) * scale;
        if (p.softcap > 0.f) z = p.softcap * tanhf(z / p.softcap);
        if (bias) z += Ts[row - (tx + 16 * j) + FN - 1];
        s[j] = (key <= pos && row < rows && (key >= lo_key || key < keep)) ? z : -INFINITY;
        mx = fmaxf(mx, s[j]);
      }
#pragma unroll
      for (int x = 8; x >= 1; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float mn = fmaxf(m[i], mx), f = m[i] == -INFINITY ? 0.f : expf(m[i] - mn), sub = mn == -INFINITY ? 0.f : mn;
      m[i] = mn;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float w = expf(s[j] - sub);
        sum += w;
        Ps[row * LP + tx + 16 * j] = w;
      }
      l[i] = fmaf(l[i], f, sum);
#pragma unroll
      for (int c = 0; c < VC; ++c)
#pragma unroll
        for (int u = 0; u < 2; ++u) { o[i][c][u].x *= f; o[i][c][u].y *= f; }
    }
    cp_async_wait<0>();
    __syncthreads();   // this V tile and every weight; K has been read
    if (it + 1 < n_it) {
      const int k1 = tile_of(it + 1) * FN;
      stage(Ks, LD, K + static_cast<long long>(k1) * D, D, FN, total - k1, D);
    }
    cp_async_commit();
    // ---- result rows ty + 8 i, columns 4 tx + 64 c ----
#pragma unroll 4
    for (int k = 0; k < FN; k += 4) {
      float4 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(Ps + (ty + 8 * i) * LP + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int c = 0; c < VC; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(Vs + (k + kk) * VP + c * 64 + tx * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float x = kk == 0 ? w[i].x : kk == 1 ? w[i].y : kk == 2 ? w[i].z : w[i].w;
            fma_x2(o[i][c][0], make_float2(x, x), make_float2(v.x, v.y));
            fma_x2(o[i][c][1], make_float2(x, x), make_float2(v.z, v.w));
          }
        }
    }
    __syncthreads();   // V, the weights and the biases may be written over
  }
  unsigned again = 0u;   // rows whose result is not finite, as far as this thread has seen it
  auto put = [&](int t, int row, int c, float4 x) {
    *reinterpret_cast<float4*>(out_row<float>(p, t, h) + c) = x;
    const float zero = fmaf(x.x, 0.f, x.y * 0.f) + fmaf(x.z, 0.f, x.w * 0.f);   // NaN where one of them is not finite
    if (zero != 0.f) again |= 1u << row;
  };
  if (splits > 1) {
    // A cluster shares the walk: block q owns the rows [q, q + 1) * 32 / splits, to which the others send their sums (over its V tile) and (m, l)
    const int mine = FM / splits;
    float* part = Vs;                     // [split][row of the slice][VP]
    float* ml = Ps;                       // [split][row of the slice][m, l]
    cp_async_wait<0>();
    __syncwarp();
    cluster_barrier();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int x = 8; x >= 1; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
      const int row = ty + 8 * i, q = row / mine, at = rank * mine + row - q * mine;
      if (tx == 0) st_cluster(cluster_addr(ml + at * 2, q), m[i], l[i]);
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        const uint32_t dst = cluster_addr(part + at * VP + c * 64 + tx * 4, q);
        st_cluster(dst, o[i][c][0].x, o[i][c][0].y);
        st_cluster(dst + 8, o[i][c][1].x, o[i][c][1].y);
      }
    }
    __syncwarp();
    cluster_barrier();
    for (int e = tid; e < mine * (VP / 4); e += F_THREADS) {
      const int r = e / (VP / 4), c = (e - r * (VP / 4)) * 4, row = rank * mine + r;
      if (row >= rows || c >= V) continue;
      float mt = -INFINITY, lt = 0.f;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int q = 0; q < splits; ++q) mt = fmaxf(mt, ml[(q * mine + r) * 2]);
      for (int q = 0; q < splits; ++q) {
        const float mq = ml[(q * mine + r) * 2], f = mq == -INFINITY ? 0.f : expf(mq - mt);
        const float4 x = *reinterpret_cast<const float4*>(part + (q * mine + r) * VP + c);
        lt = fmaf(ml[(q * mine + r) * 2 + 1], f, lt);
        a = make_float4(fmaf(x.x, f, a.x), fmaf(x.y, f, a.y), fmaf(x.z, f, a.z), fmaf(x.w, f, a.w));
      }
      const int t = off + q0 + row;
      const float inv = (lt > 0.f ? 1.f / lt : 0.f) * out_factor<float>(p, t, h);
      put(t, row, c, make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int x = 8; x >= 1; x >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);
      const int row = ty + 8 * i;
      if (row >= rows) continue;
      const int t = off + q0 + row;
      const float inv = (l[i] > 0.f ? 1.f / l[i] : 0.f) * out_factor<float>(p, t, h);
#pragma unroll
      for (int c = 0; c < VC; ++c)
        if (c * 64 + tx * 4 < V) put(t, row, c * 64 + tx * 4, make_float4(o[i][c][0].x * inv, o[i][c][0].y * inv, o[i][c][1].x * inv, o[i][c][1].y * inv));
    }
  }
  if (__syncthreads_or(again != 0u)) {
    unsigned* rows_again = reinterpret_cast<unsigned*>(Ts);
    if (tid == 0) *rows_again = 0u;
    __syncthreads();
    if (again) atomicOr(rows_again, again);
    __syncthreads();
    for (unsigned w = *rows_again, k = 0; w; w &= w - 1, ++k)
      if ((k & 3) == tid >> 5) attn_row_again<float>(p, b, h, off + q0 + __ffs(w) - 1, first + __ffs(w) - 1, 0, V);
  }
}

// The blocks of a cluster that share a walk: a key tile costs a block 7 us at dim + vdim = 256 whether it has its SM alone or not (its four warps wait for
// their own products), set-up and end 3, with a merge 6, 1 less where every block has an SM to itself (64 tokens behind 100, 4 heads of 36: a block per
// walk 17 us, four 11; with 16 entries, 512 blocks of four, 17 and 26); a launch of more than one wave ends 15 % behind its average.
int choose_splits(const pcs_attn_params& p, const int (&slots)[4]) {
  const double tile = 7.1 * (p.dim + p.vdim) / 256.0, over[4] = {3.0, 6.0, 6.5, 7.0};
  const int keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap, n = (p.max_len + FM - 1) / FM;
  const double blocks = fmin(static_cast<double>(p.n_seqs) * n, p.n_tokens / static_cast<double>(FM) + p.n_seqs) * p.n_heads;
  double sum = 0.0, longest = 0.0, best = 1e30;   // (longest: in tiles)
  for (int t = 0; t < n; ++t) {
    double k = fmax(fmin(keys, keys - p.max_len + (t + 1.0) * FM), 1.0);
    if (p.window > 0) k = fmin(k, p.window + FM + fmax(p.keep_first, 0) + FN);
    if (p.chunk > 0) k = fmin(k, p.chunk + FN);
    longest = fmax(longest, ceil(k / FN));
    sum += ceil(k / FN) * tile;
  }
  int splits = 1;
  for (int i = 0; i < 4; ++i) {
    const int s = 1 << i;
    if (slots[i] < s) continue;
    double t = ceil(longest / s) * tile + over[i] - (s > 1 && blocks * s <= FSMs);   // (a walk of one tile is not shared)
    if (blocks * s > slots[i]) t = fmax(t, 1.15 * (sum / n * blocks + blocks * s * over[i]) / slots[i]);
    if (t < best) { best = t; splits = s; }
  }
  return splits;
}

template <int VP>
int launch(const pcs_attn_params& p, unsigned grid, cudaStream_t st) {
  auto kernel = attn_f32_kernel<VP>;
  const size_t smem = (static_cast<size_t>(FM + FN) * (p.dim + 4) + FN * VP + FM * (FN + 4) + 96) * sizeof(float);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.blockDim = dim3(F_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  struct Info { int slots[2][4]; };   // blocks that run side by side in clusters of 2^i, at rows of up to 128 elements and of more
  static PerDevice<Info> per_device;
  const Info* info;
  if (int rc = per_device.get(&info, [&](Info& x) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        for (int w = 0; w < 2; ++w)
          for (int i = 0; i < 4 && err == cudaSuccess; ++i) {
            int n = 0;
            attr[0].val.clusterDim.x = 1u << i;
            cfg.gridDim = dim3(1u << i);
            cfg.dynamicSmemBytes = (static_cast<size_t>(FM + FN) * ((w ? 256 : 128) + 4) + FN * VP + FM * (FN + 4) + 96) * sizeof(float);
            err = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
            x.slots[w][i] = n << i;
          }
        return err;
      }))
    return rc;
  const int splits = choose_splits(p, info->slots[p.dim > 128]);
  cfg.gridDim = dim3(grid * splits);
  cfg.dynamicSmemBytes = smem;
  attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
  PCS_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, splits));
  count_launch();
  return PCS_OK;
}

}  // namespace

int launch_attn_f32(const pcs_attn_params& p, cudaStream_t st, bool* handled) {
  *handled = false;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (p.dtype != PCS_F32 || p.max_len < 16 || (p.v_row_stride != 0 && p.v_row_stride != p.vdim) || p.dim % 4 != 0 || p.vdim % 4 != 0 || p.dim > 256 || p.vdim > 128)
    return PCS_OK;
  if (!p.seq_pos0 || !p.seq_len || !p.seq_off || !al16(p.q) || !al16(p.k_pool) || !al16(p.v_pool) || !al16(p.out) || p.out_stride % 4 != 0) return PCS_OK;
  // Few tokens over few keys: a block per token and head begins and ends sooner.  Decoding kernels (a workspace is given) / plain kernel / tiles, B200, us: 16 tokens of 8
  // heads of 128 over 16 keys 6.5 / 10.5 / 12.6, over 66 8.3 / 14.5 / 16.5; 40 over 40 8.5 / 12.4 / 15.2; 24 x 4 entries over 24 - / 10.7 / 12.5, 24 over 72
  // - / 14.6 / 15.9, 16 x 16 entries over 16 - / 16.5 / 12.6; of 12 heads of 64: 16 over 16 - / 8.5 / 10.4, 48 over 48 - / 10.6 / 10.5.
  // (Rows of more than 128 are not the grouped decoding kernel's: 16 tokens over 1016 keys, 8 heads of 192, a block per head 45, tiles 27.)
  const int keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap;
  const long long pairs = static_cast<long long>(p.n_tokens) * p.n_heads;
  const bool workspace = p.workspace && p.workspace_floats >= pairs * kAttnMaxSplits * (p.vdim + 2);   // (the decoding kernels refuse one that is too small)
  if (workspace ? (p.n_tokens <= 16 && p.dim <= 128) || (static_cast<long long>(keys) * (p.dim + p.vdim) <= 49152 && pairs <= 1024)
                  : keys <= (p.dim + p.vdim >= 256 ? 80 : 32) && pairs <= 1024 && pairs * keys <= 32768)
    return PCS_OK;
  const long long grid = (p.max_len + FM - 1LL) / FM * p.n_seqs * p.n_heads;
  if (grid * kMaxSplits > 0x7fffffffLL) return PCS_OK;
  *handled = true;
  return p.vdim <= 64 ? launch<64>(p, static_cast<unsigned>(grid), st) : launch<128>(p, static_cast<unsigned>(grid), st);
}

}  // namespace pcs
