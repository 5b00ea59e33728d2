// The chunkwise matrix-memory recurrence (seq_mlstm_chunk.cu gives the formulas) with the chunks side by side.
//
// The serial form walks an entry's chunks one after the other in every column slice: 32 chunks of 64 tokens at ~9 us, four warps per SM, q k^T
// formed again in every slice.  Only the state has to be passed on, and that is an element-wise step, so:
//   gates   per (entry, head): every chunk's running sums and maxima, the stabiliser passed from chunk to chunk, the factors of every token
//   sums    per (chunk, head, 128 columns): U = k^T (v e^{a_s - g_e}), the chunk's own contribution, and its normaliser
//   scan    per element: S <- e^{m_in - g_e} S + U over the chunks in 32-bit; the state every chunk starts from replaces U, already as the
//           two bfloat16 operands hi + lo that the products read (the serial kernel formed the same pair)
//   out     per (chunk, head): (q k^T weights) v + q S, normaliser, the head's norm and the output gate; no raw result in memory
// Products are m16n8k16 bfloat16 with 32-bit accumulators; every 32-bit factor enters as hi + lo, as in the serial form.  Bound by the traffic of the
// states (written twice and read twice, 4 bytes an element; half of it stays in L2) and by the legacy tensor path in `out`.
//
// 2048 tokens, 4 heads of 256 x 512 (B200): 317 -> 123 us (gates 6, sums 26, scan 20, out 63); 3900 tokens, 2 heads of 128 x 256: 377 -> 66 us.  `out` with 256
// threads and operand loads directly before their products took 21 us more, with the index divisions of a run-time width 10 us more.
#include "seq_common.cuh"
#include "seq_mma.cuh"

namespace pcs {

namespace {

constexpr int CL = 64;      // tokens per chunk
constexpr int PT = 256;     // threads of a block of `sums` and `scan`
constexpr int OT = 512;     // and of `out`
constexpr int US = 128;     // columns of a block of `sums`
constexpr int UROW = US + 8, PROW = CL + 8;

// The scratch of one launch.  An entry's chunks are consecutive slots behind those of the entries before it (whatever the order of their rows); there are at
// most n_tokens / 64 + n_seqs of them.
struct Scratch {
  float *u, *n, *tok, *ce;   // [slot][head][dim * vdim], [slot][head][dim], [slot][head][5][64], [slot][head]
  int* first;                // [entry] its first slot
  __host__ __device__ Scratch(float* base, long long slots, int H, int D, int V) {
    u = base;
    n = u + slots * H * D * V;
    tok = n + slots * H * D;
    ce = tok + slots * H * 5 * CL;
    first = reinterpret_cast<int*>(ce + slots * H);
  }
};

// a chunk's running sums b and a_s = i_s - b_s, two tokens per lane, and the running maximum of a
struct ChunkGates {
  float b0, b1, a0, a1, cm;
  __device__ __forceinline__ ChunkGates(const pcs_mlstm_params& p, int off, int n, int head, int lane) {
    const int t = 2 * lane;
    const float f0 = t < n ? p.fg[static_cast<long long>(off + t) * p.heads + head] : 0.f, f1 = t + 1 < n ? p.fg[static_cast<long long>(off + t + 1) * p.heads + head] : 0.f;
    const float i0 = t < n ? p.ig[static_cast<long long>(off + t) * p.heads + head] : -INFINITY;
    const float i1 = t + 1 < n ? p.ig[static_cast<long long>(off + t + 1) * p.heads + head] : -INFINITY;
    float x = f0 + f1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    b1 = x;
    b0 = x - f1;
    a0 = i0 - b0;
    a1 = i1 - b1;
    cm = fmaxf(a0, a1);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, cm, o);
      if (lane >= o) cm = fmaxf(cm, y);
    }
  }
};

__global__ void __launch_bounds__(512) mlstm_par_gates_kernel(const pcs_mlstm_params p, float* scratch, long long slots) {
  extern __shared__ float sm[];   // per chunk: its last b, its largest a (then the stabiliser it starts from)
  const Scratch sc(scratch, slots, p.heads, p.dim, p.vdim);
  const int b = blockIdx.x, head = blockIdx.y, H = p.heads, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int len = p.seq_len[b], off = p.seq_off[b];
  if (len <= 0) return;
  const int nc = (len + CL - 1) / CL;
  int at0 = 0;   // the chunks of the entries before this one
  for (int i = lane; i < b; i += 32) at0 += (max(p.seq_len[i], 0) + CL - 1) / CL;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) at0 += __shfl_xor_sync(0xffffffffu, at0, o);
  if (head == 0 && threadIdx.x == 0) sc.first[b] = at0;
  float *be = sm, *am = sm + nc;
  float* mg = p.m_pool + static_cast<long long>(p.seq_slot[b]) * H + head;
  for (int c = warp; c < nc; c += nw) {
    const int n = min(CL, len - c * CL);
    const ChunkGates g(p, off + c * CL, n, head, lane);
    const float e = __shfl_sync(0xffffffffu, ((n - 1) & 1) ? g.b1 : g.b0, (n - 1) >> 1), a = __shfl_sync(0xffffffffu, g.cm, 31);
    if (lane == 0) { be[c] = e; am[c] = a; }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = p.seq_pos0[b] == 0 ? 0.f : *mg;
    for (int c = 0; c < nc; ++c) {
      const float next = be[c] + fmaxf(m, am[c]);
      am[c] = m;
      m = next;
    }
    *mg = m;
  }
  __syncthreads();
  for (int c = warp; c < nc; c += nw) {
    const int n = min(CL, len - c * CL), e = n - 1;
    const float m_in = am[c];
    const ChunkGates g(p, off + c * CL, n, head, lane);
    float before = __shfl_up_sync(0xffffffffu, g.cm, 1);
    if (lane == 0) before = -INFINITY;
    const float g0 = fmaxf(fmaxf(m_in, before), g.a0), g1 = fmaxf(g0, g.a1);
    const float ge = __shfl_sync(0xffffffffu, (e & 1) ? g1 : g0, e >> 1);
    const long long at = static_cast<long long>(at0 + c) * H + head;
    float2* t = reinterpret_cast<float2*>(sc.tok + at * 5 * CL) + lane;
    t[0] = make_float2(g.a0, g.a1);
    t[CL / 2] = make_float2(g0, g1);
    t[2 * CL / 2] = make_float2(expf(m_in - g0), expf(m_in - g1));
    t[3 * CL / 2] = make_float2(expf(-(g.b0 + g0)), expf(-(g.b1 + g1)));
    t[4 * CL / 2] = make_float2(expf(g.a0 - ge), expf(g.a1 - ge));   // tokens past the end: a = -inf, weight 0
    if (lane == 0) sc.ce[at] = expf(m_in - ge);
  }
}

__global__ void __launch_bounds__(PT) mlstm_par_sums_kernel(const pcs_mlstm_params p, float* scratch, long long slots) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int D = p.dim, V = p.vdim, H = p.heads, QROW = D + 8;
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [64][QROW]
  __nv_bfloat16* Vh = Ks + CL * QROW + 32;                          // [64][UROW] the weighted values, hi and lo
  __nv_bfloat16* Vl = Vh + CL * UROW;
  __shared__ float we[CL];
  const Scratch sc(scratch, slots, H, D, V);
  const int c = blockIdx.x, b = blockIdx.y / H, head = blockIdx.y - b * H, v0 = blockIdx.z * US;
  const int len = p.seq_len[b], i0 = c * CL;
  if (i0 >= len) return;
  const int n = min(CL, len - i0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3;
  const long long at = static_cast<long long>((b ? sc.first[b] : 0) + c) * H + head;
  const __nv_bfloat16* rows = static_cast<const __nv_bfloat16*>(p.proj) + static_cast<long long>(p.seq_off[b] + i0) * p.row_stride;
  const int pieces = D / 8;
  for (int e = tid; e < CL * pieces; e += PT) {
    const int r = e / pieces, k = (e - r * pieces) * 8;
    if (r < n) cp_async16(Ks + r * QROW + k, rows + r * p.row_stride + p.k_off + head * D + k);
    else *reinterpret_cast<uint4*>(Ks + r * QROW + k) = make_uint4(0u, 0u, 0u, 0u);
  }
  cp_async_commit();
  if (tid < CL) we[tid] = sc.tok[at * 5 * CL + 4 * CL + tid];
  uint4 vr[CL * US / 8 / PT];
#pragma unroll
  for (int u = 0; u < CL * US / 8 / PT; ++u) {
    const int e = tid + u * PT, r = e / (US / 8), k = (e - r * (US / 8)) * 8;
    vr[u] = make_uint4(0u, 0u, 0u, 0u);
    if (r < n && v0 + k < V) vr[u] = *reinterpret_cast<const uint4*>(rows + r * p.row_stride + p.v_off + head * V + v0 + k);
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < CL * US / 8 / PT; ++u) {
    const int e = tid + u * PT, r = e / (US / 8), k = (e - r * (US / 8)) * 8;
    float v[8];
    ld16(reinterpret_cast<const __nv_bfloat16*>(&vr[u]), v);
    const float w = we[r];
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = split_pair(v[2 * i] * w, v[2 * i + 1] * w, l[i]);
    *reinterpret_cast<uint4*>(Vh + r * UROW + k) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(Vl + r * UROW + k) = make_uint4(l[0], l[1], l[2], l[3]);
  }
  cp_async_wait<0>();
  __syncthreads();
  if (blockIdx.z == 0)
    for (int d = tid; d < D; d += PT) {
      float a = 0.f;
#pragma unroll 8
      for (int s = 0; s < CL; ++s) a = fmaf(we[s], ldf(Ks + s * QROW + d), a);
      sc.n[at * D + d] = a;
    }
  // U: 32 state rows x 64 columns per warp and turn
  const uint32_t kt_base = static_cast<uint32_t>(__cvta_generic_to_shared(Ks)) + (((lane & 7) + ((lane >> 4) & 1) * 8) * QROW + ((lane >> 3) & 1) * 8) * 2;
  const int bt = ((lane & 15) * UROW + (lane >> 4) * 8) * 2;
  const uint32_t vh_base = static_cast<uint32_t>(__cvta_generic_to_shared(Vh)) + bt, vl_base = static_cast<uint32_t>(__cvta_generic_to_shared(Vl)) + bt;
  float* U = sc.u + at * D * V;
  const int turns = (D + 31) / 32 * (US / 64);
  for (int w = warp; w < turns; w += PT / 32) {
    const int d0 = (w / (US / 64)) * 32, c0 = (w % (US / 64)) * 64;
    if (v0 + c0 >= V) continue;
    float acc[2][8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < CL / 16; ++ks) {
      uint32_t a[2][4], hf[4][4], lf[4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ldsm_x4_t(kt_base + (ks * 16 * QROW + d0 + i * 16) * 2, a[i][0], a[i][1], a[i][2], a[i][3]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ldsm_x4_t(vh_base + (ks * 16 * UROW + c0 + u * 16) * 2, hf[u][0], hf[u][1], hf[u][2], hf[u][3]);
        ldsm_x4_t(vl_base + (ks * 16 * UROW + c0 + u * 16) * 2, lf[u][0], lf[u][1], lf[u][2], lf[u][3]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          mma_bf16(acc[i][2 * u], a[i][0], a[i][1], a[i][2], a[i][3], hf[u][0], hf[u][1]);
          mma_bf16(acc[i][2 * u + 1], a[i][0], a[i][1], a[i][2], a[i][3], hf[u][2], hf[u][3]);
        }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          mma_bf16(acc[i][2 * u], a[i][0], a[i][1], a[i][2], a[i][3], lf[u][0], lf[u][1]);
          mma_bf16(acc[i][2 * u + 1], a[i][0], a[i][1], a[i][2], a[i][3], lf[u][2], lf[u][3]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int d = d0 + i * 16 + grp, col = v0 + c0 + j * 8 + qd * 2;
        if (col >= V) continue;   // vdim is a multiple of 8: both columns of the pair exist
        if (d < D) *reinterpret_cast<float2*>(U + static_cast<long long>(d) * V + col) = make_float2(acc[i][j][0], acc[i][j][1]);
        if (d + 8 < D) *reinterpret_cast<float2*>(U + static_cast<long long>(d + 8) * V + col) = make_float2(acc[i][j][2], acc[i][j][3]);
      }
  }
}

// eight neighbouring elements of a state per thread; the block behind the last one takes the normaliser
__global__ void __launch_bounds__(PT) mlstm_par_scan_kernel(const pcs_mlstm_params p, float* scratch, long long slots) {
  constexpr int AHEAD = 4;
  const int D = p.dim, V = p.vdim, H = p.heads, b = blockIdx.z, head = blockIdx.y;
  const Scratch sc(scratch, slots, H, D, V);
  const int len = p.seq_len[b];
  if (len <= 0) return;
  const int nc = (len + CL - 1) / CL;
  const bool fresh = p.seq_pos0[b] == 0;
  const long long at0 = static_cast<long long>(b ? sc.first[b] : 0) * H + head, pool = static_cast<long long>(p.seq_slot[b]) * H + head;
  if (blockIdx.x == gridDim.x - 1) {
    for (int d = threadIdx.x; d < D; d += PT) {
      float* ng = p.n_pool + pool * D + d;
      float x = fresh ? 0.f : *ng;
      for (int c = 0; c < nc; ++c) {
        float* u = sc.n + (at0 + static_cast<long long>(c) * H) * D + d;
        const float own = *u;
        *u = x;
        x = fmaf(x, sc.ce[at0 + static_cast<long long>(c) * H], own);
      }
      *ng = x;
    }
    return;
  }
  const long long e = (static_cast<long long>(blockIdx.x) * PT + threadIdx.x) * 8;
  if (e >= static_cast<long long>(D) * V) return;
  float* sg = p.s_pool + pool * D * V + e;
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = 0.f;
  if (!fresh) ldx(sg, s);
  const long long step = static_cast<long long>(H) * D * V;
  float* u = sc.u + at0 * D * V + e;
  float own[AHEAD][8], f[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < nc) {
      ldx(u + i * step, own[i]);
      f[i] = sc.ce[at0 + static_cast<long long>(i) * H];
    }
  for (int c0 = 0; c0 < nc; c0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int c = c0 + i;
      if (c < nc) {
        float x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = own[i][k];
        const float fc = f[i];
        if (c + AHEAD < nc) {
          ldx(u + (c + AHEAD) * step, own[i]);
          f[i] = sc.ce[at0 + static_cast<long long>(c + AHEAD) * H];
        }
        uint32_t h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = split_pair(s[2 * k], s[2 * k + 1], l[k]);
        uint4* d = reinterpret_cast<uint4*>(u + c * step);
        d[0] = make_uint4(h[0], h[1], h[2], h[3]);
        d[1] = make_uint4(l[0], l[1], l[2], l[3]);
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = fmaf(s[k], fc, x[k]);
      }
    }
  }
  stx(sg, s);
}

template <int VP>
struct OutCfg {
  static constexpr int SROW = VP + 8, kStages = 4, kStage = 2 * 16 * SROW;   // a stage: 16 state rows, hi and lo
  static constexpr int kRing = kStages * kStage > CL * SROW ? kStages * kStage : CL * SROW;  // the V tile lies over the ring
  static size_t smem(int D) { return (2 * static_cast<size_t>(CL) * (D + 8) + kRing + 2 * CL * PROW) * 2 + (4 * CL + 4 * CL + CL + 4 * CL) * 4; }
};

template <int VP>
__global__ void __launch_bounds__(OT, 1) mlstm_par_out_kernel(const pcs_mlstm_params p, float* scratch, long long slots) {
  using C = OutCfg<VP>;
  constexpr int SROW = C::SROW, NT = VP / 32, WC = VP / 4;   // a warp: 16 tokens x a quarter of the columns
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int D = p.dim, V = p.vdim, H = p.heads, QROW = D + 8;
  __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [64][QROW]
  __nv_bfloat16* Ks = Qs + CL * QROW;
  __nv_bfloat16* ring = Ks + CL * QROW;
  __nv_bfloat16* Ph = ring + C::kRing;                              // [64][PROW] the weights, hi and lo
  __nv_bfloat16* Pl = Ph + CL * PROW;
  float* tok = reinterpret_cast<float*>(Pl + CL * PROW);            // a, g, e^{m_in - g}, e^{-m}
  float* psum = tok + 4 * CL;                                       // [4][64] sums of the weights
  float* nq = psum + 4 * CL;                                        // [64] q . n of the state
  float* ss = nq + CL;                                              // [4][64] sums of squares
  const Scratch sc(scratch, slots, H, D, V);
  const int c = blockIdx.x, b = blockIdx.y / H, head = blockIdx.y - b * H;
  const int len = p.seq_len[b], i0 = c * CL;
  if (i0 >= len) return;
  const int n = min(CL, len - i0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3;
  const long long at = static_cast<long long>((b ? sc.first[b] : 0) + c) * H + head, t0 = p.seq_off[b] + i0;
  const __nv_bfloat16* rows = static_cast<const __nv_bfloat16*>(p.proj) + t0 * p.row_stride;
  const int pieces = D / 8, ksteps = D / 16, vp8 = V / 8;
  const float* S = sc.u + at * D * V;
  if (V < VP)
    for (int e = tid; e < C::kRing / 8; e += OT) reinterpret_cast<uint4*>(ring)[e] = make_uint4(0u, 0u, 0u, 0u);   // columns past vdim stay zero
  for (int e = tid; e < CL * pieces; e += OT) {
    const int r = e / pieces, k = (e - r * pieces) * 8;
    if (r < n) {
      cp_async16(Qs + r * QROW + k, rows + r * p.row_stride + p.q_off + head * D + k);
      cp_async16(Ks + r * QROW + k, rows + r * p.row_stride + p.k_off + head * D + k);
    } else {
      *reinterpret_cast<uint4*>(Qs + r * QROW + k) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(Ks + r * QROW + k) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  cp_async_commit();
  for (int e = tid; e < 4 * CL; e += OT) tok[e] = sc.tok[at * 5 * CL + e];
  __syncthreads();   // the ring is clear
  auto load_state = [&](int ks) {   // 16 rows of hi and lo pieces
    __nv_bfloat16* dst = ring + (ks % C::kStages) * C::kStage;
#pragma unroll
    for (int u = 0; u < (16 * VP / 8 + OT - 1) / OT; ++u) {
      const int e = tid + u * OT, r = e / (VP / 8), k = e % (VP / 8);
      if (r >= 16 || k >= vp8) continue;
      const float* src = S + static_cast<long long>(ks * 16 + r) * V + k * 8;
      cp_async16(dst + r * SROW + k * 8, src);
      cp_async16(dst + 16 * SROW + r * SROW + k * 8, src + 4);
    }
  };
  load_state(0);
  cp_async_commit();
  if (ksteps > 1) load_state(1);
  cp_async_commit();
  if (ksteps > 2) load_state(2);
  cp_async_commit();
  cp_async_wait<3>();
  __syncthreads();   // q and k
  // ---- weights e^{a_s - g_t} (q_t . k_s) / sqrt(dim), s <= t: 16 tokens x 16 keys per warp; q . n: 4 tokens per warp ----
  const int wr = (warp & 3) * 16, wc = (warp >> 2) * WC, ra = wr + grp, rb = ra + 8;
  const uint32_t q_base = static_cast<uint32_t>(__cvta_generic_to_shared(Qs)) + ((wr + (lane & 15)) * QROW + (lane >> 4) * 8) * 2;
  {
    const int k0 = (warp >> 2) * 16;
    const uint32_t k_base = static_cast<uint32_t>(__cvta_generic_to_shared(Ks)) + ((k0 + (lane & 7) + ((lane >> 4) & 1) * 8) * QROW + ((lane >> 3) & 1) * 8) * 2;
    float s[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < ksteps; ++kk) {
      uint32_t a0, a1, a2, a3, f[4];
      ldsm_x4(q_base + kk * 32, a0, a1, a2, a3);
      ldsm_x4(k_base + kk * 32, f[0], f[1], f[2], f[3]);
      mma_bf16(s[0], a0, a1, a2, a3, f[0], f[1]);
      mma_bf16(s[1], a0, a1, a2, a3, f[2], f[3]);
    }
    const float ga = tok[CL + ra], gb = tok[CL + rb];
    float sa = 0.f, sb = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int col = k0 + i * 8 + qd * 2;
      const float x0 = tok[col], x1 = tok[col + 1];
      s[i][0] = col <= ra ? s[i][0] * p.q_scale * __expf(x0 - ga) : 0.f;
      s[i][1] = col + 1 <= ra ? s[i][1] * p.q_scale * __expf(x1 - ga) : 0.f;
      s[i][2] = col <= rb ? s[i][2] * p.q_scale * __expf(x0 - gb) : 0.f;
      s[i][3] = col + 1 <= rb ? s[i][3] * p.q_scale * __expf(x1 - gb) : 0.f;
      sa += s[i][0] + s[i][1];
      sb += s[i][2] + s[i][3];
      uint32_t lo;
      uint32_t hi = split_pair(s[i][0], s[i][1], lo);
      *reinterpret_cast<uint32_t*>(Ph + ra * PROW + col) = hi;
      *reinterpret_cast<uint32_t*>(Pl + ra * PROW + col) = lo;
      hi = split_pair(s[i][2], s[i][3], lo);
      *reinterpret_cast<uint32_t*>(Ph + rb * PROW + col) = hi;
      *reinterpret_cast<uint32_t*>(Pl + rb * PROW + col) = lo;
    }
    sa += __shfl_xor_sync(0xffffffffu, sa, 1);
    sa += __shfl_xor_sync(0xffffffffu, sa, 2);
    sb += __shfl_xor_sync(0xffffffffu, sb, 1);
    sb += __shfl_xor_sync(0xffffffffu, sb, 2);
    if (qd == 0) { psum[(warp >> 2) * CL + ra] = sa; psum[(warp >> 2) * CL + rb] = sb; }
    const float* ns = sc.n + at * D;
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d = lane; d < D; d += 32) {
      const float x = ns[d];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = fmaf(x, ldf(Qs + (warp * 4 + i) * QROW + d), a[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = warp_sum(a[i]);
      if (lane == 0) nq[warp * 4 + i] = a[i] * p.q_scale * tok[2 * CL + warp * 4 + i];
    }
  }
  // ---- q S: 16 tokens x VP / 4 columns per warp, 16 state rows at a time; four operand loads ahead of their products ----
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  constexpr int UB = NT / 2 < 4 ? NT / 2 : 4;
  const uint32_t ring_base = static_cast<uint32_t>(__cvta_generic_to_shared(ring)) + ((lane & 15) * SROW + (lane >> 4) * 8 + wc) * 2;
  for (int ks = 0; ks < ksteps; ++ks) {
    cp_async_wait<2>();
    __syncthreads();   // these rows have landed, and every warp is done with the stage that is filled next
    if (ks + 3 < ksteps) load_state(ks + 3);
    cp_async_commit();
    uint32_t a0, a1, a2, a3;
    ldsm_x4(q_base + ks * 32, a0, a1, a2, a3);
    const uint32_t st = ring_base + (ks % C::kStages) * C::kStage * 2;
#pragma unroll
    for (int part = 0; part < 2; ++part)   // hi, then lo
#pragma unroll
      for (int u0 = 0; u0 < NT / 2; u0 += UB) {
        uint32_t f[UB][4];
#pragma unroll
        for (int u = 0; u < UB; ++u) ldsm_x4_t(st + (part * 16 * SROW + (u0 + u) * 16) * 2, f[u][0], f[u][1], f[u][2], f[u][3]);
#pragma unroll
        for (int u = 0; u < UB; ++u) {
          mma_bf16(acc[2 * (u0 + u)], a0, a1, a2, a3, f[u][0], f[u][1]);
          mma_bf16(acc[2 * (u0 + u) + 1], a0, a1, a2, a3, f[u][2], f[u][3]);
        }
      }
  }
  __syncthreads();   // the ring is free: the values go there
#pragma unroll
  for (int u = 0; u < CL * VP / 8 / OT; ++u) {
    const int e = tid + u * OT, r = e / (VP / 8), k = e % (VP / 8) * 8;
    if (r < n && k < V) cp_async16(ring + r * SROW + k, rows + r * p.row_stride + p.v_off + head * V + k);
    else *reinterpret_cast<uint4*>(ring + r * SROW + k) = make_uint4(0u, 0u, 0u, 0u);
  }
  cp_async_commit();
  {
    const float ca = tok[2 * CL + ra] * p.q_scale, cb = tok[2 * CL + rb] * p.q_scale;
#pragma unroll
    for (int j = 0; j < NT; ++j) { acc[j][0] *= ca; acc[j][1] *= ca; acc[j][2] *= cb; acc[j][3] *= cb; }
  }
  // what the epilogue reads is requested before the last products
  const __nv_bfloat16* nw = static_cast<const __nv_bfloat16*>(p.norm_w) + head * V;
  uint32_t gate[2][NT];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int r = ra + 8 * i, col = wc + j * 8 + qd * 2;
      gate[i][j] = (r < n && col < V) ? *reinterpret_cast<const uint32_t*>(rows + r * p.row_stride + p.g_off + head * V + col) : 0u;
    }
  cp_async_wait<0>();
  __syncthreads();
  // ---- + weights x values ----
  {
    const uint32_t ph = static_cast<uint32_t>(__cvta_generic_to_shared(Ph)) + ((wr + (lane & 15)) * PROW + (lane >> 4) * 8) * 2;
    const uint32_t pl = static_cast<uint32_t>(__cvta_generic_to_shared(Pl)) + ((wr + (lane & 15)) * PROW + (lane >> 4) * 8) * 2;
#pragma unroll
    for (int ks = 0; ks < CL / 16; ++ks) {
      if (ks * 16 > wr) break;   // keys behind all of this warp's tokens
      uint32_t h[4], l[4];
      ldsm_x4(ph + ks * 32, h[0], h[1], h[2], h[3]);
      ldsm_x4(pl + ks * 32, l[0], l[1], l[2], l[3]);
#pragma unroll
      for (int u0 = 0; u0 < NT / 2; u0 += UB) {
        uint32_t f[UB][4];
#pragma unroll
        for (int u = 0; u < UB; ++u) ldsm_x4_t(ring_base + (ks * 16 * SROW + (u0 + u) * 16) * 2, f[u][0], f[u][1], f[u][2], f[u][3]);
#pragma unroll
        for (int u = 0; u < UB; ++u) {
          mma_bf16(acc[2 * (u0 + u)], h[0], h[1], h[2], h[3], f[u][0], f[u][1]);
          mma_bf16(acc[2 * (u0 + u) + 1], h[0], h[1], h[2], h[3], f[u][2], f[u][3]);
        }
#pragma unroll
        for (int u = 0; u < UB; ++u) {
          mma_bf16(acc[2 * (u0 + u)], l[0], l[1], l[2], l[3], f[u][0], f[u][1]);
          mma_bf16(acc[2 * (u0 + u) + 1], l[0], l[1], l[2], l[3], f[u][2], f[u][3]);
        }
      }
    }
  }
  // ---- normaliser, the head's norm, the output gate ----
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = ra + 8 * i;
    const float den = 1.f / (fmaxf(fabsf(nq[r] + (psum[r] + psum[CL + r]) + (psum[2 * CL + r] + psum[3 * CL + r])), tok[3 * CL + r]) + 1e-6f);
    float x = 0.f;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float &y0 = acc[j][i * 2], &y1 = acc[j][i * 2 + 1];
      y0 *= den;
      y1 *= den;
      x = fmaf(y0, y0, fmaf(y1, y1, x));
    }
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    if (qd == 0) ss[(warp >> 2) * CL + r] = x;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = ra + 8 * i;
    if (r >= n) continue;
    const float inv = 1.f / sqrtf((ss[r] + ss[CL + r] + ss[2 * CL + r] + ss[3 * CL + r]) / static_cast<float>(V) + p.eps);
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + (t0 + r) * (static_cast<long long>(H) * V) + head * V;
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int col = wc + j * 8 + qd * 2;
      if (col >= V) continue;
      const float2 w2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(nw + col)), g2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[i][j]));
      *reinterpret_cast<uint32_t*>(o + col) = pack_bf16(acc[j][i * 2] * inv * w2.x * sigmoidf_(g2.x), acc[j][i * 2 + 1] * inv * w2.y * sigmoidf_(g2.y));
    }
  }
}

template <int VP>
int launch_out(const pcs_mlstm_params& p, float* scratch, long long slots, dim3 grid, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    PCS_CHECK_CUDA(cudaFuncSetAttribute(mlstm_par_out_kernel<VP>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(OutCfg<VP>::smem(256))));
    configured = true;
  }
  mlstm_par_out_kernel<VP><<<grid, OT, OutCfg<VP>::smem(p.dim), st>>>(p, scratch, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  return PCS_OK;
}

}  // namespace

long long mlstm_par_floats(int n_tokens, int n_seqs, int heads, int dim, int vdim) {
  const long long slots = n_tokens / CL + n_seqs;
  return slots * heads * (static_cast<long long>(dim) * vdim + dim + 5 * CL + 1) + n_seqs;
}

// The caller has checked type, alignment and dim (a multiple of 16, at most 256).  Four launches against one walk and two: fewer than four chunks (eight where
// a head has more than 256 columns, whose last kernel alone takes 40 us) stay with the serial form.  Serial / side by side, B200, us: 100 tokens of 2 heads 64 x 128
// 22 / 32, 200 tokens of 2 heads 128 x 256 37 / 35, 128 tokens of a head 256 x 512 31 / 72, 700 tokens of 8 heads 256 x 512 218 / 107.
bool mlstm_par_serves(const pcs_mlstm_params& p) {
  auto al4 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 3) == 0; };
  return p.vdim <= 512 && p.max_len > CL * (p.vdim > 256 ? 7 : 3) && p.g_off % 2 == 0 && al4(p.norm_w) && al4(p.out) &&
         (reinterpret_cast<uintptr_t>(p.s_pool) & 15) == 0 && static_cast<long long>(p.n_seqs) * p.heads <= 65535 && (p.max_len + CL - 1) / CL <= 5000;
}

int launch_mlstm_par(const pcs_mlstm_params& p, cudaStream_t st, bool* handled) {
  *handled = false;
  if (!p.chunk_scratch || !mlstm_par_serves(p) || (reinterpret_cast<uintptr_t>(p.chunk_scratch) & 15) != 0 ||
      p.chunk_floats < mlstm_par_floats(p.n_tokens, p.n_seqs, p.heads, p.dim, p.vdim))
    return PCS_OK;
  const long long slots = p.n_tokens / CL + p.n_seqs;
  const int chunks = (p.max_len + CL - 1) / CL;
  *handled = true;
  float* s = p.chunk_scratch;
  mlstm_par_gates_kernel<<<dim3(p.n_seqs, p.heads), 512, 2 * chunks * sizeof(float), st>>>(p, s, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  static bool configured = false;
  auto sums_smem = [](int D) { return (static_cast<size_t>(CL) * (D + 8) + 32 + 2 * CL * UROW) * 2; };
  if (!configured) {
    PCS_CHECK_CUDA(cudaFuncSetAttribute(mlstm_par_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sums_smem(256))));
    configured = true;
  }
  mlstm_par_sums_kernel<<<dim3(chunks, p.n_seqs * p.heads, (p.vdim + US - 1) / US), PT, sums_smem(p.dim), st>>>(p, s, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  const int groups = p.dim * p.vdim / 8;
  mlstm_par_scan_kernel<<<dim3((groups + PT - 1) / PT + 1, p.heads, p.n_seqs), PT, 0, st>>>(p, s, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  const dim3 grid(chunks, p.n_seqs * p.heads);
  int rc = p.vdim <= 128 ? launch_out<128>(p, s, slots, grid, st) : p.vdim <= 256 ? launch_out<256>(p, s, slots, grid, st) : launch_out<512>(p, s, slots, grid, st);
  if (rc) return rc;
  count_launch(4);
  return PCS_OK;
}

}  // namespace pcs

PCS_API int64_t pcs_mlstm_scratch_floats(int n_tokens, int n_seqs, int heads, int dim, int vdim) {
  if (n_tokens <= 0 || n_seqs <= 0 || heads <= 0 || dim <= 0 || vdim <= 0) return 0;
  return pcs::mlstm_par_floats(n_tokens, n_seqs, heads, dim, vdim);
}
