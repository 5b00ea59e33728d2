// The chunkwise matrix-memory recurrence (seq_mlstm_chunk.cu gives the formulas) with the chunks side by side.
//
// The serial form walks an entry's chunks one after the other in every column slice: 32 chunks of 64 tokens at ~9 us, four warps per SM, q k^T
// formed again in every slice.  Only the state has to be passed on, so:
//   gates   per (entry, head): every chunk's running sums and maxima, the stabiliser passed from chunk to chunk, the factors of every token
//   state   per (entry, head, 64 x 64 of the state): the walk over the chunks in 32-bit, S <- e^{m_in - g_e} S + k^T (v e^{a_s - g_e}); the state every chunk starts from goes to
//           the scratch as the two bfloat16 operands hi + lo that the products read (the serial kernel formed the same pair)
//   out     per (chunk, head): (q k^T weights) v + q S, normaliser, the head's norm and the output gate; no raw result in memory
// Products are m16n8k16 bfloat16 with 32-bit accumulators; every 32-bit factor enters as hi + lo, as in the serial form.  Bound by the latency of a chunk's step in `state`
// (1450 cycles, 530 of them products) and by the traffic of the states in `out` (4 bytes an element, written and read once).
//
// 2048 tokens, 4 heads of 256 x 512 (B200): serial 317 us; 122 with the chunks' own sums, a scan over them and operand loads shared by a block (gates 6, sums 26, scan 20, out 63);
// 76 in this form (gates 6, state 32, out 34).  40 drawn calls of 150 to 4100 tokens: none more than 2 % slower than with those sums and that scan, 1.15 times as fast in the mean.
#include "seq_common.cuh"
#include "seq_mma.cuh"

namespace pcs {

namespace {

constexpr int CL = 64;      // tokens per chunk
constexpr int PROW = CL + 8;

// The scratch of one launch.  An entry's chunks are consecutive slots behind those of the entries before it (whatever the order of their rows); there are at
// most n_tokens / 64 + n_seqs of them.  A walk in segments has more behind these: what the segments add up to.
struct Scratch {
  float *u, *n, *tok, *ce, *left, *left_n;   // [slot][head][dim * vdim], [slot][head][dim], [slot][head][5][64], [slot][head], [entry][segment][head][tile][64 * 64],
                                             // [entry][segment][head][dim]
  int* first;                                // [entry] its first slot
  static constexpr int kLeft = 148 * 64 * 64, kLeftN = 148 * 64;   // (at most 148 tiles of all segments, each of which has at most 64 rows)
  // floats up to `left`, which begins on 16 bytes as the scratch does
  static __host__ __device__ long long whole(long long slots, int n_seqs, int H, int D, int V) {
    return (slots * H * (static_cast<long long>(D) * V + D + 5 * CL + 1) + n_seqs + 3) / 4 * 4;
  }
  __host__ __device__ Scratch(float* base, long long slots, const pcs_mlstm_params& p) {
    const int H = p.heads, D = p.dim, V = p.vdim;
    u = base;
    n = u + slots * H * D * V;
    tok = n + slots * H * D;
    ce = tok + slots * H * 5 * CL;
    first = reinterpret_cast<int*>(ce + slots * H);
    left = base + whole(slots, p.n_seqs, H, D, V);
    left_n = left + kLeft;
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
  const Scratch sc(scratch, slots, p);
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

// Block = 64 state rows x 64 columns of one (entry, head), the chunks in order.  Per chunk the state it starts from leaves as hi + lo,
// U = k^T (v e^{a_s - g_e}) for the tile, S <- e^{m_in - g_e} S + U.  The chunks' own sums never pass through memory; k and v are read again by every tile (16 KB a chunk, from L2).
// Four warps, one per scheduler, hold 16 columns x 64 rows each and form U transposed, (v w)^T k: a lane's numbers are then pairs of neighbouring
// rows at one column, which, rounded, are the operand fragments of q S.  The states lie in the scratch as those fragments: [dim / 16][vdim / 8][lane] 16 bytes, rows 2t, 2t + 1 and
// 2t + 8, 2t + 9 of column g as hi, then as lo, so that a fragment is written and read by one 16-byte access a lane.  The values are weighed and split in registers, by the only warp that uses them.
// Four other warps keep the loads four chunks ahead, and CHAIN of them sum the normaliser, token by token: a warp takes 64 / CHAIN tokens of a chunk and goes on from where the warp before it
// ended, a step earlier, so the last one is CHAIN - 1 chunks behind.  One barrier per chunk.  us a call with chains of 1 / 2 / 4: 32 chunks of 4 heads of 256 x 512 80.0 / 77.7 / 76.6, 20 of 4 of 128 x 256
// in segments 36.9 / 36.1 / 36.7, 7 of 4 of 128 x 128 24.5 / 23.8 / 24.3: four from 24 chunks in one walk on, two elsewhere.  (Four sums of sixteen tokens added at the end: 0 to 2 % faster, other bits.)
// 32 chunks of 4 heads of 256 x 512: 46 us as sums of the chunks and an element-wise scan over them, 32 in this form; the products alone take 9.  What a step waits for is the
// one warp per scheduler: with eight warps that multiply (each weighing for itself) it took 38 us, with the values weighed by the helpers 34 to 40.
constexpr int kSTHalf = 128, kST = 2 * kSTHalf, kSAhead = 4, kSRow = 72, kSTile = CL * kSRow;

// Few tiles leave most of the GPU idle over a long walk: it is then cut into `segs` segments side by side.  A first launch (SUMS) walks all but the last without
// writing states and leaves what they add up to; in the second a segment starts from those before it.  Twice the products, 1 / segs of the steps.
constexpr int kMaxTiles = 148, kTileFloats = 64 * 64;   // segments of all tiles are at most one per SM

template <int CHAIN>
constexpr int kStateSmem = (kSAhead + CHAIN) * (2 * kSTile * 2 + CL * 4) + (CHAIN - 1) * 2 * 64 * 4;

template <bool SUMS, int CHAIN>
__global__ void __launch_bounds__(kST) mlstm_par_state_kernel(const pcs_mlstm_params p, float* scratch, long long slots, int segs) {
  constexpr int kSStages = kSAhead + CHAIN;
  static_assert(CL % CHAIN == 0 && CHAIN <= 4, "equal parts of a chunk's tokens");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [stages][64][72]
  __nv_bfloat16* Vs = Ks + kSStages * kSTile;
  float* we = reinterpret_cast<float*>(Vs + kSStages * kSTile);     // [stages][64]
  float* carry = we + kSStages * CL;                                // [chain - 1][2][64] sums of k over the first tokens of a chunk
  const int D = p.dim, V = p.vdim, H = p.heads, b = blockIdx.z / segs, seg = blockIdx.z % segs, head = blockIdx.y, vtiles = (V + 63) / 64;
  const int d0 = static_cast<int>(blockIdx.x) / vtiles * 64, v0 = static_cast<int>(blockIdx.x) % vtiles * 64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3;
  const Scratch sc(scratch, slots, p);
  const int all = p.seq_len[b];
  if (all <= 0) return;
  const int per = ((all + CL - 1) / CL + segs - 1) / segs, c_lo = seg * per, len = min(all - c_lo * CL, per * CL);   // this segment's chunks and tokens
  const bool last = c_lo * CL + len >= all;
  if (len <= 0 || (SUMS && last)) return;
  const int nc = (len + CL - 1) / CL, off = p.seq_off[b] + c_lo * CL;
  const bool fresh = p.seq_pos0[b] == 0;
  const long long entry0 = static_cast<long long>(b ? sc.first[b] : 0) * H + head, at0 = entry0 + static_cast<long long>(c_lo) * H;
  const long long pool = static_cast<long long>(p.seq_slot[b]) * H + head;
  // where the entry's segments leave their sums; the last one's place holds the state that the entry starts from (its own is not there any more once the last segment has ended)
  const long long left0 = (static_cast<long long>(b) * segs) * H + head;
  auto left = [&](int j) { return sc.left + ((left0 + static_cast<long long>(j) * H) * gridDim.x + blockIdx.x) * kTileFloats + (tid & (kSTHalf - 1)) * 4; };
  auto left_n = [&](int j) { return sc.left_n + (left0 + static_cast<long long>(j) * H) * D + d0; };
  auto factor = [&](int j) {   // of segment j
    float f = 1.f;
#pragma unroll 4
    for (int i = 0; i < per; ++i) f *= sc.ce[entry0 + static_cast<long long>(j * per + i) * H];
    return f;
  };
  const bool from_pool = SUMS ? seg == 0 : seg == 0 && last;
  if (tid >= kSTHalf) {
    const int ht = tid - kSTHalf, hw = ht >> 5, lr = ht >> 3, lk = (ht & 7) * 8;   // this thread's piece of every sixteenth row
    const bool k_in = d0 + lk < D, v_in = v0 + lk < V, sums = v0 == 0;
    const long long rs = p.row_stride;
    const __nv_bfloat16* kg = static_cast<const __nv_bfloat16*>(p.proj) + (static_cast<long long>(off) + lr) * rs + p.k_off + head * D + d0 + lk;
    const long long rs16 = 16 * rs;
    const float* tg = sc.tok + at0 * 5 * CL + 4 * CL + ht * 4;
    const __nv_bfloat16 *next = kg, *next_v = kg + ((p.v_off + head * V + v0) - (p.k_off + head * D + d0));   // chunk `loaded`'s pieces
    int loaded = 0, stage = 0;
    auto load = [&]() {
      if (loaded < nc) {
        __nv_bfloat16 *kd = Ks + stage * kSTile + lr * kSRow + lk, *vd = kd + kSStages * kSTile;
        const int left = len - loaded * CL - lr;
        if (k_in && v_in && left > CL - 16) {   // (few instructions: one warp per scheduler does this, and the products wait for it)
#pragma unroll
          for (int u = 0; u < CL / 16; ++u) cp_async16(kd + 16 * u * kSRow, next + u * rs16);
#pragma unroll
          for (int u = 0; u < CL / 16; ++u) cp_async16(vd + 16 * u * kSRow, next_v + u * rs16);
        } else {
#pragma unroll 1
          for (int u = 0; u < CL / 16; ++u) {
            if (16 * u < left && k_in) cp_async16(kd + 16 * u * kSRow, next + u * rs16);
            else *reinterpret_cast<uint4*>(kd + 16 * u * kSRow) = make_uint4(0u, 0u, 0u, 0u);
            if (16 * u < left && v_in) cp_async16(vd + 16 * u * kSRow, next_v + u * rs16);
            else *reinterpret_cast<uint4*>(vd + 16 * u * kSRow) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        if (ht < CL / 4) cp_async16(we + stage * CL + ht * 4, tg + static_cast<long long>(loaded) * H * 5 * CL);
        next += CL * rs;
        next_v += CL * rs;
        ++loaded;
        stage = stage + 1 == kSStages ? 0 : stage + 1;
      }
      cp_async_commit();
    };
#pragma unroll 1
    for (int c = 0; c < kSAhead; ++c) load();
    const int row = 2 * lane;   // and the next
    const bool of_n = sums && hw == CHAIN - 1 && d0 + row < D;
    float ns[2] = {0.f, 0.f}, fc = sums ? sc.ce[at0] : 0.f;
    if (of_n) {
      if (from_pool && !fresh) {
        ns[0] = p.n_pool[pool * D + d0 + row];
        ns[1] = p.n_pool[pool * D + d0 + row + 1];
      }
      if (SUMS) {
        if (seg == 0) *reinterpret_cast<float2*>(left_n(segs - 1) + row) = make_float2(ns[0], ns[1]);
      } else if (!from_pool) {
        for (int j = 0; j == 0 || j < seg; ++j) {
          const float f = j ? factor(j) : 0.f;
          const float2 x = *reinterpret_cast<const float2*>(left_n(seg ? j : segs - 1) + row);
          ns[0] = fmaf(ns[0], f, x.x);
          ns[1] = fmaf(ns[1], f, x.y);
        }
      }
    }
    const int steps = sums ? nc + CHAIN - 1 : nc;
    for (int c = 0; c < steps; ++c) {
      if (c < nc) {
        cp_async_wait<kSAhead - 1>();
        __syncthreads();   // chunk c has landed; what the chunk before the last one that is summed lay in is free
        load();
      } else {
        asm volatile("bar.sync 1, 128;" ::: "memory");   // (these warps alone)
      }
      const int ch = c - hw, st = ch % kSStages;
      if (!sums || hw >= CHAIN || ch < 0 || ch >= nc) continue;
      float2 x = make_float2(0.f, 0.f);
      if (hw) x = *reinterpret_cast<const float2*>(carry + ((hw - 1) * 2 + ((c - 1) & 1)) * 64 + row);
      const __nv_bfloat16* k = Ks + st * kSTile + hw * (CL / CHAIN) * kSRow + row;
      const float* w = we + st * CL + hw * (CL / CHAIN);
#pragma unroll
      for (int t = 0; t < CL / CHAIN; ++t) {
        const uint32_t kk = *reinterpret_cast<const uint32_t*>(k + t * kSRow);
        x.x = fmaf(w[t], __uint_as_float(kk << 16), x.x);
        x.y = fmaf(w[t], __uint_as_float(kk & 0xffff0000u), x.y);
      }
      if (hw < CHAIN - 1) {
        *reinterpret_cast<float2*>(carry + (hw * 2 + (c & 1)) * 64 + row) = x;
      } else {
        if (of_n && !SUMS) *reinterpret_cast<float2*>(sc.n + (at0 + static_cast<long long>(ch) * H) * D + d0 + row) = make_float2(ns[0], ns[1]);
        ns[0] = fmaf(ns[0], fc, x.x);
        ns[1] = fmaf(ns[1], fc, x.y);
        if (ch + 1 < nc) fc = sc.ce[at0 + static_cast<long long>(ch + 1) * H];
      }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      if (of_n && SUMS) left_n(seg)[row + x] = ns[x];
      if (of_n && !SUMS && last) p.n_pool[pool * D + d0 + row + x] = ns[x];
    }
    return;
  }
  // this lane's state: columns vr and vr + 8, rows d0 + 8 j + 2 qd and the next
  const int vr = v0 + warp * 16 + grp;
  float s[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int d = d0 + 8 * j + 2 * qd + (x & 1), v = vr + 8 * (x >> 1);
      s[j][x] = from_pool && !fresh && d < D && v < V ? p.s_pool[(pool * D + d) * V + v] : 0.f;
    }
  if (SUMS) {
    if (seg == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(left(segs - 1) + j * 512) = make_float4(s[j][0], s[j][1], s[j][2], s[j][3]);
    }
  } else if (!from_pool) {
    // (the next segment's numbers are under way while those before it are added)
    float4 x[8];
    auto fetch = [&](int i) {
      const float* l = left(seg ? i : segs - 1);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = *reinterpret_cast<const float4*>(l + j * 512);
    };
    fetch(0);
#pragma unroll
    for (int j = 0; j < 8; ++j) { s[j][0] = x[j].x; s[j][1] = x[j].y; s[j][2] = x[j].z; s[j][3] = x[j].w; }
    if (seg > 1) {
      float f = factor(1);
      fetch(1);
#pragma unroll 1
      for (int i = 1; i < seg; ++i) {
        const float now = f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s[j][0] = fmaf(s[j][0], now, x[j].x);
          s[j][1] = fmaf(s[j][1], now, x[j].y);
          s[j][2] = fmaf(s[j][2], now, x[j].z);
          s[j][3] = fmaf(s[j][3], now, x[j].w);
        }
        if (i + 1 < seg) {
          fetch(i + 1);
          f = factor(i + 1);
        }
      }
    }
  }
  float fc = sc.ce[at0];
  // operands of sixteen tokens: the warp's 16 columns of v (transposed reads of rows of tokens), 64 rows of the state
  const uint32_t v_base = static_cast<uint32_t>(__cvta_generic_to_shared(Vs + ((lane & 7) + ((lane >> 4) & 1) * 8) * kSRow + ((lane >> 3) & 1) * 8 + warp * 16));
  const uint32_t k_base = static_cast<uint32_t>(__cvta_generic_to_shared(Ks + (lane & 15) * kSRow + (lane >> 4) * 8));
  uint4* U = reinterpret_cast<uint4*>(sc.u + at0 * D * V) + (static_cast<long long>(d0 / 16) * (V / 8) + v0 / 8 + warp * 2) * 32 + lane;
  const long long step = static_cast<long long>(H) * D * V / 4;
  const int to_next = V / 8 * 32;   // sixteen rows on
#pragma unroll 1
  for (int c = 0, st = 0; c < nc; ++c, U += step) {
    const float f = fc;
    if (c + 1 < nc) fc = sc.ce[at0 + static_cast<long long>(c + 1) * H];
    __syncthreads();   // chunk c stands
    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const uint32_t va = v_base + st * kSTile * 2, ka = k_base + st * kSTile * 2;
    const float* w = we + st * CL + 2 * qd;
    uint32_t a[4], k[2][4][4], h[2][4], l[2][4];
    float2 w0, w1;
    auto fetch = [&](int ks, int x) {
      ldsm_x4_t(va + ks * 16 * kSRow * 2, a[0], a[1], a[2], a[3]);
      w0 = *reinterpret_cast<const float2*>(w + 16 * ks);
      w1 = *reinterpret_cast<const float2*>(w + 16 * ks + 8);
#pragma unroll
      for (int u = 0; u < 4; ++u) ldsm_x4_t(ka + (ks * 16 * kSRow + u * 16) * 2, k[x][u][0], k[x][u][1], k[x][u][2], k[x][u][3]);
    };
    auto weigh = [&](int x) {   // registers 0, 1: tokens 2 qd, 2 qd + 1 of columns grp, grp + 8; 2, 3: tokens 8 on
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 ww = i < 2 ? w0 : w1;
        h[x][i] = split_pair(__uint_as_float(a[i] << 16) * ww.x, __uint_as_float(a[i] & 0xffff0000u) * ww.y, l[x][i]);
      }
    };
    // a quarter of the state this chunk starts from: sixteen rows, both groups of eight columns
    auto leave = [&](int ks) {
      if (!SUMS && d0 + 16 * ks < D) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          uint4 o;
          o.x = split_pair(s[2 * ks][2 * i], s[2 * ks][2 * i + 1], o.z);
          o.y = split_pair(s[2 * ks + 1][2 * i], s[2 * ks + 1][2 * i + 1], o.w);
          if (v0 + warp * 16 + 8 * i < V) U[ks * to_next + i * 32] = o;
        }
      }
    };
    fetch(0, 0);
    leave(0);
    weigh(0);
#pragma unroll
    for (int ks = 0; ks < CL / 16; ++ks) {   // (weights and states are formed under products that are on their way)
      const int x = ks & 1;
      if (ks + 1 < CL / 16) fetch(ks + 1, x ^ 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        mma_bf16(acc[2 * u], h[x][0], h[x][1], h[x][2], h[x][3], k[x][u][0], k[x][u][1]);
        mma_bf16(acc[2 * u + 1], h[x][0], h[x][1], h[x][2], h[x][3], k[x][u][2], k[x][u][3]);
      }
      if (ks + 1 < CL / 16) weigh(x ^ 1);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        mma_bf16(acc[2 * u], l[x][0], l[x][1], l[x][2], l[x][3], k[x][u][0], k[x][u][1]);
        mma_bf16(acc[2 * u + 1], l[x][0], l[x][1], l[x][2], l[x][3], k[x][u][2], k[x][u][3]);
      }
      if (ks + 1 < CL / 16) leave(ks + 1);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int x = 0; x < 4; ++x) s[j][x] = fmaf(s[j][x], f, acc[j][x]);
    st = st + 1 == kSStages ? 0 : st + 1;
  }
  if (SUMS) {
#pragma unroll
    for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(left(seg) + j * 512) = make_float4(s[j][0], s[j][1], s[j][2], s[j][3]);
  } else if (last) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int d = d0 + 8 * j + 2 * qd + (x & 1), v = vr + 8 * (x >> 1);
        if (d < D && v < V) p.s_pool[(pool * D + d) * V + v] = s[j][x];
      }
  }
}

// Block = (chunk, entry and head), a warp = 16 MT tokens x 32 value columns: o = q S + weights x values, normaliser, the head's norm and the output gate.
// S comes as operand fragments and the values as rows, sixteen of either a step, through a ring of the warp's own in shared memory that it fills by cp.async, so that no step
// waits for another warp and the values travel under the products before them.  MT: with all 64 tokens a warp reads every staged number once; narrow heads have
// too few columns to fill a block that way (four warps of 32 columns at 128: 44 us a call against 29 with sixteen).
constexpr int kWStage = 2048, kWStages = 4, kVRow = 40;   // (bytes a step; a row of values: 64 bytes in 80, eight of them in different banks)
constexpr int kOutWarps = 16;
constexpr int kOutFloats = 4 * CL + 4 * CL + CL + CL;

// Shared memory: q, k, the weights and the rings; later every warp's results (32-bit) and gates
__host__ __device__ __forceinline__ int out_tiles(int D, int warps, int MT) {
  const int a = (2 * CL * (D + 8) + 2 * CL * PROW) * 2 + warps * kWStages * kWStage, b = warps * MT * 16 * 192;
  return a > b ? a : b;
}
static int out_smem(int D, int warps, int MT) { return out_tiles(D, warps, MT) + kOutFloats * 4; }

template <int MT>
__global__ void __launch_bounds__(kOutWarps * 32, 1) mlstm_par_out_kernel(const pcs_mlstm_params p, float* scratch, long long slots) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int TG = 4 / MT;   // groups of tokens
  const int D = p.dim, V = p.vdim, H = p.heads, QROW = D + 8, nthr = blockDim.x, nw = nthr >> 5, ncol = nw / TG;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, grp = lane >> 2, qd = lane & 3, tg = warp / ncol, wc = warp - tg * ncol, m0 = tg * MT;
  __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(smem_raw);   // [64][QROW]
  __nv_bfloat16* Ks = Qs + CL * QROW;
  __nv_bfloat16* Ph = Ks + CL * QROW;                               // [64][PROW] the weights, hi and lo
  __nv_bfloat16* Pl = Ph + CL * PROW;
  unsigned char* ring = reinterpret_cast<unsigned char*>(Pl + CL * PROW) + warp * (kWStages * kWStage);
  float* tok = reinterpret_cast<float*>(smem_raw + out_tiles(D, nw, MT));   // [4][64] a, g, e^{m_in - g}, e^{-m}
  float* psum = tok + 4 * CL;                                       // [4][64] sums of the weights over 16 keys
  float* nq = psum + 4 * CL;                                        // [64] q . n of the state
  float* inv = nq + CL;                                             // [64] 1 / rms
  const Scratch sc(scratch, slots, p);
  const int c = blockIdx.x, b = blockIdx.y / H, head = blockIdx.y - b * H;
  const int len = p.seq_len[b], i0 = c * CL;
  if (i0 >= len) return;
  const int n = min(CL, len - i0);
  const long long at = static_cast<long long>((b ? sc.first[b] : 0) + c) * H + head, t0 = p.seq_off[b] + i0, rs = p.row_stride;
  const __nv_bfloat16* rows = static_cast<const __nv_bfloat16*>(p.proj) + t0 * rs;
  const int mts = (n + 15) / 16, kvs = min(mts, m0 + MT);   // tiles of 16 tokens that hold one; those that some token of the warp sees
  const int ksteps = D / 16, steps = ksteps + kvs, c0 = wc * 32;
  const bool g16 = p.g_off % 8 == 0, o16 = (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
  const int pieces = D / 8;
  for (int e = tid; e < 2 * CL * pieces; e += nthr) {   // q, then k (a row a warp left most lanes of narrow heads idle: 64 x 128 10.8 us a launch against 9.8)
    const int r = e / pieces, k = (e - r * pieces) * 8, t = r & (CL - 1);
    if (t < n) cp_async16(Qs + r * QROW + k, rows + t * rs + (r < CL ? p.q_off : p.k_off) + head * D + k);
    else *reinterpret_cast<uint4*>(Qs + r * QROW + k) = make_uint4(0u, 0u, 0u, 0u);
  }
  cp_async_commit();
  // step s of this warp: the fragments of sixteen state rows, then the values of sixteen tokens
  const float* S = sc.u + at * D * V + (c0 / 8) * 128 + lane * 4;
  const __nv_bfloat16* vals = rows + (lane >> 2) * rs + p.v_off + head * V + c0 + (lane & 3) * 8;
  auto load = [&](int s) {
    unsigned char* dst = ring + (s % kWStages) * kWStage;
    if (s < ksteps) {
      const float* src = S + static_cast<long long>(s) * 16 * V;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (c0 + 8 * q < V) cp_async16(dst + q * 512 + lane * 16, src + q * 128);
        else *reinterpret_cast<uint4*>(dst + q * 512 + lane * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
    } else if (s < steps) {
      const int t = (s - ksteps) * 16 + (lane >> 2);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dst) + ((lane >> 2) + 8 * u) * kVRow + (lane & 3) * 8;
        if (t + 8 * u < n && c0 + (lane & 3) * 8 < V) cp_async16(d, vals + ((s - ksteps) * 16 + 8 * u) * rs);
        else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int s = 0; s < kWStages; ++s) load(s);
  for (int e = tid; e < 4 * CL; e += nthr) tok[e] = sc.tok[at * 5 * CL + e];
  cp_async_wait<kWStages>();
  __syncthreads();   // q and k
  // ---- weights e^{a_s - g_t} (q_t . k_s) / sqrt(dim), s <= t: ten tiles of 16 tokens x 16 keys, a warp each; q . n: 4 tokens per warp ----
  const uint32_t q_base = static_cast<uint32_t>(__cvta_generic_to_shared(Qs)) + ((lane & 15) * QROW + (lane >> 4) * 8) * 2;
#pragma unroll 1
  for (int job = warp; job < 10; job += nw) {
    const int mi = job < 1 ? 0 : job < 3 ? 1 : job < 6 ? 2 : 3, nj = job - mi * (mi + 1) / 2, k0 = nj * 16, ra = mi * 16 + grp, rb = ra + 8;
    const uint32_t k_base = static_cast<uint32_t>(__cvta_generic_to_shared(Ks)) + ((k0 + (lane & 7) + ((lane >> 4) & 1) * 8) * QROW + ((lane >> 3) & 1) * 8) * 2;
    float s[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < ksteps; ++kk) {
      uint32_t a0, a1, a2, a3, f[4];
      ldsm_x4(q_base + mi * 16 * QROW * 2 + kk * 32, a0, a1, a2, a3);
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
    if (qd == 0) { psum[nj * CL + ra] = sa; psum[nj * CL + rb] = sb; }
  }
  const float* ns = sc.n + at * D;
#pragma unroll 1
  for (int t = (nw - 1 - warp) * 4; t < CL; t += nw * 4) {   // (the last warps have no tile above)
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    for (int d = lane; d < D; d += 32) {
      const float x = ns[d];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = fmaf(x, ldf(Qs + (t + i) * QROW + d), a[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = warp_sum(a[i]);
      if (lane == 0) nq[t + i] = a[i] * p.q_scale * tok[2 * CL + t + i];
    }
  }
  // ---- q S, sixteen state rows a step ----
  float acc[MT][4][4];             // [tile of tokens][tile of 8 columns]
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[m][j][0] = acc[m][j][1] = acc[m][j][2] = acc[m][j][3] = 0.f;
#pragma unroll 1
  for (int ks = 0; ks < ksteps; ++ks) {
    cp_async_wait<kWStages - 1>();   // (a lane reads the pieces that it fetched itself)
    uint4 f[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) f[q] = *reinterpret_cast<const uint4*>(ring + (ks % kWStages) * kWStage + q * 512 + lane * 16);
    if (ks + kWStages >= ksteps) __syncwarp();   // (rows of values: other lanes' pieces)
    load(ks + kWStages);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      if (m0 + m >= mts) break;
      uint32_t a[4];
      ldsm_x4(q_base + (m0 + m) * 16 * QROW * 2 + ks * 32, a[0], a[1], a[2], a[3]);
#pragma unroll
      for (int q = 0; q < 4; ++q) mma_bf16(acc[m][q], a[0], a[1], a[2], a[3], f[q].x, f[q].y);
#pragma unroll
      for (int q = 0; q < 4; ++q) mma_bf16(acc[m][q], a[0], a[1], a[2], a[3], f[q].z, f[q].w);
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const float ca = tok[2 * CL + 16 * (m0 + m) + grp] * p.q_scale, cb = tok[2 * CL + 16 * (m0 + m) + grp + 8] * p.q_scale;
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[m][j][0] *= ca; acc[m][j][1] *= ca; acc[m][j][2] *= cb; acc[m][j][3] *= cb; }
  }
  // the gates of a lane's eight columns of every eighth token
  const int col = c0 + (lane & 3) * 8;
  uint4 gate[2 * MT];
#pragma unroll
  for (int h = 0; h < 2 * MT; ++h) {
    const int r = 16 * m0 + 8 * h + (lane >> 2);
    const __nv_bfloat16* src = rows + r * rs + p.g_off + head * V + col;
    gate[h] = make_uint4(0u, 0u, 0u, 0u);
    if (r < n && col < V) {
      if (g16) gate[h] = *reinterpret_cast<const uint4*>(src);
      else {
        const uint32_t* s4 = reinterpret_cast<const uint32_t*>(src);
        gate[h] = make_uint4(s4[0], s4[1], s4[2], s4[3]);
      }
    }
  }
  __syncthreads();   // the weights, their sums and q . n
  // ---- + weights x values ----
  {
    const uint32_t ph = static_cast<uint32_t>(__cvta_generic_to_shared(Ph)) + ((m0 * 16 + (lane & 15)) * PROW + (lane >> 4) * 8) * 2, pl = ph + CL * PROW * 2;
    const uint32_t ring_base = static_cast<uint32_t>(__cvta_generic_to_shared(ring)) + ((lane & 15) * kVRow + (lane >> 4) * 8) * 2;
#pragma unroll 1
    for (int kv = 0; kv < kvs; ++kv) {
      cp_async_wait<kWStages - 1>();
      __syncwarp();
      uint32_t f[2][4];
      const uint32_t st = ring_base + ((ksteps + kv) % kWStages) * kWStage;
#pragma unroll
      for (int u = 0; u < 2; ++u) ldsm_x4_t(st + u * 32, f[u][0], f[u][1], f[u][2], f[u][3]);
      cp_async_commit();   // (nothing is fetched any more; the count of groups goes on, so that the last rows have landed when the loop ends)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (m0 + m < kv || m0 + m >= mts) continue;   // (tiles before these tokens do not see them)
        uint32_t h[4], l[4];
        ldsm_x4(ph + (m * 16 * PROW + kv * 16) * 2, h[0], h[1], h[2], h[3]);
        ldsm_x4(pl + (m * 16 * PROW + kv * 16) * 2, l[0], l[1], l[2], l[3]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma_bf16(acc[m][2 * u], h[0], h[1], h[2], h[3], f[u][0], f[u][1]);
          mma_bf16(acc[m][2 * u + 1], h[0], h[1], h[2], h[3], f[u][2], f[u][3]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma_bf16(acc[m][2 * u], l[0], l[1], l[2], l[3], f[u][0], f[u][1]);
          mma_bf16(acc[m][2 * u + 1], l[0], l[1], l[2], l[3], f[u][2], f[u][3]);
        }
      }
    }
  }
  // ---- normaliser, the head's norm, the output gate ----
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 16 * (m0 + m) + grp + 8 * i;
      float w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = k <= m0 + m ? psum[k * CL + r] : 0.f;
      const float den = 1.f / (fmaxf(fabsf(nq[r] + (w[0] + w[1]) + (w[2] + w[3])), tok[3 * CL + r]) + 1e-6f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[m][j][i * 2] *= den;
        acc[m][j][i * 2 + 1] *= den;
      }
    }
  __syncthreads();   // (what lies in shared memory up to here has been read)
  // The warp's results pass through shared memory, 16-byte pieces of a row exchanged by its number: a lane then has eight columns of a
  // row, and the code is a short loop (a block runs it once: straight-line code is fetched more slowly than it runs, 17 000 cycles against 5 000).
  constexpr int kMine = MT * 16 * 48;   // floats of a warp: its results, then its gates
  float* mine = reinterpret_cast<float*>(smem_raw) + warp * kMine;
  uint4* gates = reinterpret_cast<uint4*>(mine + MT * 16 * 32) + lane;
  auto at_row = [&](int row, int j) { return row * 32 + (((2 * j + (qd >> 1)) ^ (2 * (grp & 3))) * 4 + (qd & 1) * 2); };   // columns 8 j + 2 qd and the next of row `row` = grp mod 8
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      *reinterpret_cast<float2*>(mine + at_row(16 * m + grp, j)) = make_float2(acc[m][j][0], acc[m][j][1]);
      *reinterpret_cast<float2*>(mine + at_row(16 * m + grp + 8, j)) = make_float2(acc[m][j][2], acc[m][j][3]);
    }
#pragma unroll
  for (int h = 0; h < 2 * MT; ++h) gates[32 * h] = gate[h];
  __syncthreads();
  // Sums of squares: a row's in sixteen chains, four lanes for each quarter of the (padded) columns, whatever the number of warps that hold them (each warp its own columns: other bits, and no
  // faster; from register to register, warp after warp: 1.9 us more a launch)
#pragma unroll 1
  for (int r = warp * 8; r < CL; r += nw * 8) {
    const int t0w = r / (16 * MT), row = r - t0w * (16 * MT) + grp;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int u = 0; u < MT; ++u) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q * MT + u >= ncol) continue;
        const float* from = reinterpret_cast<const float*>(smem_raw) + (t0w * ncol + q * MT + u) * kMine;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 y = *reinterpret_cast<const float2*>(from + at_row(row, j));
          x[q] = fmaf(y.x, y.x, fmaf(y.y, y.y, x[q]));
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q] += __shfl_xor_sync(0xffffffffu, x[q], 1);
      x[q] += __shfl_xor_sync(0xffffffffu, x[q], 2);
    }
    if (qd == 0) inv[r + grp] = 1.f / sqrtf((((x[0] + x[1]) + x[2]) + x[3]) / static_cast<float>(V) + p.eps);
  }
  __syncthreads();
  if (col >= V) return;   // (vdim is a multiple of 8)
  float w[8];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint32_t u = reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(p.norm_w) + head * V + col)[k];
    w[2 * k] = __uint_as_float(u << 16);
    w[2 * k + 1] = __uint_as_float(u & 0xffff0000u);
  }
  const long long os = static_cast<long long>(H) * V;
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + (t0 + 16 * m0) * os + head * V + col;
  const int nm = min(16 * MT, n - 16 * m0);
#pragma unroll 1
  for (int r = lane >> 2; r < nm; r += 8, gates += 32) {
    const float f = inv[16 * m0 + r];
    const int e = 2 * (r & 3);
    float x[8];
    const float4 a = *reinterpret_cast<const float4*>(mine + r * 32 + ((2 * (lane & 3)) ^ e) * 4), d = *reinterpret_cast<const float4*>(mine + r * 32 + ((2 * (lane & 3) + 1) ^ e) * 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = d.x; x[5] = d.y; x[6] = d.z; x[7] = d.w;
    const uint4 gv = *gates;
    const uint32_t g[4] = {gv.x, gv.y, gv.z, gv.w};
    uint32_t y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      y[k] = pack_bf16(x[2 * k] * f * w[2 * k] * sigmoid_nr_(__uint_as_float(g[k] << 16)), x[2 * k + 1] * f * w[2 * k + 1] * sigmoid_nr_(__uint_as_float(g[k] & 0xffff0000u)));
    __nv_bfloat16* o = out + r * os;
    if (o16) *reinterpret_cast<uint4*>(o) = make_uint4(y[0], y[1], y[2], y[3]);
    else {
#pragma unroll
      for (int k = 0; k < 4; ++k) reinterpret_cast<uint32_t*>(o)[k] = y[k];
    }
  }
}

// Segments of a walk over `chunks`.  us, fitted: one walk 1.9 and 0.955 a chunk; two launches 5.3, 1.35 a chunk of a segment and 0.38 a segment (the later ones add up those before them).  Tiles x chunks,
// as one walk / in so many segments: 4 x 7 8.5 / 8.6 in 4, 4 x 10 11.3 / 9.9 in 5, 8 x 13 13.9 / 9.9 in 7, 32 x 11 12.4 / 11.1 in 4, 32 x 16 17.0 / 13.2 in 4, 4 x 47 45.1 / 15.6 in 12.
static int state_segments(long long tiles, int chunks) {
  int best = 1;
  double least = 0.98 * (1.9 + 0.955 * chunks);
  for (int per = 2; per < chunks; ++per) {
    const int segs = (chunks + per - 1) / per;
    const double us = 5.3 + 1.35 * per + 0.38 * segs;
    if (us < least && segs * tiles <= kMaxTiles) {
      least = us;
      best = segs;
    }
  }
  return best;
}

template <bool SUMS, int CHAIN>
int launch_state(const pcs_mlstm_params& p, float* scratch, long long slots, dim3 grid, int segs, cudaStream_t st) {
  static PerDevice<NoInfo> set_up;
  if (int rc = set_up.once([&] { return cudaFuncSetAttribute(mlstm_par_state_kernel<SUMS, CHAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStateSmem<CHAIN>); })) return rc;
  mlstm_par_state_kernel<SUMS, CHAIN><<<grid, kST, kStateSmem<CHAIN>, st>>>(p, scratch, slots, segs);
  PCS_CHECK_CUDA(cudaGetLastError());
  return PCS_OK;
}

template <int MT>
int launch_out(const pcs_mlstm_params& p, float* scratch, long long slots, dim3 grid, cudaStream_t st) {
  static PerDevice<NoInfo> set_up;
  if (int rc = set_up.once([&] { return cudaFuncSetAttribute(mlstm_par_out_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_smem(256, kOutWarps, MT)); })) return rc;
  const int warps = (p.vdim + 31) / 32 * (4 / MT);
  mlstm_par_out_kernel<MT><<<grid, warps * 32, out_smem(p.dim, warps, MT), st>>>(p, scratch, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  return PCS_OK;
}

static long long tiles_of(int n_seqs, int heads, int dim, int vdim) { return static_cast<long long>((dim + 63) / 64) * ((vdim + 63) / 64) * heads * n_seqs; }

static long long floats(int n_tokens, int n_seqs, int heads, int dim, int vdim, bool cut) {
  return Scratch::whole(n_tokens / CL + n_seqs, n_seqs, heads, dim, vdim) + (cut ? Scratch::kLeft + Scratch::kLeftN : 0);
}

}  // namespace

long long mlstm_par_wanted(const pcs_mlstm_params& p) {
  return floats(p.n_tokens, p.n_seqs, p.heads, p.dim, p.vdim, state_segments(tiles_of(p.n_seqs, p.heads, p.dim, p.vdim), (p.max_len + CL - 1) / CL) > 1);
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
      p.chunk_floats < floats(p.n_tokens, p.n_seqs, p.heads, p.dim, p.vdim, false))
    return PCS_OK;
  const long long slots = p.n_tokens / CL + p.n_seqs;
  const int chunks = (p.max_len + CL - 1) / CL;
  *handled = true;
  float* s = p.chunk_scratch;
  mlstm_par_gates_kernel<<<dim3(p.n_seqs, p.heads), 512, 2 * chunks * sizeof(float), st>>>(p, s, slots);
  PCS_CHECK_CUDA(cudaGetLastError());
  const int tiles = ((p.dim + 63) / 64) * ((p.vdim + 63) / 64);
  const int segs = p.chunk_floats < floats(p.n_tokens, p.n_seqs, p.heads, p.dim, p.vdim, true) ? 1 : state_segments(tiles_of(p.n_seqs, p.heads, p.dim, p.vdim), chunks);
  const dim3 walks(tiles, p.heads, p.n_seqs * segs);
  if (segs > 1)
    if (int rc = launch_state<true, 2>(p, s, slots, walks, segs, st)) return rc;
  if (int rc = segs == 1 && chunks >= 24 ? launch_state<false, 4>(p, s, slots, walks, 1, st) : launch_state<false, 2>(p, s, slots, walks, segs, st)) return rc;
  const dim3 grid(chunks, p.n_seqs * p.heads);
  const int rc = p.vdim <= 128 ? launch_out<1>(p, s, slots, grid, st) : p.vdim <= 256 ? launch_out<2>(p, s, slots, grid, st) : launch_out<4>(p, s, slots, grid, st);
  if (rc) return rc;
  count_launch(segs > 1 ? 4 : 3);
  return PCS_OK;
}

}  // namespace pcs

// What any call of these sizes may want: its longest entry, which decides on segments, has up to n_tokens
PCS_API int64_t pcs_mlstm_scratch_floats(int n_tokens, int n_seqs, int heads, int dim, int vdim) {
  if (n_tokens <= 0 || n_seqs <= 0 || heads <= 0 || dim <= 0 || vdim <= 0) return 0;
  const long long tiles = pcs::tiles_of(n_seqs, heads, dim, vdim);
  bool cut = false;
  for (int c = 2; !cut && 2 * tiles <= pcs::kMaxTiles && c <= (n_tokens + pcs::CL - 1) / pcs::CL; ++c) cut = pcs::state_segments(tiles, c) > 1;
  return pcs::floats(n_tokens, n_seqs, heads, dim, vdim, cut);
}
