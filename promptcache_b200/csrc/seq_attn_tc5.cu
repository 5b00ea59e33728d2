// tcgen05 attention over the slot pool for prompts (bfloat16 storage, 32-bit scores, softmax and accumulation).
//
// One block = two tiles ("halves") of 128 query rows that share the K / V tiles of 64 keys they walk.  A half is 128 consecutive new tokens of one
// sequence and head; its softmax belongs to a warpgroup (one thread per query row), its products to an MMA-issuing warp of its own:
//
//   TMA warp      K and V tiles through a ring of 3 or 4 stages (3-d tensor maps over the pool, 128-byte swizzle)
//   MMA warp      S(j) = Q K_j^T into one of two TMEM buffers, two tiles ahead;  O += P_hi V_j + P_lo V_j  with P in TMEM
//   warpgroup     reads S, applies scale / cap / bias / masks in the base-2 domain, online softmax, writes P over S as two bfloat16 operands
//
// The 32-bit weights enter the tensor cores as P = hi + lo (hi = bf16(P), lo = bf16(P - hi)), so ~16 bits of each are kept: three 128 x 64 x 128
// products per tile and half where a plain flash kernel has two.  TMEM: S 4 x 64 columns, O 2 x vdim columns.  The accumulator is rescaled only when
// a row's maximum grew by more than 2^8 (P then stays below 2^8, exact in the same 16 bits).  The products multiply hidden keys of a tile by 0: a row
// whose result is not finite is formed again from the keys it sees (attn_row_again).
//
// Which two tiles a block takes: neighbours of one head (2m, 2m + 1), those with the most keys in the first blocks; or one from either end (m,
// n - 1 - m), which gives every block of a sequence the same work.  Where that leaves SMs idle (few new tokens behind many stored ones) a cluster of 2,
// 4 or 8 blocks shares the walk over the keys and merges through distributed shared memory.  The choice is a cost model on the host (Plan).
//
// What bounds it (B200, bfloat16, 16 heads, dim = vdim = 128): 1.4 us per key tile of both halves, of which the 24 products take 0.95 us at full
// rate; without any softmax arithmetic the walk takes 1.24 us.  Against the mma.sync kernel it replaces (seq_attn_tc.cu, which still serves wider heads and short entries):
//   2048 new tokens        122 -> 47 us        6144 and 2311 new tokens                      842 -> 286 us (617 TFLOP/s of the two-product count)
//   256 behind 4000 stored 164 -> 50 us (8 heads 164 -> 27)      four continued prompts, window 1024, cap  177 -> 85 us
#include "seq_attn.cuh"
#include "seq_mma.cuh"
#include "seq_tc5.cuh"

namespace pcs {

namespace {

constexpr int BM = 128, BN = 64;
constexpr int kThreads = 352;  // warpgroups 0 and 1, TMA warp 8, MMA warps 9 and 10
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescale = 8.0f;
constexpr int kMaxSplits = 8;  // blocks of a cluster that share one walk
constexpr int kTab = 192;      // distances of a tile pair of 128 rows and 64 keys (191)

__device__ int attn_tc5_timeouts;  // blocks one of whose waits ran out

template <int DP, int VP>
struct Cfg {
  static constexpr int kQBytes = BM * DP * 2, kKBytes = BN * DP * 2, kVBytes = BN * VP * 2;
  static constexpr int kTabBytes = 2 * 2 * kTab * 4;
  static constexpr int kRoom = 227 * 1024 - 1024 - 2 * kQBytes - kTabBytes - 512;
  static constexpr int kFit = kRoom / (kKBytes + kVBytes);
  static constexpr int kStages = kFit < 4 ? kFit : 4;
  static_assert(kStages >= 2, "the K/V ring needs two stages");
  static constexpr int kOffKV = 2 * kQBytes;
  // the merge of a split walk lays its partial results over Q and the ring: [split][half][column of the slice][row], then (m, l)
  static constexpr int kPartBytes = 2 * BM * VP * 4, kMergeBytes = kPartBytes + kMaxSplits * 2 * BM * 8;
  static constexpr int kRing = kOffKV + kStages * (kKBytes + kVBytes);
  static constexpr int kOffTab = kRing > kMergeBytes ? kRing : kMergeBytes;
  static constexpr int kOffBars = kOffTab + kTabBytes;
  static constexpr int kSmem = 1024 + kOffBars + 512;
  static constexpr int kColO = 256;
};


// The tiles one half walks: [0, n_first) and [lo, hi)
struct Range {
  int rows, q0, n_first, lo, hi;
  __device__ __forceinline__ bool has(int k) const { return k < n_first || (k >= lo && k < hi); }
};

template <int DP, int VP, bool BIAS, bool CAP>
__global__ void __launch_bounds__(kThreads, 1) attn_tc5_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ pcs_attn_params p, const int ends,
                                                               const int splits) {
  using C = Cfg<DP, VP>;
  constexpr int ST = C::kStages;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* sQ = smem;
  unsigned char* sKV = smem + C::kOffKV;
  float* sTab = reinterpret_cast<float*>(smem + C::kOffTab);
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + C::kOffBars);
  uint64_t* ragged = q_full + 1;          // the last K / V tile of a sequence, before its rows past the end are cleared
  uint64_t* k_full = ragged + 1;          // [stages]
  uint64_t* v_full = k_full + ST;
  uint64_t* kv_empty = v_full + ST;       // [2 halves][stages]
  uint64_t* s_full = kv_empty + 2 * ST;   // [2 halves][2 buffers]
  uint64_t* p_full = s_full + 4;
  uint64_t* o_full = p_full + 4;
  uint64_t* drained = o_full + 4;         // [2 halves] every product has ended
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  // ---- which two tiles ----
  const int b_all = blockIdx.x / splits, rank = blockIdx.x - b_all * splits;
  int b, h, t0, t1;
  {
    const int per = p.n_seqs * p.n_heads, tile = b_all / per, rem = b_all - tile * per;
    b = rem / p.n_heads;
    h = rem - b * p.n_heads;
    const int n = (p.seq_len[b] + BM - 1) / BM, n_max = (p.max_len + BM - 1) / BM;
    if (ends & 1) {
      t0 = n - 1 - tile; t1 = tile;
      if (t1 > t0) return;
      if (t1 == t0) t1 = -1;
    } else {
      t0 = 2 * ((n_max + 1) / 2 - 1 - tile); t1 = t0 + 1;
      if (t0 >= n) return;
      if (t1 >= n) t1 = -1;
    }
  }
  const int len = p.seq_len[b], pos0 = p.seq_pos0[b], off = p.seq_off[b], slot = p.pool_slot ? p.pool_slot[b] : p.seq_slot[b];
  const int total_keys = pos0 + len;
  const int plane = slot * p.n_kv_heads + h / (p.n_heads / p.n_kv_heads);
  const bool windowed = p.window > 0, chunked = p.chunk > 0;
  const int keep = windowed ? min(max(p.keep_first, 0), total_keys) : 0;
  Range rg[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    Range& r = rg[x];
    const int t = x ? t1 : t0;
    r.q0 = max(t, 0) * BM;
    r.rows = t < 0 ? 0 : min(BM, len - r.q0);
    const int first = pos0 + r.q0;
    r.hi = r.rows > 0 ? (first + r.rows + BN - 1) / BN : 0;
    r.lo = windowed ? max(0, first - p.window + 1) / BN : chunked ? first / p.chunk * p.chunk / BN : 0;
    r.n_first = (keep + BN - 1) / BN;
    if (r.n_first >= r.lo) { r.n_first = 0; r.lo = 0; }
    if (r.rows <= 0) r.n_first = r.lo = 0;
  }
  // the walk covers both
  int nf = max(rg[0].n_first, rg[1].n_first), lo = rg[1].rows > 0 ? min(rg[0].lo, rg[1].lo) : rg[0].lo;
  const int hi = max(rg[0].hi, rg[1].hi);
  if (nf >= lo) nf = lo = 0;
  const int n_all = nf + hi - lo, it0 = rank * n_all / splits, n_it = (rank + 1) * n_all / splits - it0;  // this block's part of it
  auto tile_of = [&](int it) { return it0 + it < nf ? it0 + it : lo + it0 + it - nf; };
  float m = -INFINITY, l = 0.f;  // (softmax threads) the row's running maximum and sum
  int j = 0;                     // and its tiles so far
  bool again = false;            // its result is not finite
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, abort_word); };
  // (ends bit 1) tests: in three blocks of four the TMA warp or one of the MMA warps gives up at some tile of the walk, as if its wait had run out
  auto dropped = [&](int it) {
    if (!(ends & 2) || warp != 8 + static_cast<int>(blockIdx.x & 3) || it != static_cast<int>(blockIdx.x >> 2 & 7)) return false;
    *abort_word = 1;
    return true;
  };

  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_init(q_full, 1);
    mbar_init(ragged, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&kv_empty[s], 1);
      mbar_init(&kv_empty[ST + s], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&o_full[i], 1);
    }
    mbar_init(&drained[0], 1);
    mbar_init(&drained[1], 1);
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 9) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 8) {
    // ===================== TMA producer =====================
    if (lane == 0) {
      mbar_expect_tx(q_full, (rg[1].rows > 0 ? 2 : 1) * C::kQBytes);
      for (int x = 0; x < 2; ++x)
        if (rg[x].rows > 0)
          for (int f = 0; f < DP / 64; ++f) tma_load_3d(sQ + x * C::kQBytes + f * BM * 128, &map_q, q_full, f * 64, h, off + rg[x].q0);
    }
    int issued = 0, ragged_it = -1;   // tiles asked for so far, the one that passes the `ragged` barrier
    for (int it = 0; it < n_it; ++it) {
      const int s = it % ST, key0 = tile_of(it) * BN;
      if (dropped(it)) break;
      if (it >= ST) {
        const uint32_t par = static_cast<uint32_t>((it / ST - 1) & 1);
        const bool free = wait(&kv_empty[s], par) && wait(&kv_empty[ST + s], par);
        if (!__all_sync(0xffffffffu, free)) break;
      }
      unsigned char* dk = sKV + s * (C::kKBytes + C::kVBytes);
      unsigned char* dv = dk + C::kKBytes;
      const int left = total_keys - key0;  // keys of this tile that exist
      if (lane == 0) {
        uint64_t *bk = left < BN ? ragged : &k_full[s], *bv = left < BN ? ragged : &v_full[s];
        if (left < BN) {
          mbar_expect_tx(ragged, C::kKBytes + C::kVBytes);
        } else {
          mbar_expect_tx(bk, C::kKBytes);
          mbar_expect_tx(bv, C::kVBytes);
        }
        for (int f = 0; f < DP / 64; ++f) tma_load_3d(dk + f * BN * 128, &map_k, bk, f * 64, key0, plane);
        for (int f = 0; f < VP / 64; ++f) tma_load_3d(dv + f * BN * 128, &map_v, bv, f * 64, key0, plane);
      }
      ++issued;
      if (left < BN) {  // the sequence's last tile: rows behind its end hold anything, and 0 * NaN is not 0
        ragged_it = it;
        __syncwarp();
        if (!__all_sync(0xffffffffu, wait(ragged, 0))) break;
        for (int f = 0; f < (DP + VP) / 64; ++f)
          for (int i = left * 8 + lane; i < BN * 8; i += 32) *reinterpret_cast<uint4*>(dk + f * BN * 128 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&k_full[s]);
          mbar_arrive(&v_full[s]);
        }
      }
    }
    // all of it has landed when this warp is done (in a walk that was given up, the tiles nobody waited for)
    mbar_drain(q_full, 0);
    for (int i = max(0, issued - ST); i < issued; ++i) {
      if (i == ragged_it) {
        mbar_drain(ragged, 0);
      } else {
        mbar_drain(&k_full[i % ST], static_cast<uint32_t>((i / ST) & 1));
        mbar_drain(&v_full[i % ST], static_cast<uint32_t>((i / ST) & 1));
      }
    }
    __syncwarp();
  } else if (warp >= 9) {
    // ===================== MMA issuers: warp 9 drives half 0, warp 10 half 1 =====================
    const int x = warp - 9;
    const Range r = x ? rg[1] : rg[0];
    const int leader = lane == 0;
    auto all_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
    constexpr uint32_t idesc_qk = idesc_bf16(BM, BN, 0), idesc_pv = idesc_bf16(BM, VP, 1);
    const uint64_t q_desc = smem_desc_sw128(smem_u32(sQ + x * C::kQBytes), 16, 1024);
    const uint64_t k_desc0 = smem_desc_sw128(smem_u32(sKV), 16, 1024);
    const uint64_t v_desc0 = smem_desc_sw128(smem_u32(sKV + C::kKBytes), BN * 128, 1024);
    const uint32_t tmem_s = tmem_base + x * 128, tmem_o = tmem_base + C::kColO + x * VP;
    int jS = 0, itS = 0, jP = 0;   // scores issued, the walk's next tile for them; weights x values issued
    bool ok = all_wait(q_full, 0);
    for (int ip = 0; ip < n_it && ok; ++ip) {
      if (dropped(ip)) break;
      // scores up to two tiles ahead of the weights, as long as the tile can arrive without this half's next release
      while (ok && jS < jP + 2) {
        while (itS < n_it && !r.has(tile_of(itS))) ++itS;
        if (itS >= n_it || itS >= ip + ST) break;
        const int s = itS % ST;
        ok = all_wait(&k_full[s], static_cast<uint32_t>((itS / ST) & 1));
        if (!ok) break;
        tc_fence_after();
        const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((s * (C::kKBytes + C::kVBytes)) >> 4);
#pragma unroll
        for (int kk = 0; kk < DP / 16; ++kk)
          umma_ss(tmem_s + (jS & 1) * BN, q_desc + static_cast<uint64_t>(((kk >> 2) * BM * 128 + (kk & 3) * 32) >> 4),
                  k_desc + static_cast<uint64_t>(((kk >> 2) * BN * 128 + (kk & 3) * 32) >> 4), idesc_qk, kk > 0 ? 1u : 0u, leader);
        tc_commit(&s_full[x * 2 + (jS & 1)], leader);
        ++jS;
        ++itS;
      }
      if (!ok) break;
      const int s = ip % ST;
      const uint32_t par = static_cast<uint32_t>((ip / ST) & 1);
      if (!r.has(tile_of(ip))) {  // the other half's tile: hand the stage back once it has been filled
        ok = all_wait(&k_full[s], par) && all_wait(&v_full[s], par);
        if (ok && leader) mbar_arrive(&kv_empty[x * ST + s]);
        continue;
      }
      ok = all_wait(&v_full[s], par) && all_wait(&p_full[x * 2 + (jP & 1)], static_cast<uint32_t>((jP >> 1) & 1));
      if (!ok) break;
      tc_fence_after();
      const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((s * (C::kKBytes + C::kVBytes)) >> 4);
      const uint32_t pa = tmem_s + (jP & 1) * BN;
#pragma unroll
      for (int kk = 0; kk < BN / 16; ++kk) umma_ts(tmem_o, pa + kk * 8, v_desc + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv, (jP > 0 || kk > 0) ? 1u : 0u, leader);
#pragma unroll
      for (int kk = 0; kk < BN / 16; ++kk) umma_ts(tmem_o, pa + 32 + kk * 8, v_desc + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv, 1u, leader);
      tc_commit(&o_full[x * 2 + (jP & 1)], leader);
      tc_commit(&kv_empty[x * ST + s], leader);
      ++jP;
    }
    __syncwarp();
    tc_commit(&drained[x], leader);   // and all products have ended
    mbar_drain(&drained[x], 0);
    __syncwarp();
  } else {
    // ===================== softmax: warpgroup x owns half x, a thread one query row =====================
    const int x = warp >> 2, row = tid & 127;
    const Range r = x ? rg[1] : rg[0];
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tmem_s0 = tmem_base + lanes + x * 128, tmem_o = tmem_base + lanes + C::kColO + x * VP;
    const int first = pos0 + r.q0, pos = first + row;
    const bool live = row < r.rows;
    // this row sees the keys [lo_key, pos] and [0, keep)
    const int lo_key = windowed ? max(0, pos - p.window + 1) : chunked ? pos / p.chunk * p.chunk : 0;
    const int end_key = live ? pos + 1 : 0;
    const float scale = p.scale * (p.head_scale ? p.head_scale[h] : 1.f), scale2 = scale * kLog2e;
    const float cap_in = CAP ? scale / p.softcap * 2.f * kLog2e : 0.f, cap_out = CAP ? p.softcap * kLog2e : 0.f;
    const float r1 = (BIAS && p.bias_r1) ? p.bias_r1[h] : 0.f, r2 = (BIAS && p.bias_r1) ? p.bias_r2[h] : 0.f;
    const float* btab = (BIAS && p.bias_table) ? p.bias_table + static_cast<long long>(h) * p.bias_len : nullptr;
    if (p.sink && rank == 0) {  // one more term of the denominator, exp(sink), without a value
      m = p.sink_logit ? p.sink_logit[h] * kLog2e : 0.f;
      l = 1.f;
    }
    // (a thread whose wait ran out goes on: the barriers below count on every thread, and the block's results are not used)
    if (r.rows > 0) {
      for (int it = 0; it < n_it; ++it) {
        const int k = tile_of(it);
        if (!r.has(k)) continue;
        const int k0 = k * BN;
        const float* tb = nullptr;
        if (BIAS) {  // the biases of the tile's 191 distances, in the base-2 domain with their sign turned; two buffers, one barrier per tile
          float* dst = sTab + (x * 2 + (j & 1)) * kTab;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int y = row + u * 128, d = first - k0 + y - 63;
            if (y < kTab) {
              float v = 0.f;
              if (d >= 0) v = btab ? -kLog2e * btab[min(d, p.bias_len - 1)] : r1 * __log2f(fmaf(r2, static_cast<float>(d), 1.f));
              dst[y] = v;
            }
          }
          named_barrier(1 + x, 128);
          tb = dst + row + 63;
        }
        const uint32_t tmem_s = tmem_s0 + (j & 1) * BN;
        wait(&s_full[x * 2 + (j & 1)], static_cast<uint32_t>((j >> 1) & 1));
        __syncwarp();
        tc_fence_after();
        float sv[BN];
        tmem_ld32(tmem_s, reinterpret_cast<uint32_t(&)[32]>(sv[0]));
        tmem_ld32(tmem_s + 32, reinterpret_cast<uint32_t(&)[32]>(sv[32]));
        tmem_ld_wait();
        const bool need_mask = k0 + BN > end_key || (lo_key > k0 && k0 + BN > keep);
        if (CAP) {  // cap tanh(s scale / cap) as 1 - 2 / (1 + e^(2x)), in the base-2 domain
          // Three uses of the exponential unit per score made a window of 1024 under a cap 96 us; four scores that share one reciprocal: 84 us.  e^(2x) is
          // held below 2^30 (tanh is 1 there), so the product of four stays in range.  (A hidden score that is no number spoils its three neighbours: such a
          // row's sum is no number either, and the row is formed again at the end.)
#pragma unroll
          for (int c = 0; c < BN; c += 4) {
            float d[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] = 1.f + ex2(min_nan(sv[c + i] * cap_in, 30.f));
            const float d01 = d[0] * d[1], d23 = d[2] * d[3], inv = __fdividef(1.f, d01 * d23), i01 = inv * d23, i23 = inv * d01;
            const float q[4] = {i01 * d[1], i01 * d[0], i23 * d[3], i23 * d[2]};
#pragma unroll
            for (int i = 0; i < 4; ++i) sv[c + i] = fmaf(q[i], -2.f * cap_out, cap_out - (BIAS ? tb[-(c + i)] : 0.f));
          }
        } else if (BIAS) {
#pragma unroll
          for (int c = 0; c < BN; ++c) sv[c] = fmaf(sv[c], scale2, -tb[-c]);
        } else {
#pragma unroll
          for (int c = 0; c < BN; c += 2) mul_x2(sv[c], sv[c + 1], scale2);
        }
        if (__any_sync(0xffffffffu, need_mask)) {
          const int a = min(max(lo_key - k0, 0), 64), e = min(max(end_key - k0, 0), 64), kp = min(max(keep - k0, 0), 64);
          auto below = [](int n) { return n >= 64 ? ~0ull : (1ull << n) - 1ull; };
          const unsigned long long vis = below(e) & (~below(a) | below(kp));
          const uint32_t v0 = static_cast<uint32_t>(vis), v1 = static_cast<uint32_t>(vis >> 32);
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (!(v0 & (1u << c))) sv[c] = -INFINITY;
            if (!(v1 & (1u << c))) sv[32 + c] = -INFINITY;
          }
        }
        float mx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          mx[i] = max3(sv[i], sv[4 + i], sv[8 + i]);
#pragma unroll
          for (int c = 12; c + 4 < BN; c += 8) mx[i] = max3(mx[i], sv[c + i], sv[c + 4 + i]);
          mx[i] = fmaxf(mx[i], sv[BN - 4 + i]);
        }
        const float m_new = max3(fmaxf(m, mx[0]), mx[1], fmaxf(mx[2], mx[3]));
        const bool grow = (m_new - m) > kRescale;  // the first finite maximum: +inf; both -inf: NaN, false
        const float alpha = grow ? ex2(m - m_new) : 1.f;
        if (grow) { m = m_new; l *= alpha; }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {
          wait(&o_full[x * 2 + ((j - 1) & 1)], static_cast<uint32_t>(((j - 1) >> 1) & 1));
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int f = 0; f < VP / 32; ++f) {
            uint32_t o[32];
            tmem_ld32(tmem_o + f * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
            tmem_st32(tmem_o + f * 32, o);
          }
        }
        const float neg = m == -INFINITY ? 0.f : -m;   // a row that has seen no key yet: its masked scores give 2^-inf = 0
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          uint32_t hi_p[16], lo_p[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float &p0 = sv[f * 32 + 2 * c], &p1 = sv[f * 32 + 2 * c + 1];
            add_x2(p0, p1, neg, neg);
            p0 = ex2(p0);
            p1 = ex2(p1);
            add_x2(sum[(c & 1) * 2], sum[(c & 1) * 2 + 1], p0, p1);
            hi_p[c] = pack_bf16(p0, p1);
            add_x2(p0, p1, __uint_as_float((hi_p[c] << 16) ^ 0x80000000u), __uint_as_float((hi_p[c] & 0xffff0000u) ^ 0x80000000u));
            lo_p[c] = pack_bf16(p0, p1);
          }
          tmem_st16(tmem_s + f * 16, hi_p);
          tmem_st16(tmem_s + 32 + f * 16, lo_p);
        }
        l += (sum[0] + sum[2]) + (sum[1] + sum[3]);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&p_full[x * 2 + (j & 1)]);
        ++j;
      }
      if (j > 0) wait(&o_full[x * 2 + ((j - 1) & 1)], static_cast<uint32_t>(((j - 1) >> 1) & 1));
      __syncwarp();
      tc_fence_after();
      if (splits == 1) {  // the result: O / l, times the constant and the head's gate
        const int t = off + r.q0 + row;
        const float inv = live ? (l > 0.f ? 1.f / l : 0.f) * out_factor<__nv_bfloat16>(p, t, h) : 0.f;
        __nv_bfloat16* out = out_row<__nv_bfloat16>(p, t, h);
        float zero[4] = {0.f, 0.f, 0.f, 0.f};   // stay 0 over finite numbers
#pragma unroll
        for (int f = 0; f < VP / 32; ++f) {
          uint32_t o[32];
          tmem_ld32(tmem_o + f * 32, o);
          tmem_ld_wait();
          if (live) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint32_t w[4];
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const float x = __uint_as_float(o[v * 8 + 2 * c]) * inv, y = __uint_as_float(o[v * 8 + 2 * c + 1]) * inv;
                zero[c] = fmaf(x, 0.f, fmaf(y, 0.f, zero[c]));
                w[c] = pack_bf16(x, y);
              }
              if (f * 32 + v * 8 < p.vdim) *reinterpret_cast<uint4*>(out + f * 32 + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
        again = (zero[0] + zero[1]) + (zero[2] + zero[3]) != 0.f;
      }
    }
  }
  if (splits > 1) {
    // Merge of the walk's parts through distributed shared memory: block q of the cluster owns the columns [q, q + 1) * VP / splits of every row.
    // After the first barrier every product and copy of every block has completed, so its Q and ring may be written over.
    const int x = (warp >> 2) & 1, row = tid & 127, vc = VP / splits;
    const Range r = x ? rg[1] : rg[0];
    const bool mine = warp < 8 && r.rows > 0;
    float* part = reinterpret_cast<float*>(smem);
    float* ml = reinterpret_cast<float*>(smem + C::kPartBytes);
    __syncwarp();
    cluster_barrier();
    if (*abort_word) m = l = __int_as_float(0x7fffffff);   // (NaN: what the cluster sees of a walk that was given up)
    if (mine) {
      const uint32_t tmem_o = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + C::kColO + x * VP;
      for (int q = 0; q < splits; ++q) st_cluster(cluster_addr(ml + ((rank * 2 + x) * BM + row) * 2, q), m, l);
#pragma unroll 1
      for (int f = 0; f < VP / 32; ++f) {
        uint32_t o[32];
        if (j > 0) {
          tmem_ld32(tmem_o + f * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) o[c] = 0u;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {  // eight columns never straddle two owners
          const int col = f * 32 + g * 8, q = col / vc;
          const uint32_t dst = cluster_addr(part + ((rank * 2 + x) * vc + (col - q * vc)) * BM + row, q);
#pragma unroll
          for (int c = 0; c < 8; ++c) st_cluster(dst + c * BM * 4, __uint_as_float(o[g * 8 + c]));
        }
      }
    }
    __syncwarp();
    cluster_barrier();
    if (mine) {
      float ms[kMaxSplits], ls[kMaxSplits], mt = -INFINITY, lt = 0.f;
#pragma unroll
      for (int q = 0; q < kMaxSplits; ++q) {
        ms[q] = q < splits ? ml[((q * 2 + x) * BM + row) * 2] : -INFINITY;
        ls[q] = q < splits ? ml[((q * 2 + x) * BM + row) * 2 + 1] : 0.f;
        mt = fmaxf(mt, ms[q]);
      }
#pragma unroll
      for (int q = 0; q < kMaxSplits; ++q) {
        ms[q] = ms[q] == -INFINITY ? 0.f : ex2(ms[q] - mt);
        lt = fmaf(ls[q], ms[q], lt);
      }
      const bool live = row < r.rows;
      const int t = off + r.q0 + row;
      const float inv = live ? (lt > 0.f ? 1.f / lt : 0.f) * out_factor<__nv_bfloat16>(p, t, h) : 0.f;
      __nv_bfloat16* out = out_row<__nv_bfloat16>(p, t, h) + rank * vc;
      float zero[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int c0 = 0; c0 < vc; c0 += 8) {
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < kMaxSplits; ++q)
          if (q < splits) {
            const float* src = part + ((q * 2 + x) * vc + c0) * BM + row;
#pragma unroll
            for (int c = 0; c < 8; ++c) a[c] = fmaf(src[c * BM], ms[q], a[c]);
          }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          a[c] *= inv;
          zero[c] = fmaf(a[c], 0.f, zero[c]);
        }
        if (live && rank * vc + c0 < p.vdim)
          *reinterpret_cast<uint4*>(out + c0) = make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
      }
      again = live && ((zero[0] + zero[1]) + (zero[2] + zero[3])) + ((zero[4] + zero[5]) + (zero[6] + zero[7])) != 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();   // TMEM has been read
  if (*abort_word) {   // a wait ran out: the block is counted, and its rows are formed again
    again = warp < 8 && (tid & 127) < ((warp >> 2) ? rg[1].rows : rg[0].rows);
    if (tid == 0) atomicAdd(&attn_tc5_timeouts, 1);
  }
  if (warp < 8) {   // rows whose result is not finite: from the keys they see alone (this block's columns of them)
    const int q0 = (warp >> 2) ? rg[1].q0 : rg[0].q0, cols = VP / splits, c0 = splits > 1 ? rank * cols : 0;
    for (uint32_t w = __ballot_sync(0xffffffffu, again && c0 < p.vdim); w; w &= w - 1) {
      const int row = q0 + (warp & 3) * 32 + __ffs(w) - 1;
      attn_row_again_call<__nv_bfloat16>(p, b, h, off + row, pos0 + row, c0, min(cols, p.vdim - c0));
    }
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_free<512>(tmem_base);
  }
}

// How a launch is cut: pairs of neighbouring tiles or of tiles from both ends, and the blocks of a cluster that share a walk.  Times in microseconds as
// measured on B200: a tile of both halves 1.4 (2.0 with a cap, whose tanh keeps the exponential unit busy), of one half alone 1.2; a block's set-up and end
// 6.5, with a merge 9.5 to 11.5; a launch of more than one wave ends 15 % behind its average.  Examples (16 heads; neighbours, ends, and clusters of 2, 4, 8 with
// the better of the two): 2048 new tokens 54 / 48 / 44 / 72 / 140, 1024: 31 / 27 / 22 / 31 / 71, 256 behind 4000: 103 / 103 / 60 / 37 / 50, 4096: 99 / 134 / 125 / 184 / 316.
struct Plan {
  int ends = 0, splits = 1;
  double best = 1e30;
  // slots[i]: blocks that run side by side in clusters of 2^i
  Plan(const pcs_attn_params& p, int dp, int vp, const int (&slots)[4]) {
    const bool ranged = p.window > 0 || p.chunk > 0;
    const double step = (1.4 + (p.softcap > 0.f ? 0.6 : 0.0)) * fmax(0.5, (dp + 2 * vp) / 384.0), single = 0.85 * step;
    const double over[4] = {6.5, 9.5, 10.0, 11.5};
    const int keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap, n = (p.max_len + BM - 1) / BM, pairs = (n + 1) / 2;
    const double blocks = fmin(static_cast<double>(p.n_seqs) * pairs, p.n_tokens / (2.0 * BM) + p.n_seqs) * p.n_heads;
    auto walk = [&](int t) {  // key tiles of query tile t of the longest entry
      double k = fmax(fmin(keys, keys - p.max_len + (t + 1.0) * BM), 1.0);
      if (p.window > 0) k = fmin(k, p.window + BM + fmax(p.keep_first, 0) + BN);
      if (p.chunk > 0) k = fmin(k, p.chunk + BN);
      return ceil(k / BN);
    };
    for (int e = 0; e < (ranged || n == 1 ? 1 : 2); ++e) {
      double longest = 0.0, sum = 0.0;
      for (int m = 0; m < pairs; ++m) {
        const int t1 = e ? m : 2 * m, t0 = e ? n - 1 - m : (2 * m + 1 < n ? 2 * m + 1 : n - 1);   // t0 walks at least as far
        const double w1 = t1 == t0 ? 0.0 : walk(t1), c = w1 * step + (walk(t0) - w1) * single;
        longest = fmax(longest, c);
        sum += c;
      }
      const double total = sum / pairs * blocks;
      for (int i = 0; i < 4; ++i) {
        const int s = 1 << i;
        if (slots[i] < s) continue;
        double t = longest / s + over[i];
        if (blocks * s > slots[i]) t = fmax(t, 1.15 * (total + blocks * s * over[i]) / slots[i]);
        if (t < best) { best = t; ends = e; splits = s; }
      }
    }
  }
};

template <int DP, int VP, bool BIAS, bool CAP>
int launch(const pcs_attn_params& p, cudaStream_t st) {
  using C = Cfg<DP, VP>;
  auto kernel = attn_tc5_kernel<DP, VP, BIAS, CAP>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  struct Info { int slots[4]; };   // blocks that run side by side in clusters of 2^i
  static PerDevice<Info> per_device;
  const Info* info;
  if (int rc = per_device.get(&info, [&](Info& x) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem);
        for (int i = 0; i < 4 && err == cudaSuccess; ++i) {
          int n = 0;
          attr[0].val.clusterDim.x = 1u << i;
          cfg.gridDim = dim3(1u << i);
          err = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
          x.slots[i] = n << i;
        }
        return err;
      }))
    return rc;
  const unsigned long long D = p.dim, V = p.vdim, cap = p.cap, H = p.n_heads;
  const unsigned long long planes = pool_planes(p);
  CUtensorMap mq, mk, mv;
  if (int rc = tensor_map_bf16(&mq, p.q, {D, H, static_cast<unsigned long long>(p.n_tokens)}, {D * 2, H * D * 2}, {64, 1, BM})) return rc;
  if (int rc = tensor_map_bf16(&mk, p.k_pool, {D, cap, planes}, {D * 2, cap * D * 2}, {64, BN, 1})) return rc;
  if (int rc = tensor_map_bf16(&mv, p.v_pool, {V, cap, planes}, {V * 2, cap * V * 2}, {64, BN, 1})) return rc;
  const Plan plan(p, DP, VP, info->slots);
  cfg.gridDim = dim3(static_cast<unsigned>(((p.max_len + BM - 1) / BM + 1) / 2) * p.n_seqs * p.n_heads * plan.splits);
  attr[0].val.clusterDim.x = static_cast<unsigned>(plan.splits);
  PCS_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, mq, mk, mv, p, plan.ends | ((p.impl & 3) == 3 ? 2 : 0), plan.splits));
  count_launch();
  return PCS_OK;
}

template <int DP, int VP>
int launch_opt(const pcs_attn_params& p, cudaStream_t st) {
  const bool bias = p.bias_r1 || p.bias_table, cap = p.softcap > 0.f;
  if (cap) return bias ? launch<DP, VP, true, true>(p, st) : launch<DP, VP, false, true>(p, st);
  return bias ? launch<DP, VP, true, false>(p, st) : launch<DP, VP, false, false>(p, st);
}

}  // namespace

// Entries of at most one tile of query rows, each of which leaves half of its block idle: where the mma.sync kernel (64 rows per block, three blocks per SM) is
// expected to be faster.  Both sides in microseconds, from 564 shapes of 16 to 128 new tokens x 1 to 48 entries behind 0 to 1000 stored (B200): a block here takes
// 3.4 to 4.1 and 1.1 per key tile, one at a time on an SM; there a key tile takes an SM 1.8 to 4.5 with one to three blocks on it.  At 16 heads of 64, mma.sync / tcgen05:
// 16 x 48 entries 12 / 31, 64 x 16 8.3 / 12.4, 64 x 48 behind 500 60 / 81, 64 behind 500 22 / 11; of 128: 64 x 48 21 / 33, 16 x 16 10 / 15, 64 x 48 behind 500 92 / 90.
bool short_entries(const pcs_attn_params& p) {
  if (p.max_len > BM || p.dim > 128) return false;
  constexpr int kSMs = 148, kOld = 64;
  const int wide = (p.dim > 64) + (p.vdim > 64);
  static const double kBase[3] = {4.6, 5.0, 6.0}, kTile[3][4] = {{0.0, 1.8, 2.1, 2.6}, {0.0, 1.95, 2.55, 3.5}, {0.0, 2.45, 3.2, 4.46}};
  const bool cap = p.softcap > 0.f;
  const double set_up = wide ? 4.1 : 3.4, tile = (wide ? 1.16 : 1.09) + (cap ? 0.45 : 0.0), merge[4] = {0.0, 3.0, 3.5, 5.0};
  double keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap;
  if (p.window > 0) keys = fmin(keys, p.window + BM + fmax(p.keep_first, 0) + BN);
  if (p.chunk > 0) keys = fmin(keys, p.chunk + BN);
  const double tiles = ceil(fmax(keys, 1.0) / BN);
  const long long blocks = static_cast<long long>(p.n_seqs) * p.n_heads;
  double here = 3.5 + (blocks + kSMs - 1) / kSMs * (set_up + tile * tiles);
  for (int i = 1; i < 4; ++i)
    if (blocks << i <= kSMs) here = fmin(here, 3.5 + set_up + merge[i] + tile * ceil(tiles / (1 << i)));
  long long there = blocks * ((p.max_len + kOld - 1) / kOld);
  const long long most = (p.n_tokens / kOld + static_cast<long long>(p.n_seqs)) * p.n_heads;
  if (there > most) there = most;
  const long long full = there / (3 * kSMs), rest = there % (3 * kSMs);
  const double old = kBase[wide] + tiles * (cap ? 1.07 : 1.0) * (full * kTile[wide][3] + kTile[wide][(rest + kSMs - 1) / kSMs]);
  return old < 0.95 * here;
}

namespace {

// Blocks of known costs, in launch order, on SMs that each take the next one when they fall free
class Schedule {
 public:
  explicit Schedule(int sms) { free_[0] = Level{0.0, sms}; }
  void run(double cost, long long blocks) {
    while (blocks > 0) {
      Level& first = free_[head_];
      const double end = first.at + cost;
      const int n = static_cast<int>(blocks < first.n ? blocks : first.n);
      blocks -= n;
      if ((first.n -= n) == 0) ++head_;
      int i = tail_;
      while (i > head_ && free_[i - 1].at > end) --i;
      if (i > head_ && end - free_[i - 1].at < kSame) {
        free_[i - 1].n += n;
      } else {
        if (tail_ == kRoom) {   // to the front
          for (int k = head_; k < tail_; ++k) free_[k - head_] = free_[k];
          i -= head_;
          tail_ -= head_;
          head_ = 0;
        }
        for (int k = tail_++; k > i; --k) free_[k] = free_[k - 1];
        free_[i] = Level{end, n};
      }
      if (end > end_) end_ = end;
    }
  }
  double end() const { return end_; }

 private:
  struct Level { double at; int n; };        // n SMs fall free
  static constexpr double kSame = 0.25;      // us
  static constexpr int kRoom = 4 * 148;      // (never more than 148 levels at a time)
  Level free_[kRoom];                        // in order of time, from head_ to tail_
  int head_ = 0, tail_ = 1;
  double end_ = 0.0;
};

}  // namespace

// What a launch of heads of 65 to 192 / 65 to 128 elements is expected to take here, or in the mma.sync kernel where short_entries() prefers that one: us on B200, the entries'
// walks one by one.  The constants are fitted to launches of ten key tiles of 128 per SM and more (1000 of them: one to 256 entries of 16 to 7000 tokens behind 0 to 8000, many of them
// uneven; 8 to 32 heads): 90 % lie within 7 %, mma.sync within 15 %.
double attn_tc5_expected(const pcs_attn_params& p, const Entries& entries) {
  const bool cap = p.softcap > 0.f, bias = p.bias_r1 || p.bias_table, ranged = p.window > 0 || p.chunk > 0, wide = p.dim > 128;
  if (short_entries(p)) {
    constexpr int kOld = 64;
    double blocks = 0.0, tiles = 0.0, longest = 0.0;
    for (int b = 0; b < entries.n; ++b) {
      const int pos0 = entries.pos_of(b), len = entries.len_of(b);
      for (int t = 0; t < len; t += kOld) {
        const int n = Walk<BN>(p, pos0, len, t, t + kOld < len ? t + kOld : len).n;
        blocks += p.n_heads;
        tiles += static_cast<double>(n) * p.n_heads;
        if (n > longest) longest = n;
      }
    }
    constexpr double kSlots = 3 * 148;
    return 2.7 + (4.4 * blocks + (4.1 + (cap ? 0.5 : 0.0) + (bias ? 0.3 : 0.0)) * tiles) / kSlots + 1.7 * longest;
  }
  const int slots[4] = {148, 148, 144, 128}, n_max = (p.max_len + BM - 1) / BM, pairs = (n_max + 1) / 2;
  const Plan plan(p, wide ? 192 : 128, 128, slots);
  const double both = 1.46 + (cap ? 0.40 : 0.0) + (bias ? 0.07 : 0.0) + (wide ? 0.15 : 0.0);   // a tile of both halves, of one
  const double single = 1.18 + (cap ? 0.27 : bias ? 0.04 : 0.0) + (wide ? 0.15 : 0.0);
  const double over = plan.splits == 1 ? 4.6 : plan.splits == 2 ? 8.0 : plan.splits == 4 ? 8.5 : 10.0;   // a block's set-up and end
  Schedule schedule((plan.splits == 1 ? 148 : plan.splits == 2 ? slots[1] : plan.splits == 4 ? slots[2] : slots[3]) / plan.splits);
  double cost = 0.0;
  long long blocks = 0;   // of that cost, in a row
  for (int m = 0; m < pairs; ++m) {
    for (int b = 0; b < entries.n; ++b) {
      const int pos0 = entries.pos_of(b), len = entries.len_of(b), n = (len + BM - 1) / BM;
      const int t1 = plan.ends ? n - 1 - m : 2 * (pairs - 1 - m) + 1, t0 = plan.ends ? m : t1 - 1;   // t0 walks no further than t1
      if (plan.ends ? t0 > t1 : t0 >= n) continue;
      auto walk = [&](int from, int tile) { return Walk<BN>(p, pos0, len, from * BM, (tile + 1) * BM < len ? (tile + 1) * BM : len).n; };
      double c;
      if (t1 >= n || t0 == t1) {
        c = walk(t0, t0) * single;
      } else if (ranged) {
        c = walk(t0, t1) * both;
      } else {
        const int common = walk(t0, t0);
        c = common * both + (walk(t1, t1) - common) * single;
      }
      c = over + c / plan.splits;
      if (c != cost) {
        schedule.run(cost, blocks);
        cost = c;
        blocks = 0;
      }
      blocks += p.n_heads;
    }
  }
  schedule.run(cost, blocks);
  return 6.6 + schedule.end();
}

// Sixteen or more new tokens of some entry, heads of up to 192 / 128 elements in 16-byte pieces
int launch_attn_tc5(const pcs_attn_params& p, cudaStream_t st, bool* handled) {
  *handled = false;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (dense_rows_off_boxes(p)) return PCS_OK;
  if (p.dtype != PCS_BF16 || p.max_len < 16 || (p.v_row_stride != 0 && p.v_row_stride != p.vdim) || p.dim % 8 != 0 || p.vdim % 8 != 0 || p.dim > 192 || p.vdim > 128)
    return PCS_OK;
  if (!p.seq_pos0 || !p.seq_len || !p.seq_off || !al16(p.q) || !al16(p.k_pool) || !al16(p.v_pool) || !al16(p.out) || p.out_stride % 8 != 0) return PCS_OK;
  if (((p.max_len + BM - 1LL) / BM + 1) / 2 * p.n_seqs * p.n_heads * kMaxSplits > 0x7fffffffLL || short_entries(p)) return PCS_OK;
  *handled = true;
  if (p.vdim <= 64) {
    if (p.dim <= 64) return launch_opt<64, 64>(p, st);
    if (p.dim <= 128) return launch_opt<128, 64>(p, st);
    return launch_opt<192, 64>(p, st);
  }
  if (p.dim <= 64) return launch_opt<64, 128>(p, st);
  if (p.dim <= 128) return launch_opt<128, 128>(p, st);
  return launch_opt<192, 128>(p, st);
}

int attn_tc5w_timeouts_so_far();   // of the form for much work

}  // namespace pcs

// blocks of the tcgen05 attention kernel one of whose bounded waits ran out so far (0 in a working system; their rows were formed without tensor cores);
// synchronises
PCS_API int pcs_attn_timeouts(void) {
  int n = -1;
  const int more = pcs::attn_tc5w_timeouts_so_far();
  if (more < 0 || cudaMemcpyFromSymbol(&n, pcs::attn_tc5_timeouts, sizeof(n)) != cudaSuccess) return -1;
  return n + more;
}
