// tcgen05 attention over the slot pool for prompts of much work (bfloat16 storage, 32-bit scores, softmax and accumulation): a persistent form of
// seq_attn_tc5.cu, which serves the others.
//
// An item of work = two tiles ("halves") of 128 query rows that walk the same K / V tiles of 128 keys: the same 128 new tokens under two heads of one K/V
// group.
//
//   TMA warp      describes the items and their tiles for the others; Q, K and V through two rings (3-d tensor maps over the pool, 128-byte swizzle)
//   MMA warps     one per half: S = Q K_j^T into TMEM;  O += P_hi V_j + P_lo V_j  with P in TMEM over S
//   softmax       two warpgroups per half, a thread one query row and 64 of a tile's 128 keys: scale / cap / bias / masks in the base-2 domain, online
//                 softmax (the row's two threads exchange their maxima), P written over S as two bfloat16 operands, 32 keys at a time
//
// The halves alternate: one's products run under the other's softmax.  Tiles of 128 keys, because a 128 x 64 x 16 product reads 6 KB of shared memory in the
// time of 32 cycles' worth of multiply-adds (48 cycles), a 128 x 128 x 16 one 8 KB in 64.  TMEM: S 2 x 128 columns, O 2 x vdim columns.
//
// The 32-bit weights enter the tensor cores as P = hi + lo (hi = bf16(P), lo = bf16(P - hi)), so ~16 bits of each are kept: three 128 x 128 x 128
// products per tile and half where a plain flash kernel has two.  The accumulator is rescaled only when
// a row's maximum grew by more than 2^8 (P then stays below 2^8, exact in the same 16 bits).  The products multiply hidden keys of a tile by 0: a row
// whose result is not finite is formed again from the keys it sees (attn_row_again).
//
// The items' tiles, end to end, are cut into as many equal runs as there are SMs.  A block works through its run; where an item is
// cut, the block that has its first tiles adds the others' (m, l, O), which pass through the caller's scratch.  A block's first
// piece is the one that others wait for, and they wait for blocks of lower index only, so the wait ends however few blocks run side by side.
//
// What bounds it (B200, dim = vdim = 128, an item per SM over 8 to 48 tiles, 1.96 GHz): 5100 cycles per key tile of both halves, 5900 with a distance bias, 7900 under a cap.  The
// 48 products keep the tensor pipe busy for 3600 of them (75 each); the rest is the chain scores - softmax - products of one half behind the other's.  An item costs another
// 8000 (its first scores, its result), each run that shares it 3 us, the launch 14 us.  So it pays from some ten tiles per SM on, and where the other form's whole
// walks leave SMs idle (pays(), below).  Against seq_attn_tc5.cu, us:
//   four continued prompts, window 1024, cap  84.2 -> 66.7      3102 tokens behind 205, 12 heads, bias              100 -> 77
//   6144 and 2311 new tokens                   280 -> 272       692, 416, 1671, 1876, one behind 2479; 8 of 192    116 -> 77
#include <atomic>
#include <chrono>

#include "seq_attn.cuh"
#include "seq_mma.cuh"
#include "seq_tc5.cuh"

namespace pcs {

namespace {

constexpr int BM = 128, BN = 128, HB = BN / 2;
constexpr int kThreads = 640;  // four softmax warpgroups (two of each half), TMA warp 16, MMA warps 17 and 18, a warp that publishes partial results
constexpr int kTmaWarp = 16, kMmaWarp = 17;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescale = 8.0f;
constexpr int kTab = 256;      // distances of a tile pair of 128 rows and 128 keys (255)
constexpr int kMaxStreamSeqs = 256;
// The TMA warp describes a tile for the others: which 64 keys it sees any of (bits 0, 1), the last tile of a piece, of the run.  It is at
// most KS + 2 tiles ahead of the softmax;
constexpr int kInfo = 8, kLast = 16, kEnd = 32;
// and a piece: it is at most three ahead (Q of the next but one waits for the scores of the next one, and these for the softmax)
constexpr int kPieces = 4;
// Cost of a piece of the stream: 4 per key tile, and what an item costs beside its tiles (one more: its Q, its first scores, its result).  A run is at
// least three tiles long (below, moving partial results costs more than it brings), and no piece is shorter than two.
constexpr int kTileCost = 4, kItemCost = 4, kMinRun = 12, kMinPiece = 2;

// What the two threads of a row exchange, arrays of BM numbers: the maxima of a tile (two buffers in turn), and behind them the sums of a piece.  Nothing stands between
// the read of the last tile's maxima and the store of the sums, so the two never share an array.
constexpr int kExchange = 12;
constexpr int max_array(int tile, int half, int part) { return ((tile & 1) * 2 + half) * 2 + part; }
constexpr int sum_array(int half, int part) { return 8 + half * 2 + part; }
constexpr bool exchange_apart() {
  int used[kExchange] = {};
  for (int half = 0; half < 2; ++half)
    for (int part = 0; part < 2; ++part) {
      ++used[max_array(0, half, part)];
      ++used[max_array(1, half, part)];
      ++used[sum_array(half, part)];
    }
  for (int n : used)
    if (n != 1) return false;
  return true;
}
static_assert(exchange_apart(), "maxima and sums of a row in arrays of their own");

__device__ int attn_tc5w_timeouts;  // blocks one of whose waits ran out

template <int DP, int VP>
struct Cfg {
  static constexpr int kQBytes = BM * DP * 2, kKBytes = BN * DP * 2, kVBytes = BN * VP * 2;
  static constexpr int kTabBytes = 2 * 2 * kTab * 4, kMaxBytes = kExchange * BM * 4;
  static constexpr int KS = DP > 128 ? 1 : 2, VS = 2;   // stages of the rings (rows of more than 128: what fits)
  static constexpr int kOffK = 2 * kQBytes, kOffV = kOffK + KS * kKBytes, kRing = kOffV + VS * kVBytes;
  static constexpr int kOffTab = kRing;
  static constexpr int kOffMax = kOffTab + kTabBytes, kOffBars = kOffMax + kMaxBytes;
  static constexpr int kSmem = kOffBars + 1024;
  static_assert(kSmem <= 227 * 1024, "shared memory of a block");
  static constexpr int kColO = 256;
  // a run's slot of the scratch: flags and end of the piece, (m, l) per half and row, O in pieces of 16 rows x 32 columns
  static constexpr int kSlotBytes = 64 + 2 * BM * 8 + 2 * BM * VP * 4;
};

// four neighbouring lanes: lane s gets number s of every one of them, in their order
__device__ __forceinline__ void transpose4(uint32_t (&w)[4], int s) {
  const bool a = s & 1, b = s & 2;
  uint32_t x = __shfl_xor_sync(0xffffffffu, a ? w[0] : w[1], 1), y = __shfl_xor_sync(0xffffffffu, a ? w[2] : w[3], 1);
  if (a) { w[0] = x; w[2] = y; } else { w[1] = x; w[3] = y; }
  x = __shfl_xor_sync(0xffffffffu, b ? w[0] : w[2], 2);
  y = __shfl_xor_sync(0xffffffffu, b ? w[1] : w[3], 2);
  if (b) { w[0] = x; w[1] = y; } else { w[2] = x; w[3] = y; }
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_flag(unsigned long long* p, unsigned long long v) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory"); }

// How the launch is cut
struct Cut {
  int give_up;                // tests: a warp of every block gives up
  unsigned char* slots;       // the scratch
  unsigned long long nonce;   // what this launch's flags hold, or kGivenUp more: nothing was stored
};
constexpr unsigned long long kGivenUp = 1;   // (nonces are odd)

// A place in the stream: entry, unit (a tile of new tokens), item of the unit (two heads), key tile
struct Place { int b, u, i, tile; };

__device__ __forceinline__ int units_of(int len) { return (len + BM - 1) / BM; }
__device__ __forceinline__ int unit_tiles(const pcs_attn_params& p, int pos0, int len, int u) { return Walk<BN>(p, pos0, len, u * BM, min(len, (u + 1) * BM)).n; }

// One warp: where the stream is cut at cost `at`; first[b]: cost of the entries before b
__device__ Place locate(const pcs_attn_params& p, const long long* first, long long at) {
  const int lane = threadIdx.x & 31, per = p.n_heads / 2;
  Place c = {p.n_seqs, 0, 0, 0};
  if (at >= first[p.n_seqs]) return c;
  int lo = 0, hi = p.n_seqs;   // first[lo] <= at < first[hi]
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (first[m] <= at) lo = m;
    else hi = m;
  }
  c.b = lo;
  const int len = p.seq_len[lo], pos0 = p.seq_pos0[lo], units = units_of(len);
  long long rem = at - first[lo];
  for (int u0 = 0; u0 < units; u0 += 32) {
    const int n = u0 + lane < units ? unit_tiles(p, pos0, len, u0 + lane) : 0;
    const long long mine = u0 + lane < units ? static_cast<long long>(n * kTileCost + kItemCost) * per : 0;
    long long sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long x = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += x;
    }
    const unsigned here = __ballot_sync(0xffffffffu, rem < sum);
    if (here) {
      const int src = __ffs(here) - 1, tiles = __shfl_sync(0xffffffffu, n, src), cost = tiles * kTileCost + kItemCost;
      rem -= __shfl_sync(0xffffffffu, sum - mine, src);
      c.u = u0 + src;
      c.i = static_cast<int>(rem / cost);
      const int r = static_cast<int>(rem - static_cast<long long>(c.i) * cost);
      c.tile = r < kItemCost ? 0 : (r - kItemCost + kTileCost / 2) / kTileCost;
      if (c.tile < kMinPiece) c.tile = 0;
      if (c.tile > tiles - kMinPiece) c.tile = tiles > kMinPiece ? tiles : r * 2 < cost ? 0 : tiles;
      if (c.tile == tiles) {   // the end of an item is the start of the next one
        c.tile = 0;
        if (++c.i == per) {
          c.i = 0;
          if (++c.u == units) {
            c.u = 0;
            do ++c.b; while (c.b < p.n_seqs && p.seq_len[c.b] <= 0);
          }
        }
      }
      return c;
    }
    rem -= __shfl_sync(0xffffffffu, sum, 31);
  }
  return c;
}

// One piece of a block's run: an item's tiles [it0, it1)
struct Piece {
  int b, h[2], q0, rows, len, pos0, off, plane, total, keep, it0, it1;
  Walk<BN> w;
  __device__ __forceinline__ Piece(const pcs_attn_params& p, const Place& at, const Place& end)
      : b(at.b), q0(at.u * BM), len(p.seq_len[at.b]), pos0(p.seq_pos0[at.b]), off(p.seq_off[at.b]), w(p, pos0, len, at.u * BM, min(len, (at.u + 1) * BM)) {
    h[0] = 2 * at.i;
    h[1] = 2 * at.i + 1;
    rows = max(0, min(BM, len - q0));
    plane = (p.pool_slot ? p.pool_slot[b] : p.seq_slot[b]) * p.n_kv_heads + h[0] / (p.n_heads / p.n_kv_heads);
    total = pos0 + len;
    keep = p.window > 0 ? min(max(p.keep_first, 0), total) : 0;
    it0 = at.tile;
    it1 = at.b == end.b && at.u == end.u && at.i == end.i ? end.tile : w.n;
  }
  // which 64 keys of the tile starting at k0 some row sees any of (bit 0: the first)
  __device__ __forceinline__ int sees(const pcs_attn_params& p, int k0) const {
    const int first = pos0 + q0, last = first + rows;
    const int lo = p.window > 0 ? max(0, first - p.window + 1) : p.chunk > 0 ? first / p.chunk * p.chunk : 0;
    auto part = [&](int k) { return rows > 0 && k < last && (k + HB > lo || k < keep); };
    return (part(k0) ? 1 : 0) | (part(k0 + HB) ? 2 : 0);
  }
};

template <int DP, int VP, bool BIAS, bool CAP>
__global__ void __launch_bounds__(kThreads, 1) attn_tc5w_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                               const __grid_constant__ CUtensorMap map_v, const __grid_constant__ pcs_attn_params p,
                                                               const __grid_constant__ Cut cut) {
  using C = Cfg<DP, VP>;
  constexpr int KS = C::KS, VS = C::VS;
  extern __shared__ __align__(1024) unsigned char smem[];   // (all addresses in it are constants of the code)
  unsigned char *sQ = smem, *sK = smem + C::kOffK, *sV = smem + C::kOffV;
  float* sTab = reinterpret_cast<float*>(smem + C::kOffTab);
  float* sMax = reinterpret_cast<float*>(smem + C::kOffMax);   // [max_array or sum_array][row]
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + C::kOffBars);
  uint64_t* q_empty = q_full + 1;
  uint64_t* ragged = q_full + 2;          // the last K / V tile of a sequence, before its rows past the end are cleared
  uint64_t* k_full = q_full + 3;          // [KS]
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;        // [VS]
  uint64_t* v_empty = v_full + VS;
  uint64_t* s_full = v_empty + VS;        // [2 halves] each:
  uint64_t* p_full = s_full + 2;          // [half][the first 32 keys of either 64, the others]
  uint64_t* o_full = p_full + 4;
  uint64_t* o_free = o_full + 2;
  uint64_t* drained = o_free + 2;         // every product has ended
  uint64_t* turn = drained + 2;           // the other half's batch is out
  uint64_t* stored = turn + 2;            // the partial result of the run's first piece is out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stored + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* redo_word = reinterpret_cast<volatile int*>(tmem_slot + 2);   // some result is not finite
  Place* ends = reinterpret_cast<Place*>(tmem_slot + 3);   // [2] of the block's run
  volatile int* run_word = reinterpret_cast<volatile int*>(ends + 2);
  volatile int* left = run_word + 1;   // [3 barriers][2 of each][2 halves] a thread of the half has given up
  int2* info = reinterpret_cast<int2*>(smem + C::kOffBars + 384);       // [kInfo] of a key tile: its first key, what is to be done with it
  Piece* pieces = reinterpret_cast<Piece*>(smem + C::kOffBars + 448);   // [kPieces] of the run, written by the TMA warp
  static_assert(448 + kPieces * sizeof(Piece) <= 1024 && (3 + 2 * KS + 2 * VS + 16) * 8 + 12 + 32 + 4 + 48 <= 384, "room behind the barriers");

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int per_unit = p.n_heads / 2;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, abort_word); };

  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);
    mbar_init(ragged, 1);
    for (int s = 0; s < KS; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 2);
    }
    for (int s = 0; s < VS; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[2 * i], 256);
      mbar_init(&p_full[2 * i + 1], 256);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_free[i], 256);
      mbar_init(&drained[i], 1);
      mbar_init(&turn[i], 1);
      mbar_init(&stored[i], 256);
    }
    *abort_word = 0;
    *redo_word = 0;
    for (int i = 0; i < 12; ++i) left[i] = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) tmem_alloc<512>(tmem_slot);
  if (warp == 10 && lane < p.n_seqs) {   // (what the roles read of an entry, into this SM's cache)
    int touched;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(touched) : "l"(p.seq_off + lane));
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(touched) : "l"((p.pool_slot ? p.pool_slot : p.seq_slot) + lane));
  }
  // ---- this block's run ----
  {
    long long* first = reinterpret_cast<long long*>(sK);
    auto cost_of = [&](int b) {   // of an entry, by one warp
      const int len = p.seq_len[b], pos0 = p.seq_pos0[b], units = units_of(len);
      long long c = 0;
      for (int u = lane; u < units; u += 32) c += unit_tiles(p, pos0, len, u) * kTileCost + kItemCost;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      return c * per_unit;
    };
    if (p.n_seqs <= 4) {   // the two warps that need them find the sums themselves
      if (warp < 2) {
        first += warp * (kMaxStreamSeqs + 1);
        long long c = 0;
        for (int b = 0; b < p.n_seqs; ++b) {
          if (lane == 0) first[b] = c;
          c += cost_of(b);
        }
        if (lane == 0) first[p.n_seqs] = c;
        __syncwarp();
      }
    } else {
      for (int b = warp; b < p.n_seqs; b += kThreads / 32) {
        const long long c = cost_of(b);
        if (lane == 0) first[b + 1] = c;
      }
      __syncthreads();
      if (warp == 0) {
        long long before = 0;
        for (int b0 = 0; b0 < p.n_seqs; b0 += 32) {
          long long c = b0 + lane < p.n_seqs ? first[b0 + lane + 1] : 0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, c, o);
            if (lane >= o) c += y;
          }
          if (b0 + lane < p.n_seqs) first[b0 + lane + 1] = before + c;
          before += __shfl_sync(0xffffffffu, c, 31);
        }
        if (lane == 0) first[0] = 0;
      }
      __syncthreads();
    }
    if (warp < 2) {
      const long long total = first[p.n_seqs];
      const int runs = static_cast<int>(max(1ll, min(static_cast<long long>(gridDim.x), total / kMinRun)));
      const int run = runs - 1 - static_cast<int>(blockIdx.x);   // (the waits of a merge are for later runs)
      Place c = {0, 0, 0, 0};
      if (run >= 0) c = locate(p, first, total * (run + warp) / runs);
      if (lane == 0) {
        ends[warp] = c;
        if (warp == 0) *run_word = run;
      }
    }
    fence_proxy_async_smem();   // (copies write where `first` was)
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the run piece by piece: the place behind a piece, whether there is one
  auto more = [&](const Place& a) {
    const Place e = ends[1];
    return a.b != e.b || a.u != e.u || a.i != e.i || a.tile != e.tile;
  };
  auto advance = [&](Place& a, const Piece& c) {
    if (c.it1 < c.w.n) { a.tile = c.it1; return; }
    a.tile = 0;
    if (++a.i == per_unit) {
      a.i = 0;
      if (++a.u == units_of(c.len)) {
        a.u = 0;
        do ++a.b; while (a.b < p.n_seqs && p.seq_len[a.b] <= 0);
      }
    }
  };
  auto piece_of = [&](const Place& a) { return Piece(p, a, ends[1]); };
  const bool any = more(ends[0]);
  // (tests) the TMA warp, one of the MMA warps or the one that publishes gives up, as if its wait had run out: at some tile of the run's first piece, or at once
  int drop_at = -1;
  if (cut.give_up && any && warp == kTmaWarp + static_cast<int>(blockIdx.x % 4)) {
    const Piece c = piece_of(ends[0]);
    drop_at = min(static_cast<int>(blockIdx.x >> 2 & 7), c.it1 - c.it0 - 1);
  }

  if (warp >= kTmaWarp) {
    if (warp == kTmaWarp) {
      // ===================== TMA producer =====================
      int n_k = 0, n_v = 0, n_q = 0, n_piece = 0, n_ragged = 0, ragged_at = -1;   // issued so far; the tile that passes the `ragged` barrier
      bool ok = true;
      for (Place a = ends[0]; ok && more(a);) {
        const Piece c = piece_of(a);
        Place after = a;
        advance(after, c);
        const bool last_piece = !more(after);
        if (lane == 0) pieces[n_piece % kPieces] = c;
        ++n_piece;
        auto load_q = [&]() {
          if (n_q > 0 && !__all_sync(0xffffffffu, wait(q_empty, static_cast<uint32_t>((n_q - 1) & 1)))) return false;
          if (lane == 0) {
            mbar_expect_tx(q_full, 2 * C::kQBytes);
            for (int x = 0; x < 2; ++x)
              for (int f = 0; f < DP / 64; ++f) tma_load_3d(sQ + x * C::kQBytes + f * BM * 128, &map_q, q_full, f * 64, c.h[x], c.off + c.q0);
          }
          ++n_q;
          return true;
        };
        const bool begins = n_q == 0;
        if (begins) load_q();
        for (int it = c.it0; it < c.it1; ++it) {
          const int ks = n_k % KS, vs = n_v % VS, key0 = c.w.tile(it) * BN, left_keys = c.total - key0;  // keys of this tile that exist
          if (n_k == drop_at) {
            *abort_word = 1;
            ok = false;
            break;
          }
          const int what = c.sees(p, key0) | (it + 1 == c.it1 ? kLast : 0) | (it + 1 == c.it1 && last_piece ? kEnd : 0);
          bool free = true;
          if (n_k >= KS) free = wait(&k_empty[ks], static_cast<uint32_t>((n_k / KS - 1) & 1));
          if (left_keys < BN && free && n_v >= VS) free = wait(&v_empty[vs], static_cast<uint32_t>((n_v / VS - 1) & 1));
          if (!__all_sync(0xffffffffu, free)) { ok = false; break; }
          bool q_due = it == c.it0 && !begins;   // (behind the piece's first keys, as Q's place is free later than theirs; a ragged tile is one transaction)
          if (q_due && left_keys < BN) {
            if (!load_q()) { ok = false; break; }
            q_due = false;
          }
          unsigned char *dk = sK + ks * C::kKBytes, *dv = sV + vs * C::kVBytes;
          uint64_t *bk = left_keys < BN ? ragged : &k_full[ks], *bv = left_keys < BN ? ragged : &v_full[vs];
          if (lane == 0) {
            info[n_k % kInfo] = make_int2(key0, what);
            mbar_expect_tx(bk, left_keys < BN ? C::kKBytes + C::kVBytes : C::kKBytes);
            for (int f = 0; f < DP / 64; ++f) tma_load_3d(dk + f * BN * 128, &map_k, bk, f * 64, key0, c.plane);
          }
          ++n_k;
          if (left_keys < BN) ragged_at = n_k - 1;
          if (q_due && !load_q()) { ok = false; break; }
          if (left_keys >= BN && n_v >= VS && !__all_sync(0xffffffffu, wait(&v_empty[vs], static_cast<uint32_t>((n_v / VS - 1) & 1)))) { ok = false; break; }
          if (lane == 0) {
            if (left_keys >= BN) mbar_expect_tx(bv, C::kVBytes);
            for (int f = 0; f < VP / 64; ++f) tma_load_3d(dv + f * BN * 128, &map_v, bv, f * 64, key0, c.plane);
          }
          ++n_v;
          if (left_keys < BN) {  // the sequence's last tile: rows behind its end hold anything, and 0 * NaN is not 0
            __syncwarp();
            if (!__all_sync(0xffffffffu, wait(ragged, static_cast<uint32_t>(n_ragged & 1)))) { ok = false; break; }
            for (int f = 0; f < DP / 64; ++f)
              for (int i = left_keys * 8 + lane; i < BN * 8; i += 32) *reinterpret_cast<uint4*>(dk + f * BN * 128 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
            for (int f = 0; f < VP / 64; ++f)
              for (int i = left_keys * 8 + lane; i < BN * 8; i += 32) *reinterpret_cast<uint4*>(dv + f * BN * 128 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&k_full[ks]);
              mbar_arrive(&v_full[vs]);
            }
            ++n_ragged;
            ragged_at = -1;
          }
        }
        a = after;
      }
      // all of it has landed when this warp is done (in a run that was given up, the tiles nobody waited for)
      if (n_q > 0) mbar_drain(q_full, static_cast<uint32_t>((n_q - 1) & 1));
      if (ragged_at >= 0) mbar_drain(ragged, static_cast<uint32_t>(n_ragged & 1));
      for (int i = max(0, n_k - KS); i < n_k; ++i)
        if (i != ragged_at) mbar_drain(&k_full[i % KS], static_cast<uint32_t>((i / KS) & 1));
      for (int i = max(0, n_v - VS); i < n_v; ++i)
        if (i != ragged_at) mbar_drain(&v_full[i % VS], static_cast<uint32_t>((i / VS) & 1));
      __syncwarp();
    } else if (warp <= kMmaWarp + 1) {
      // ===================== MMA issuers: warp 17 drives half 0, warp 18 half 1 =====================
      // In turns: the products of a tile and the scores of the next one go out as one batch, then it is the other half's turn, which meanwhile has made its waits.
      // (Without turns the halves' products interleave, both halves wait for scores at the same time and work at the same time: a tile took a third longer.
      // One warp for both halves: its own waits stand between the batches, 3 % longer.)
      // Everything that decides is the same in all lanes and known to be (uniform), and nothing in the loop is a lane's own: descriptors then stay in
      // uniform registers.  Otherwise a product is issued every 90 to 100 cycles; it takes 64 to 74.
      const int leader = lane == 0, x = warp - kMmaWarp;
      auto uniform = [](uint32_t v) { return __reduce_or_sync(0xffffffffu, v); };
      auto all_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
      constexpr uint32_t idesc_qk = idesc_bf16(BM, BN, 0), idesc_pv = idesc_bf16(BM, VP, 1);
      const uint32_t tm = uniform(tmem_base), base = uniform(smem_u32(smem)), tm_s = tm + x * BN, tm_o = tm + C::kColO + x * VP;
      const uint64_t q_desc = smem_desc_sw128(base + x * C::kQBytes, 16, 1024), k_desc0 = smem_desc_sw128(base + C::kOffK, 16, 1024),
                     v_desc0 = smem_desc_sw128(base + C::kOffV, BN * 128, 1024);
      uint32_t n = 0, n_piece = 0, n_p = 0, n_turn = 0;   // the run's tiles so far, its pieces, sets of weights, turns
      uint32_t code = 0;
      const int drop = static_cast<int>(uniform(static_cast<uint32_t>(drop_at)));
      bool ok = uniform(any) != 0;
      auto arrived = [&](uint32_t t) {   // tile t's keys are there, and what is to be done with them
        if (!all_wait(&k_full[t % KS], (t / KS) & 1)) return 0xffffffffu;
        tc_fence_after();
        return uniform(static_cast<uint32_t>(info[t % kInfo].y));
      };
      auto take_turn = [&]() {
        const bool mine = (x == 0 && n_turn == 0) || all_wait(&turn[x], (x == 0 ? n_turn - 1 : n_turn) & 1);
        ++n_turn;
        return mine;
      };
      auto pass_turn = [&]() {
        if (leader) mbar_arrive(&turn[x ^ 1]);
      };
      // scores with tile t of the run (which has arrived); S is written over the weights of the tile before: products of one thread run in order
      auto scores = [&](uint32_t t, uint32_t sees) {
        const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((t % KS * C::kKBytes) >> 4);
        if (!sees) pass_turn();
        if (sees) {
#pragma unroll
          for (int kk = 0; kk < DP / 16; ++kk) {
            if (kk == DP / 16 - 3) pass_turn();   // (the other half's warp takes some 200 cycles to begin: three products)
            umma_ss(tm_s, q_desc + static_cast<uint64_t>(((kk >> 2) * BM * 128 + (kk & 3) * 32) >> 4),
                    k_desc + static_cast<uint64_t>(((kk >> 2) * BN * 128 + (kk & 3) * 32) >> 4), idesc_qk, kk > 0 ? 1u : 0u, leader);
          }
        }
        tc_commit(&s_full[x], leader);   // (also where no product was issued: the softmax counts tiles by it)
      };
      while (ok) {   // a piece: its first scores, then tile by tile
        if (!(ok = all_wait(q_full, n_piece & 1))) break;
        if ((code = arrived(n)) == 0xffffffffu || !take_turn()) break;
        scores(n, code & 3);
        tc_commit(&k_empty[n % KS], leader);
        if (code & kLast) tc_commit(q_empty, leader);
        uint32_t into = 0;   // O holds products of this piece
        while (true) {
          const uint32_t sees = code & 3;
          uint32_t next = 0;
          if (static_cast<int>(n) == drop) *abort_word = 1;
          if (!(ok = static_cast<int>(n) != drop && all_wait(&v_full[n % VS], (n / VS) & 1))) break;
          if (n_piece > 0 && !into && (sees || (code & kLast)) && !(ok = all_wait(&o_free[x], (n_piece - 1) & 1))) break;
          const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((n % VS * C::kVBytes) >> 4);
          if (KS > 1 && !(code & kLast) && (next = arrived(n + 1)) == 0xffffffffu) { ok = false; break; }
          if (sees && !(ok = all_wait(&p_full[2 * x], n_p & 1))) break;
          if (!(ok = take_turn())) break;
          if (sees) {
#pragma unroll
            for (int step = 0; step < 2; ++step) {   // 32 keys of either 64
              if (step == 1 && !(ok = all_wait(&p_full[2 * x + 1], n_p & 1))) break;
              tc_fence_after();
#pragma unroll
              for (int part = 0; part < 2; ++part) {
                if (!(sees >> part & 1)) continue;
                const uint32_t pa = tm_s + part * HB + step * 32;   // hi of 32 keys in 16 columns, then lo
                const uint64_t vd = v_desc + static_cast<uint64_t>(((part * HB + step * 32) * 128) >> 4);
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) umma_ts(tm_o, pa + kk * 8, vd + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv, kk > 0 ? 1u : into, leader);
                into = 1;
#pragma unroll
                for (int kk = 0; kk < 2; ++kk) umma_ts(tm_o, pa + 16 + kk * 8, vd + static_cast<uint64_t>((kk * 2048) >> 4), idesc_pv, 1u, leader);
              }
            }
            if (!ok) break;
            ++n_p;
          }
          if (code & kLast) {
            pass_turn();
            tc_commit(&o_full[x], leader);
            tc_commit(&v_empty[n % VS], leader);
            ++n;
            break;
          }
          if (KS == 1 && (next = arrived(n + 1)) == 0xffffffffu) { ok = false; break; }   // (one stage: the keys cannot come before the turn)
          scores(n + 1, next & 3);
          tc_commit(&v_empty[n % VS], leader);
          ++n;
          tc_commit(&k_empty[n % KS], leader);
          if (next & kLast) tc_commit(q_empty, leader);
          code = next;
        }
        ++n_piece;
        if (code & kEnd) break;
      }
      __syncwarp();
      tc_commit(&drained[x], leader);   // and all products have ended
      mbar_drain(&drained[x], 0);
      __syncwarp();
    } else if (warp == kMmaWarp + 2 && any && ends[0].tile > 0) {
      // ===================== partial results: the flag behind the stores =====================
      // (The softmax warps store numbers, or NaN where the run was given up.  Where the wait for them runs out, what the scratch holds is not theirs: the flag then says so, and
      // the block that waits for it forms its rows again.)
      for (int x = 0; x < 2; ++x) {
        const bool out = drop_at < 0 && __all_sync(0xffffffffu, mbar_drain(&stored[x], 0));
        __threadfence();
        if (lane == 0) {
          st_flag(reinterpret_cast<unsigned long long*>(cut.slots + static_cast<long long>(*run_word) * C::kSlotBytes) + x, cut.nonce + (out ? 0 : kGivenUp));
          if (!out) *abort_word = 1;
        }
      }
      __syncwarp();
    }
  } else {
    // ===================== softmax: a thread one query row and 64 of a tile's 128 keys =====================
    // (Two warpgroups per half: with one, a thread's 128 scores took as long as the products, a warp per scheduler waiting for its own instructions.  The block has 96
    // registers per thread: what describes a piece stays in shared memory, and 32 scores are held at a time; spilled scores made a tile three times as long.)
    const int x = warp >> 3, part = warp >> 2 & 1, row = tid & 127;
    const uint32_t lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem_base + lanes + x * BN + part * HB, tmem_o = tmem_base + lanes + C::kColO + x * VP + part * (VP / 2);   // its half of the columns of O
    float m = -INFINITY, l = 0.f;   // the row's running maximum and sum
    int j = 0;                      // the piece's tiles so far
    int n = 0, n_piece = 0;         // tiles and pieces of the run so far
    // Where a thread's wait ran out, the half's 256 threads learn of it at their next barrier and leave together (what the TMA warp would have described is
    // not there to go by, and the barriers count on all of them).  (A word per barrier and turn: it is written before the barrier, read behind it, and not
    // used again before the barrier after that.)
    bool ok = true;
    auto together = [&](int which, int turns) {
      volatile int* word = left + (which * 2 + (turns & 1)) * 2 + x;
      if (!ok) *word = 1;
      named_barrier(1 + x, 256);
      return ok = *word == 0;
    };
    for (bool last = !any; !last; ++n_piece) {
      ok = wait(&s_full[x], static_cast<uint32_t>(n & 1));   // the piece is described when its first scores are there
      const Piece& c = pieces[n_piece % kPieces];
      const int h = ok ? c.h[x] : 0, first = c.pos0 + c.q0, n_tiles = ok ? c.it1 - c.it0 : 1, rows = c.rows, pos = first + row, keep = c.keep;
      // this row sees the keys [lo_key, pos] and [0, keep)
      const int lo_key = p.window > 0 ? max(0, pos - p.window + 1) : p.chunk > 0 ? pos / p.chunk * p.chunk : 0, end_key = row < rows ? pos + 1 : 0;
      const float scale = p.scale * (p.head_scale ? p.head_scale[h] : 1.f), scale2 = scale * kLog2e;
      const float cap_in = CAP ? scale / p.softcap * 2.f * kLog2e : 0.f, cap_out = CAP ? p.softcap * kLog2e : 0.f;
      const float mult = (BIAS || CAP || !(scale2 > 0.f)) ? 1.f : scale2;   // what is left to multiply the scores by when the exponentials are formed
      // the biases of a tile's 255 distances, in the base-2 domain with their sign turned, into the buffer of tile number k of this piece
      auto biases = [&](int k) {
        const int y = part * BM + row, d = first - c.w.tile(c.it0 + k) * BN + y - (BN - 1);
        float v = 0.f;
        if (ok && d >= 0)
          v = p.bias_table ? -kLog2e * p.bias_table[static_cast<long long>(h) * p.bias_len + min(d, p.bias_len - 1)] : p.bias_r1[h] * __log2f(fmaf(p.bias_r2[h], static_cast<float>(d), 1.f));
        sTab[(x * 2 + (k & 1)) * kTab + y] = v;
      };
      m = -INFINITY;
      l = 0.f;
      j = 0;
      if (p.sink && c.it0 == 0) {  // one more term of the denominator, exp(sink), without a value
        m = p.sink_logit ? p.sink_logit[h] * kLog2e : 0.f;
        l = part == 0 ? 1.f : 0.f;
      }
      if (BIAS) {
        biases(0);
        if (!together(0, n_piece)) break;
      }
      for (int it = 0; it < n_tiles; ++it, ++n) {
        if (BIAS && it + 1 < n_tiles) biases(it + 1);   // (for the next tile: the barrier below stands between)
        if (it > 0) ok = wait(&s_full[x], static_cast<uint32_t>(n & 1));
        const int2 what = info[n % kInfo];
        const int sees = ok ? what.y & 3 : 0;
        __syncwarp();
        tc_fence_after();
        // Its scores in two steps of 32, the second one first: that one goes back to TMEM where it was changed and is read again when its turn comes
        const bool mine = sees >> part & 1;
        float s[32], mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (__any_sync(0xffffffffu, mine)) {
          const int kp0 = what.x + part * HB;
          const float* tb = BIAS ? sTab + (x * 2 + (it & 1)) * kTab + row + (BN - 1) - part * HB : nullptr;
          const bool need_mask = __any_sync(0xffffffffu, kp0 + HB > end_key || (lo_key > kp0 && kp0 + HB > keep));
#pragma unroll
          for (int step = 1; step >= 0; --step) {
            tmem_ld32(tmem_s + step * 32, reinterpret_cast<uint32_t(&)[32]>(s));
            tmem_ld_wait();
            if (CAP) {  // cap tanh(s scale / cap) as 1 - 2 / (1 + e^(2x)), in the base-2 domain
              // Three uses of the exponential unit per score made a window of 1024 under a cap 96 us; four scores that share one reciprocal: 84 us.  e^(2x) is
              // held below 2^30 (tanh is 1 there), so the product of four stays in range.  (A hidden score that is no number spoils its three neighbours: such
              // a row's sum is no number either, and the row is formed again at the end.  A polynomial for small scores, multiply-adds only: no faster.)
#pragma unroll
              for (int k = 0; k < 32; k += 4) {
                float d[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) d[i] = 1.f + ex2(min_nan(s[k + i] * cap_in, 30.f));
                const float d01 = d[0] * d[1], d23 = d[2] * d[3], inv = __fdividef(1.f, d01 * d23), i01 = inv * d23, i23 = inv * d01;
                const float q[4] = {i01 * d[1], i01 * d[0], i23 * d[3], i23 * d[2]};
#pragma unroll
                for (int i = 0; i < 4; ++i) s[k + i] = fmaf(q[i], -2.f * cap_out, cap_out - (BIAS ? tb[-(step * 32 + k + i)] : 0.f));
              }
            } else if (BIAS) {
#pragma unroll
              for (int k = 0; k < 32; ++k) s[k] = fmaf(s[k], scale2, -tb[-(step * 32 + k)]);
            } else if (mult == 1.f) {
#pragma unroll
              for (int k = 0; k < 32; k += 2) mul_x2(s[k], s[k + 1], scale2);
            }
            if (need_mask) {
              const int k0 = kp0 + step * 32, lo_c = min(max(lo_key - k0, 0), 32), end_c = min(max(end_key - k0, 0), 32), keep_c = min(max(keep - k0, 0), 32);
              auto below = [](int k) { return k >= 32 ? ~0u : (1u << k) - 1u; };
              const uint32_t vis = below(end_c) & (~below(lo_c) | below(keep_c));
#pragma unroll
              for (int k = 0; k < 32; ++k)
                if (!(vis & (1u << k))) s[k] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int k = 0; k < 32; k += 8) mx[i] = max3(mx[i], s[k + i], s[k + 4 + i]);
            if (step == 1 && (CAP || BIAS || mult == 1.f || need_mask)) tmem_st32(tmem_s + 32, reinterpret_cast<uint32_t(&)[32]>(s));
          }
        }
        const float top = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
        // (two buffers: the barrier of the next tile stands before the next use of this one)
        sMax[max_array(n, x, part) * BM + row] = top;
        if (!together(1, n)) break;
        if (!sees) continue;
        const float m_new = fmaxf(m, fmaxf(top, sMax[max_array(n, x, part ^ 1) * BM + row]) * mult);
        const bool grow = (m_new - m) > kRescale;  // the first finite maximum: +inf; both -inf: NaN, false
        const float alpha = grow ? ex2(m - m_new) : 1.f;
        if (grow) { m = m_new; l *= alpha; }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {   // (the products so far ended before this tile's scores)
#pragma unroll 1
          for (int f = 0; f < VP / 32; ++f) {
            uint32_t o[16];
            tmem_ld16(tmem_o + f * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
            tmem_st16(tmem_o + f * 16, o);
          }
        }
        const float neg = m == -INFINITY ? 0.f : -m;   // a row that has seen no key yet: its masked scores give 2^-inf = 0
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int step = 0; step < 2; ++step) {
          if (mine) {
            if (step == 1) {
              tmem_ld32(tmem_s + 32, reinterpret_cast<uint32_t(&)[32]>(s));
              tmem_ld_wait();
            }
            uint32_t hi_p[16], lo_p[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              float &p0 = s[2 * k], &p1 = s[2 * k + 1];
              if (BIAS || CAP) add_x2(p0, p1, neg, neg);
              else fma_x2(p0, p1, mult, neg);
              p0 = ex2(p0);
              p1 = ex2(p1);
              add_x2(sum[(k & 1) * 2], sum[(k & 1) * 2 + 1], p0, p1);
              hi_p[k] = pack_bf16(p0, p1);
              add_x2(p0, p1, __uint_as_float((hi_p[k] << 16) ^ 0x80000000u), __uint_as_float((hi_p[k] & 0xffff0000u) ^ 0x80000000u));
              lo_p[k] = pack_bf16(p0, p1);
            }
            tmem_st16(tmem_s + step * 32, hi_p);
            tmem_st16(tmem_s + step * 32 + 16, lo_p);
          }
          tmem_st_wait();
          tc_fence_before();
          mbar_arrive(&p_full[2 * x + step]);
        }
        l += (sum[0] + sum[2]) + (sum[1] + sum[3]);
        ++j;
      }
      if (!ok) break;
      // the row's sum over both parts of the tiles
      sMax[sum_array(x, part) * BM + row] = l;
      ok = wait(&o_full[x], static_cast<uint32_t>(n_piece & 1));
      __syncwarp();
      tc_fence_after();
      if (!together(2, n_piece)) break;
      l += sMax[sum_array(x, part ^ 1) * BM + row];
      last = info[(n - 1) % kInfo].y & kEnd;
      const int q0 = c.q0;
      const bool live = row < rows;
      constexpr int VH = VP / 2;   // this thread's half of the columns of O: [part VH, part VH + VH)
      // O leaves TMEM in pieces of 16 rows x 32 columns with the columns across four neighbouring lanes (a row per lane means 32 lines per store)
      const int quad = lane >> 2, sub = lane & 3;
      // of a scratch slot: pieces [half][part][32 columns][16 rows of 32], in each 4 float4 of every lane of the four warps
      auto piece_at = [&](int f, int hh) { return ((((x * 2 + part) * (VH / 32) + f) * 2 + hh) * 4 + (warp & 3)) * 128 + lane; };
      if (c.it0 > 0) {
        // the end or the middle of an item: (m, l, O) to the block that has its first tiles
        unsigned char* mine = cut.slots + static_cast<long long>(*run_word) * C::kSlotBytes;
        float4* o_out = reinterpret_cast<float4*>(mine + 64 + 2 * BM * 8);
#pragma unroll 1
        for (int f = 0; f < VH / 32; ++f)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            float r[16];
            tmem_ld_rows16(tmem_o + (hh * 16 << 16) + f * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 4; ++k)
              __stcg(o_out + piece_at(f, hh) + k * 32, j > 0 ? make_float4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]) : make_float4(0.f, 0.f, 0.f, 0.f));
          }
        tc_fence_before();
        mbar_arrive(&o_free[x]);
        if (part == 0) __stcg(reinterpret_cast<float2*>(mine + 64) + x * BM + row, make_float2(m, l));
        if (row == 0 && part == 0) __stcg(reinterpret_cast<int*>(mine + 16) + x, c.it1);
        mbar_arrive(&stored[x]);   // (the publishing warp raises the flag: nobody here waits for the stores)
      } else {
        // the result: O / l, times the constant and the head's gate; where the item was cut, with the later runs' sums
        const unsigned char* slot = cut.slots + static_cast<long long>(*run_word + 1) * C::kSlotBytes;
        int others = 0;
        float mt = m, lt = l;
        for (int upto = c.it1; upto < c.w.n; ++others) {
          const unsigned char* s = slot + static_cast<long long>(others) * C::kSlotBytes;
          bool got = true;
          if (lane == 0) {
            const unsigned long long* flag = reinterpret_cast<const unsigned long long*>(s) + x;
            unsigned long long seen;
            int tries = 0;
            while ((seen = ld_acquire(flag)) != cut.nonce && seen != cut.nonce + kGivenUp && !*abort_word && ++tries < kWaitTries) __nanosleep(20);
            got = seen == cut.nonce;
            if (!got) *abort_word = 1;
          }
          __syncwarp();
          if (!__shfl_sync(0xffffffffu, got, 0)) break;
          upto = __ldcg(reinterpret_cast<const int*>(s + 16) + x);
          const float2 q = __ldcg(reinterpret_cast<const float2*>(s + 64) + x * BM + row);
          const float mn = fmaxf(mt, q.x);
          lt = lt * (mt == -INFINITY ? 0.f : ex2(mt - mn)) + q.y * (q.x == -INFINITY ? 0.f : ex2(q.x - mn));
          mt = mn;
        }
        if (others > 0) {   // O = O 2^(m - mt) + the others', in its place
          const float own = j > 0 && m != -INFINITY ? ex2(m - mt) : 0.f;
#pragma unroll 1
          for (int i = 0; i < others; ++i) {
            const unsigned char* s = slot + static_cast<long long>(i) * C::kSlotBytes;
            const float4* y = reinterpret_cast<const float4*>(s + 64 + 2 * BM * 8) + piece_at(0, 0);
            const float mq = __ldcg(reinterpret_cast<const float2*>(s + 64) + x * BM + row).x, fq = mq == -INFINITY ? 0.f : ex2(mq - mt);
#pragma unroll 1
            for (int k8 = 0; k8 < VH / 16; ++k8) {   // [32 columns][16 rows]
              const int hh = k8 & 1;
              float4 o[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) o[k] = __ldcg(y + k8 * 512 + k * 32);
              float r[16];
              tmem_ld_rows16(tmem_o + (hh * 16 << 16) + (k8 >> 1) * 32, r);
              const float w = i == 0 ? own : 1.f;
              const float a0 = __shfl_sync(0xffffffffu, w, quad + 16 * hh), a1 = __shfl_sync(0xffffffffu, w, quad + 16 * hh + 8);
              const float q0f = __shfl_sync(0xffffffffu, fq, quad + 16 * hh), q1f = __shfl_sync(0xffffffffu, fq, quad + 16 * hh + 8);
              tmem_ld_wait();
              const bool has = j > 0 || i > 0;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                r[4 * k] = fmaf(o[k].x, q0f, has ? r[4 * k] * a0 : 0.f);
                r[4 * k + 1] = fmaf(o[k].y, q0f, has ? r[4 * k + 1] * a0 : 0.f);
                r[4 * k + 2] = fmaf(o[k].z, q1f, has ? r[4 * k + 2] * a1 : 0.f);
                r[4 * k + 3] = fmaf(o[k].w, q1f, has ? r[4 * k + 3] * a1 : 0.f);
              }
              tmem_st_rows16(tmem_o + (hh * 16 << 16) + (k8 >> 1) * 32, r);
            }
            tmem_st_wait();   // (the next one's sums are added to what was stored here)
          }
        }
        const float inv = live ? (lt > 0.f ? 1.f / lt : 0.f) * out_factor<__nv_bfloat16>(p, c.off + q0 + row, h) : 0.f;
        const bool has = j > 0 || others > 0;
        __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);   // stays 0 over finite numbers
        const int r0 = (warp & 3) * 32 + quad;   // this lane's rows: r0 + 8 i, whose factors are in the lanes quad + 8 i
#pragma unroll 1
        for (int hh = 0; hh < 2; ++hh) {   // rows r0 + 16 hh and 8 further
          const float f0 = __shfl_sync(0xffffffffu, inv, quad + 16 * hh), f1 = __shfl_sync(0xffffffffu, inv, quad + 16 * hh + 8);
          __nv_bfloat16* out = out_row<__nv_bfloat16>(p, c.off + q0 + r0 + 16 * hh, h) + part * VH + 8 * sub;
          const long long row8 = 8 * (p.out_stride > 0 ? p.out_stride : static_cast<long long>(p.n_heads) * p.vdim);
#pragma unroll 1
          for (int f = 0; f < VH / 32; ++f) {
            float r[16];
            tmem_ld_rows16(tmem_o + (hh * 16 << 16) + f * 32, r);
            tmem_ld_wait();
            if (has) {
#pragma unroll
              for (int k = 0; k < 16; k += 2) mul_x2(r[k], r[k + 1], k & 2 ? f1 : f0);
            } else {
#pragma unroll
              for (int k = 0; k < 16; ++k) r[k] = 0.f;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {   // lane `sub` of four gets the eight columns 8 sub of its row
              uint32_t w[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) w[k] = pack_bf16(r[4 * k + 2 * i], r[4 * k + 2 * i + 1]);
              transpose4(w, sub);
              if (r0 + 16 * hh + 8 * i < rows && part * VH + f * 32 + 8 * sub < p.vdim) {
#pragma unroll
                for (int k = 0; k < 4; ++k) zero = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&w[k]), __floats2bfloat162_rn(0.f, 0.f), zero);
                *reinterpret_cast<uint4*>(out + i * row8 + f * 32) = make_uint4(w[0], w[1], w[2], w[3]);
              }
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&o_free[x]);
        if (__low2float(zero) + __high2float(zero) != 0.f) *redo_word = 1;
      }
    }
    if (!ok && n_piece == 0 && ends[0].tile > 0) {   // a run that was given up in a piece that another block waits for: NaN
      unsigned char* mine = cut.slots + static_cast<long long>(*run_word) * C::kSlotBytes;
      const float nan = __int_as_float(0x7fffffff);
      if (part == 0) __stcg(reinterpret_cast<float2*>(mine + 64) + x * BM + row, make_float2(nan, nan));
      if (row == 0 && part == 0) __stcg(reinterpret_cast<int*>(mine + 16) + x, piece_of(ends[0]).it1);
      mbar_arrive(&stored[x]);
    }
  }
  tc_fence_before();
  __syncthreads();   // TMEM has been read
  if (*abort_word && tid == 0) atomicAdd(&attn_tc5w_timeouts, 1);   // a wait ran out: the block is counted
  if (*abort_word || *redo_word) {
    // rows whose result is not finite, or any row of a run that was given up: from the keys they see alone
    for (Place a = ends[0]; more(a);) {
      const Piece c = piece_of(a);
      for (int i = warp; i < 2 * BM && c.it0 == 0; i += kThreads / 32) {
        const int h = i >> 7 ? c.h[1] : c.h[0], row = i & (BM - 1), t = c.off + c.q0 + row;
        if (row >= c.rows) continue;
        const __nv_bfloat16* out = out_row<__nv_bfloat16>(p, t, h);
        bool bad = *abort_word != 0;
        for (int k = lane; k < p.vdim; k += 32) bad = bad || !(fabsf(ldf(out + k)) < INFINITY);
        if (__any_sync(0xffffffffu, bad)) attn_row_again_call<__nv_bfloat16>(p, c.b, h, t, c.pos0 + c.q0 + row, 0, p.vdim);
      }
      advance(a, c);
    }
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_free<512>(tmem_base);
  }
}

// The flags of a launch hold a number that no other launch of this process uses (and that memory holds by chance once in 2^64)
unsigned long long next_nonce() {
  static std::atomic<unsigned long long> n{static_cast<unsigned long long>(std::chrono::high_resolution_clock::now().time_since_epoch().count()) * 0x9e3779b97f4a7c15ull | 1ull};
  return n.fetch_add(2, std::memory_order_relaxed);
}

constexpr int kSMs = 148;   // runs of a launch
template <int DP, int VP>
constexpr long long kScratchFloats = static_cast<long long>(kSMs) * Cfg<DP, VP>::kSlotBytes / 4;

template <int DP, int VP, bool BIAS, bool CAP>
int launch(const pcs_attn_params& p, float* scratch, long long floats, cudaStream_t st, bool* handled) {
  using C = Cfg<DP, VP>;
  if (floats < kScratchFloats<DP, VP> || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0) return PCS_OK;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusActive;
  PCS_CHECK_CUDA(cudaStreamIsCapturing(st, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return PCS_OK;   // (a captured launch would come again with the flags that it left)
  auto kernel = attn_tc5w_kernel<DP, VP, BIAS, CAP>;
  struct Info {};
  static PerDevice<Info> per_device;
  const Info* info;
  if (int rc = per_device.get(&info, [&](Info&) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem); })) return rc;
  const unsigned long long D = p.dim, V = p.vdim, cap = p.cap, H = p.n_heads;
  const unsigned long long planes = pool_planes(p);
  CUtensorMap mq, mk, mv;
  if (int rc = tensor_map_bf16(&mq, p.q, {D, H, static_cast<unsigned long long>(p.n_tokens)}, {D * 2, H * D * 2}, {64, 1, BM})) return rc;
  if (int rc = tensor_map_bf16(&mk, p.k_pool, {D, cap, planes}, {D * 2, cap * D * 2}, {64, BN, 1})) return rc;
  if (int rc = tensor_map_bf16(&mv, p.v_pool, {V, cap, planes}, {V * 2, cap * V * 2}, {64, BN, 1})) return rc;
  const Cut cut = {(p.impl & 3) == 3, reinterpret_cast<unsigned char*>(scratch), next_nonce()};
  kernel<<<kSMs, kThreads, C::kSmem, st>>>(mq, mk, mv, p, cut);
  PCS_CHECK_CUDA(cudaGetLastError());
  count_launch();
  *handled = true;
  return PCS_OK;
}

template <int DP>
int launch_opt(const pcs_attn_params& p, float* scratch, long long floats, cudaStream_t st, bool* handled) {
  const bool bias = p.bias_r1 || p.bias_table, cap = p.softcap > 0.f;
  if (cap) return bias ? launch<DP, 128, true, true>(p, scratch, floats, st, handled) : launch<DP, 128, false, true>(p, scratch, floats, st, handled);
  return bias ? launch<DP, 128, true, false>(p, scratch, floats, st, handled) : launch<DP, 128, false, false>(p, scratch, floats, st, handled);
}

}  // namespace

bool short_entries(const pcs_attn_params& p);
double attn_tc5_expected(const pcs_attn_params& p, const Entries& entries);   // in the other forms

namespace {

// Forms this kernel has: an even number of heads per K/V group, heads of 65 to 192 / 65 to 128 elements in 16-byte pieces, at most 256 entries
bool serves(const pcs_attn_params& p) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return !dense_rows_off_boxes(p) && p.dtype == PCS_BF16 && p.max_len >= 16 && (p.v_row_stride == 0 || p.v_row_stride == p.vdim) && p.dim % 8 == 0 && p.vdim % 8 == 0 && p.dim > 64 && p.dim <= 192 &&
         p.vdim > 64 && p.vdim <= 128 && p.n_heads / p.n_kv_heads % 2 == 0 && p.n_seqs <= kMaxStreamSeqs && p.seq_pos0 && p.seq_len && p.seq_off && al16(p.q) &&
         al16(p.k_pool) && al16(p.v_pool) && al16(p.out) && p.out_stride % 8 == 0;
}

// At least ten key tiles of 128 per SM where all entries are like the longest one, and less time than the other forms, as both are expected from the entries' walks.  The constants
// here are fitted to the same launches (90 % within 8 %): 13.6 us and, per SM, 4.9 for an item and 2.8 to 4.4 for a key tile; 3.1 for each run that shares an item.  One per cent (15 where the
// other one is the mma.sync kernel, whose time is known less well) is left between the two.  Of 1100 shapes drawn from one to four entries of 200 to 7000 tokens, this one then takes 187, two of them
// slower than the other form by 6 and 10 %, the others 0.97 to 2.1 times as fast; all 1100 together are 1.031 times as fast as without it, 1.039 if each took the better form.
// Examples, the other form / this one in us:
//   785 tokens of 16 heads                       20.6 / 28.8      four prompts under a window, cap                  86 / 67
//   2048 tokens                                  47.1 / 47.1      3102 tokens behind 205, 12 heads, bias           100 / 77
//   12 entries of 200 behind 1500, 12 heads      49.0 / 60.8      24 entries of 16 behind 4000, 8 heads            166 / 88
//   200 entries of 16, nothing stored            61 / 79          64 entries of 128 behind 250, 32 heads           174 / 98
//   5255 tokens of 12 heads, bias                135 / 147        692, 416, 1671, 1876, one behind 2479; 8 of 192  116 / 77
// Heads that share no K/V rows, neighbouring tiles instead: 4020 tokens in three entries of 16 heads 62 / 76; heads of 64: 6715 tokens 225 / 232.
bool pays(const pcs_attn_params& p, const Entries& entries) {
  const int keys = p.max_keys > 0 && p.max_keys < p.cap ? p.max_keys : p.cap, n = (p.max_len + BM - 1) / BM;
  const double items = fmin(static_cast<double>(p.n_seqs) * n, p.n_tokens / static_cast<double>(BM) + p.n_seqs) * (p.n_heads / 2);
  double sum = 0.0;   // key tiles of a unit of the longest entry
  for (int u = 0; u < n; ++u) {
    double k = fmax(fmin(keys, keys - p.max_len + (u + 1.0) * BM), 1.0);
    if (p.window > 0) k = fmin(k, p.window + BM + fmax(p.keep_first, 0) + BN);
    if (p.chunk > 0) k = fmin(k, p.chunk + BM);
    sum += ceil(k / BN);
  }
  if (sum / n * items < 10.0 * kSMs) return false;
  const bool cap = p.softcap > 0.f, bias = p.bias_r1 || p.bias_table, wide = p.dim > 128;
  double its = 0.0, tiles = 0.0, longest = 0.0;
  for (int b = 0; b < entries.n; ++b) {
    const int pos0 = entries.pos_of(b), len = entries.len_of(b);
    for (int t = 0; t < len; t += BM) {
      const int k = Walk<BN>(p, pos0, len, t, t + BM < len ? t + BM : len).n;
      its += p.n_heads / 2;
      tiles += static_cast<double>(k) * (p.n_heads / 2);
      if (k > longest) longest = k;
    }
  }
  its /= kSMs;
  tiles /= kSMs;
  const double here = 13.6 + its * (4.9 + (wide ? 0.8 : 0.0) - (cap ? 0.3 : 0.0)) + tiles * (2.84 + (bias ? 0.42 : 0.0) + (cap ? 1.52 : 0.0) + (wide ? 0.16 : 0.0)) +
                      3.1 * longest / fmax(tiles + its, 3.0);
  return here < (short_entries(p) ? 0.85 : 0.99) * attn_tc5_expected(p, entries);
}

}  // namespace

// (Whether it pays is asked once, by whom allocates: a launch that is given the scratch takes this form.)
int launch_attn_tc5w(const pcs_attn_params& p, float* scratch, long long floats, cudaStream_t st, bool* handled) {
  *handled = false;
  if (!scratch || !serves(p)) return PCS_OK;
  return p.dim <= 128 ? launch_opt<128>(p, scratch, floats, st, handled) : launch_opt<192>(p, scratch, floats, st, handled);
}

int attn_tc5w_timeouts_so_far() {
  int n = -1;
  return cudaMemcpyFromSymbol(&n, attn_tc5w_timeouts, sizeof(n)) == cudaSuccess ? n : -1;
}

}  // namespace pcs

PCS_API int64_t pcs_attn_prompt_scratch_wanted(const pcs_attn_params* p, const int32_t* pos0, const int32_t* len) {
  if (!p || p->n_tokens <= 0 || p->n_seqs <= 0 || p->talk || !pcs::automatic(*p) || p->n_heads <= 0 || p->n_kv_heads <= 0 || p->dim <= 0 || p->vdim <= 0 || p->cap <= 0)
    return 0;
  if (!pcs::serves(*p) || (p->impl < 4 && !pcs::pays(*p, pcs::Entries(*p, pos0, len)))) return 0;
  return p->dim <= 128 ? pcs::kScratchFloats<128, 128> : pcs::kScratchFloats<192, 128>;
}
