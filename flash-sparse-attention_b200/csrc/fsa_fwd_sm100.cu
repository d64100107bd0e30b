// Forward attention for sm_100a: tcgen05 MMAs with TMEM accumulators, TMA-fed K/V rings,
// warp-specialised roles.
//
// One CTA owns TWO consecutive 128-row query tiles of one head (so every K/V tile it pulls from
// L2 is used by 256 query rows) and walks the key tiles both tiles visit, in descending order.
// Replaces, per CTA, two programs of the reference's `_fwd_{dense,sparse}_kernel`
// (flash_sparse_attn/ops/triton/flash_sparse_fwd.py:91-502, flash_dense_fwd.py:89-498) at
// TILE_M = TILE_N = 128: same tile schedule, same masks, same online-softmax recurrences and the
// same per-tile skip rule (activations.py:103-166), evaluated independently for each 128-row tile.
//
// Roles (384 threads = 3 warpgroups, registers rebalanced with setmaxnreg; gated: 640 threads, see FwdRoles):
//   warps 0-3  : softmax group 0 (query tile 0), one thread per query row / TMEM lane
//   warps 4-7  : softmax group 1 (query tile 1)
//   warp  8    : producer - TMA loads of Q, K ring, V ring; allocates / frees TMEM
//   warp  9    : MMA issuer - S = Q K^T and O_tile = P V on the tensor cores
//   warps 10-11: idle
//
// TMEM columns: S0 | S1 | O0 | O1, 128 each (O uses HD columns). P (16-bit) is written back over the
// first 64 columns of its own S block and consumed from TMEM as the A operand of P V.
// The output accumulates in TMEM across key tiles. A softmax thread keeps a reference maximum per
// row that is only moved (and O rescaled in TMEM) when the true running maximum has drifted by
// more than 2^8 from it: sums and outputs stay exact up to rounding because every term carries the
// same reference, and the skip rule reads the same in terms of the reference pair (m, l).
#include <cooperative_groups.h>

#include <type_traits>

#include "fsa_ptx.cuh"
#include "fsa_params.h"
#include "fsa_schedule.h"


namespace fsa {

namespace {

constexpr int TM = 128;  // query rows per softmax group
constexpr int TN = 128;  // keys per tile
// Warps by kind. One softmax thread per query row, four warps a group; the gated kind has two threads a row, 64 key columns
// each, eight warps a group (up to head size 128): the gate's chains (an exponential, then five dependent multiply-adds) take a warp 15
// cycles a column where four warps of a scheduler together take 9. B1 S8192, 32 / 8 heads of 128, with the gate worked out ahead of the
// scores: full 1951 -> 1713 us, causal 984 -> 942, windows of 512 to 4096 (B4) 1741 -> 1708; head size 64 causal 968 -> 921.
template <int HD, int KIND>
struct FwdRoles {
  static constexpr int HALVES = KIND == KIND_GATED && HD <= 128 ? 2 : 1;  // threads per query row
  static constexpr int GW = 4 * HALVES;                      // softmax warps of a group
  static constexpr int W_PROD = 2 * GW, W_MMA = W_PROD + 1, W_STAGE = W_PROD + 2;
  static constexpr int NTHREADS = (W_PROD + 4) * 32;
};
// Two K and two V stages. V(t) and K(t + 1) are consumed by the same loop step of the MMA issuer, so they
// arrive on one barrier and one "consumed" barrier per step releases both: every barrier the issuer touches
// costs it 130-250 cycles even when it is already complete. (A third V stage, loaded a whole step earlier, did
// not shorten the issuer's wait: it is not load latency.)
// Head sizes above 128 (the 192- and 256-wide instantiations): a tile is 48 / 64 KB, so a CTA holds ONE query tile
// (the second softmax group idles; its TMEM columns belong to the wider output accumulator of the first) and one
// stage of V - the load of V(t) then starts when P V(t - 1) has completed and runs under the softmax of tile t. K
// keeps two stages where they fit (192 wide).
template <int HD>
struct FwdShape {
  static constexpr int QT = HD > 128 ? 1 : 2;       // query tiles (softmax groups at work) per CTA
  static constexpr int KSTAGES = HD > 192 ? 1 : 2;
  static constexpr int VSTAGES = HD > 128 ? 1 : 2;
};

template <int HD, int ES, int KIND, bool CL>
struct FwdSmem {
  static constexpr int kTileBytes = TM * HD * ES;  // one Q / K / V tile of ES-byte elements
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + FwdShape<HD>::QT * kTileBytes;
  static constexpr int kV = kK + FwdShape<HD>::KSTAGES * kTileBytes;
  static constexpr int kBar = kV + FwdShape<HD>::VSTAGES * kTileBytes;
  // (maximum, sum) of rows: of a row's halves, [group][half][row] (gated), or of the rows whose cluster merges, [group][row]
  static constexpr int kXch = kBar + 2048;
  static constexpr int kTotal = kXch + (FwdRoles<HD, KIND>::HALVES == 2 || CL ? 4096 : 0) + 1024;  // barriers/flags/delta ring + alignment slack
};

// Output / gate element type that goes with an input element type.
template <typename T>
struct OutType {
  using type = T;
};
template <>
struct OutType<__nv_fp8_e4m3> {
  using type = __nv_bfloat16;
};
template <>
struct OutType<__nv_fp8_e5m2> {
  using type = __nv_bfloat16;
};

constexpr int MAX_RANKED = FSA_FWD_MAX_RANKED;  // (query tile pair, sequence) items that a CTA ranks at most

struct FwdBars {
  uint64_t q_full;
  uint64_t k0_full;     // first K tile
  uint64_t kv_full[2];  // step t (slot t & 1): V(t) and K(t + 1) have landed (two producer arrivals)
  uint64_t kv_empty[2];  // signal c (slot c & 1): K(c) and V(c - 1) have been consumed; c = 0 comes from the prologue
  // p_full: P of a kept tile is in TMEM (FP8: its first half); p_rest: FP8, the second half; wg_sync: every warp of the group has
  // read the tile's scores and voted (the kinds that skip tiles)
  uint64_t s_full[2], p_full[2], p_rest[2], o_final[2], wg_sync[2];
  uint64_t d_full[2], d_empty[2];  // gated: delta ring (stager warp -> softmax warps)
  uint32_t tmem_base;
  int abort_flag;
  uint64_t pair_sync[2][4];  // two threads a row: the two warps of a lane quadrant have written their halves' (maximum, sum)
  alignas(16) int vote_any[2][2][8]; // [group][parity][warp]: bit0 = some row wants the tile, bit1 = some row votes skip
  // What the producer worked out about the tiles, for the MMA issuer: low word the tile index (-1: none), then bit q: group q
  // takes part in it, bit 2 + q: it is group q's last. Slot 2: the first tile, published with k0_full. Slot t & 1: the
  // tile after step t (and whether the one of step t is a group's last), published with kv_full.
  unsigned long long step_info[3];
  // gated: delta of the key tile as fp32 (read as float4), then as integers the tile index (-1: the end) and the mask mode
  // of the two groups (-1: the group does not compute the tile)
  alignas(16) float dl[2][TN + 4];
};

static_assert(offsetof(FwdBars, dl) % 16 == 0 && sizeof(FwdBars) <= 2048, "FwdBars layout");
static_assert(sizeof(FwdBars::dl) >= (MAX_RANKED + 1) * sizeof(int), "room for the items' ranks");

struct SeqInfo {
  int b, split, head, hkv;  // head = query head, or kv head when packing GQA rows
  int off_q, off_k, sq, sk;
  FsaWindow w;
};

// Row-local view of the masks in flash_sparse_attn/ops/triton/mask.py:60-102: for one query row
// the visible key columns form up to three intervals (near band, distant band, sink prefix).
struct RowMask {
  int diag;            // last causally visible column: q_idx + (sk - sq)
  int near_lo;         // near band    = (near_lo, diag]
  int far_lo, far_hi;  // distant band = (far_lo, far_hi]
  int sink_hi;         // sink         = [0, sink_hi) intersected with [0, diag]
  int sk;
  bool row_ok;
};

// Visible columns of one row inside key tile [k0, k0 + TN), as three half-open intervals of the
// tile-local index, already clipped to the key length. Unused intervals are empty (len 0).
struct TileMask {
  int lo[3];
  unsigned len[3];
};

__device__ __forceinline__ TileMask make_tile_mask(const RowMask& rm, int mode, int k0) {
  TileMask tm;
  const int seq_hi = rm.row_ok ? min(rm.sk - k0, TN) : 0;
  auto clip = [&](int idx, int a, int b) {  // [a, b) in key coordinates -> tile-local, clipped
    a = max(a - k0, 0);
    b = min(b - k0, seq_hi);
    tm.lo[idx] = a;
    tm.len[idx] = b > a ? unsigned(b - a) : 0u;
  };
  if (mode == FSA_MASK_SEQLEN) {
    clip(0, 0, rm.sk);
    clip(1, 0, 0);
    clip(2, 0, 0);
  } else if (mode == FSA_MASK_CAUSAL) {
    clip(0, 0, rm.diag + 1);
    clip(1, 0, 0);
    clip(2, 0, 0);
  } else {
    clip(0, rm.near_lo + 1, rm.diag + 1);
    clip(1, rm.far_lo + 1, rm.far_hi + 1);
    if (mode == FSA_MASK_LOCAL_SINK)
      clip(2, 0, min(rm.sink_hi, rm.diag + 1));
    else
      clip(2, 0, 0);
  }
  return tm;
}
// Visible columns [base, base + 32) as bits, and their application: the row's other entries become -inf. One test of a bit
// per entry whatever the mask is made of; a masked tile's code is met cold (two of nine tiles under a 1024-token window),
// so its length counts most.
__device__ __forceinline__ uint32_t tile_bits(const TileMask& tm, int base) {
  return interval_bits(tm.lo[0], tm.len[0], base) | interval_bits(tm.lo[1], tm.len[1], base) |
         interval_bits(tm.lo[2], tm.len[2], base);
}
__device__ __forceinline__ void mask_cols32(uint32_t* r, uint32_t bits) {
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (!(bits & (1u << i))) r[i] = 0xff800000u;
}

// BSCALE: FP8 inputs with one scale per 128-position block (a separate instantiation: as a run-time switch it cost
// the per-tensor FP8 forward 10 %).
// CL: the CTAs of a cluster take shares of the key tiles of the same query tiles and merge their outputs (fwd_cluster_size).
template <int HD, typename T, int KIND, bool BSCALE = false, bool CL = false>
__global__ void __launch_bounds__(FwdRoles<HD, KIND>::NTHREADS, 1) fwd_kernel(const __grid_constant__ FwdKernelParams p) {
  // T is the element type of Q, K, V and of P: bf16 / fp16 (kind::f16) or FP8 e4m3 / e5m2 (kind::f8f6f4,
  // flash_sparse_attn/ops/triton/flash_sparse_fwd.py:49, :84-86 under IS_QUANT). Outputs and the gate
  // vectors are 16-bit (bf16 for FP8 inputs, flash_sparse_fwd.py:634).
  constexpr int ES = sizeof(T);
  constexpr bool F8 = ES == 1;
  constexpr int SLAB = 128 / ES;      // elements per 128-byte swizzle row
  using TO = typename OutType<T>::type;
  using SM = FwdSmem<HD, ES, KIND, CL>;
  using RO = FwdRoles<HD, KIND>;
  constexpr int KK_QK = HD * ES / 32;  // MMAs per S tile: every MMA consumes 32 bytes of the head dimension
  constexpr int KK_PV = TN * ES / 32;  // MMAs per P V tile: 32 bytes of the key dimension each
  constexpr int QT = FwdShape<HD>::QT, KSTAGES = FwdShape<HD>::KSTAGES, VSTAGES = FwdShape<HD>::VSTAGES;
  constexpr bool IS_BF16 = (sizeof(T) == 2) && !__is_same(T, __half);
  static_assert(!F8 || HD == 128, "FP8 tiles are one 128-byte swizzle row wide");
  constexpr uint32_t TMEM_S0 = 0, TMEM_O0 = 256;
  // FP8: P is handed to the MMA issuer in two halves, so that the first MMAs of P V run under the second half of the
  // exponentials (B2 S6000 causal, a call: 529 -> 510 us). With 16-bit inputs, whose P V takes twice as long, the second barrier
  // costs the issuer more than that gains (S = 16384: 1.91 -> 1.96 ms).
  constexpr bool HALVES = F8 && RO::HALVES == 1;
  // Who walks the tiles for the MMA issuer: the producer, ahead of time, except above head size 128 (not gated), where one query
  // tile leaves the issuer time and reading the producer's record costs more than the walk (dense causal S = 8192,
  // 16 / 4 heads of 192: 501 us, 523 with the record; a 1024-token window 183 and 187).
  constexpr bool HANDED = KIND == KIND_GATED || HD <= 128;

  after_previous();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  FwdBars* bars = reinterpret_cast<FwdBars*>(smem + SM::kBar);
  volatile int* abort_flag = &bars->abort_flag;

  // (through a shuffle: the roles' branches are then known to be the same for the whole warp)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const bool causal = p.flags & F_CAUSAL, local = p.flags & F_LOCAL, split_kv = p.flags & F_SPLIT;

  // ---- work decode: heads fastest (K/V reuse in L2), heavy query tiles first --------------------
  SeqInfo si;
  int pair;
  {
    int idx = CL ? blockIdx.x / p.cluster : blockIdx.x;
    si.head = idx % p.hgrid;
    idx /= p.hgrid;
    const int bs = idx % (p.B * p.num_splits);
    pair = p.num_pairs - 1 - idx / (p.B * p.num_splits);
    si.b = bs / p.num_splits;
    si.split = bs - si.b * p.num_splits;
    // Sequences of unequal length: the items in the order of their key tiles, most first, so that the longest CTAs are not
    // among the last to start (fsa_fwd_longest_first says when: four chunks of 500 queries at 2000 to 12 000 keys, 256 CTAs, 329 -> 245 us).
    // Every CTA ranks the items itself: one thread an item works out its key tiles and counts the items in front of it. (What is
    // decoded above stands unless they are ranked: decoding by way of the item cost CTAs of one key tile 1 %.)
    if (p.flags & F_LONGEST_FIRST) {
      int* tiles = reinterpret_cast<int*>(&bars->dl[0][0]);  // [items], then the item of this CTA; not in use yet
      const int items = p.B * p.num_pairs;
      int item = idx / p.num_splits;  // (query tile pair, sequence), sequences fastest, last pair first
      int mine = 0;
      if (tid < items) {
        const int b = tid % p.B, pr = p.num_pairs - 1 - tid / p.B;
        const int sq = (p.flags & F_USED_Q) ? p.used_q[b] : ((p.flags & F_VARLEN_Q) ? p.cu_q[b + 1] - p.cu_q[b] : p.sq);
        const int sk = (p.flags & F_USED_K) ? p.used_k[b] : ((p.flags & F_VARLEN_K) ? p.cu_k[b + 1] - p.cu_k[b] : p.sk);
        const int end = min((pr + 1) * QT * TM / p.gpack, sq);  // query rows of the pair end here
        if (pr * QT * TM < sq * p.gpack) mine = 1 + fsa_cdiv(max(causal ? min(end + sk - sq, sk) : sk, 0), TN);
        tiles[tid] = mine;
      }
      __syncthreads();
      if (tid < items) {
        int rank = 0;
        for (int j = 0; j < items; ++j) rank += tiles[j] > mine || (tiles[j] == mine && j < tid);
        if (rank == item) tiles[MAX_RANKED] = tid;
      }
      __syncthreads();
      item = __shfl_sync(0xffffffffu, tiles[MAX_RANKED], 0);  // known to be uniform: kept out of the threads' registers
      si.b = item % p.B;
      pair = p.num_pairs - 1 - item / p.B;
    }
    si.hkv = (p.flags & F_PACK_GQA) ? si.head : si.head / p.G;
    si.off_q = (p.flags & F_VARLEN_Q) ? p.cu_q[si.b] : 0;
    si.off_k = (p.flags & F_VARLEN_K) ? p.cu_k[si.b] : 0;
    si.sq = (p.flags & F_USED_Q) ? p.used_q[si.b]
                                 : ((p.flags & F_VARLEN_Q) ? p.cu_q[si.b + 1] - si.off_q : p.sq);
    si.sk = (p.flags & F_USED_K) ? p.used_k[si.b]
                                 : ((p.flags & F_VARLEN_K) ? p.cu_k[si.b + 1] - si.off_k : p.sk);
    if (local) {
      const int* wp = p.windows + (long long)si.hkv * p.win_stride;
      si.w.sink = wp[0];
      si.w.left = wp[1];
      si.w.right = wp[2];
      si.w.near_ = wp[3];
    } else {
      si.w.sink = si.w.left = si.w.right = si.w.near_ = 0;
    }
  }
  const int share = CL ? blockIdx.x % p.cluster : si.split, shares = CL ? p.cluster : p.num_splits;  // of the key tiles
  const int gpack = p.gpack;
  const int m_blocks_here = fsa_cdiv(si.sq * gpack, TM);  // query tiles this sequence really has
  if (pair * QT >= m_blocks_here) return;  // the grid is laid out for the longest sequence: nothing to do or to write

  // Both groups' schedules are needed by every role; gated: by those that walk the tiles, the softmax warps read the stager's.
  const bool walks = KIND != KIND_GATED || warp >= RO::W_PROD;
  FsaFwdSched sched[2];
  bool q_valid[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int mb = pair * QT + q;
    q_valid[q] = q < QT && mb < m_blocks_here;
    // One query position with windows and split-KV: the reference's rounding drops the first, partial tile of
    // the near band (block_info.py:60-64) although its eager ground truth sees those keys; like the decode
    // kernel, this one visits them (the flag only matters for that combination).
    if (walks)
      sched[q] = fsa_fwd_schedule(si.sq, si.sk, mb, share, si.w, shares, TN, TM, causal, local, split_kv || CL,
                                  gpack, /*cover_single_query=*/true);
    if (!walks || !q_valid[q] || fsa_fwd_sched_empty(sched[q])) {
      sched[q].n_min = sched[q].n_max = sched[q].n_max_no_mask = 0;
      sched[q].win_min = sched[q].win_max = sched[q].win_min_no_mask = sched[q].win_max_no_mask = 0;
      sched[q].sink_min = sched[q].sink_max = 0;
    }
  }
  auto first_tile = [&]() {
    const int a = fsa_fwd_next_tile_below(sched[0], 1 << 28, local);
    const int b = fsa_fwd_next_tile_below(sched[1], 1 << 28, local);
    return fsa_imax(a, b);
  };
  auto next_tile = [&](int n) {
    // common case first: the tile just below is visited by one of the two groups
    const int c = n - 1;
    if (!local && ((c >= sched[0].n_min && c < sched[0].n_max) || (c >= sched[1].n_min && c < sched[1].n_max))) return c;
    const int a = fsa_fwd_next_tile_below(sched[0], n, local);
    const int b = fsa_fwd_next_tile_below(sched[1], n, local);
    return fsa_imax(a, b);
  };

  // ---- gated: which tiles each group really computes ---------------------------------------------
  // The gate bound of a tile (flash_sparse_attn/ops/triton/activations.py:265-299) needs only the extremes of alpha
  // over the query tile and of delta over the key tile - both computed beforehand by gate_ext_kernel - and one
  // running scalar per query tile. The producer and the delta stager walk the tiles with their own copies of that
  // scalar and reach the same decisions; the producer passes them to the MMA issuer, the stager to the softmax warps. A
  // tile that both groups skip is never loaded, multiplied or staged (flash_gated_fwd.py:54-56 runs nothing for it).
  // The first tile of a group is never skipped: its running bound starts at -inf, the difference is +inf.
  float gw_amax[2] = {0.f, 0.f}, gw_amin[2] = {0.f, 0.f}, gw_thr[2] = {0.f, 0.f}, gw_run[2] = {-INFINITY, -INFINITY};
  float gw_c = 0.f;
  const float2* gw_dext = nullptr;
  if (KIND == KIND_GATED && walks) {
    gw_c = p.qkv_scale ? p.scale_log2 * p.qkv_scale[0] * p.qkv_scale[1] : p.scale_log2;
    const float2* aext = reinterpret_cast<const float2*>(p.gate_ws);
    gw_dext = aext + (long long)p.B * p.hgrid * p.num_m_blocks + ((long long)si.b * p.Hkv + si.hkv) * p.n_tiles_k;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int mb = pair * QT + q;
      if (mb < p.num_m_blocks) {
        const float2 e = __ldg(aext + ((long long)si.b * p.hgrid + si.head) * p.num_m_blocks + mb);
        gw_amax[q] = e.x;
        gw_amin[q] = e.y;
      }
      // flash_sparse_attn/ops/triton/seqlen_info.py:156-191: the adaptive bound is smallest at the tile's first row
      float g_thr = p.gate_thr;
      if (causal && (p.flags & F_ADAPT_GATE))
        g_thr = p.gate_thr * (float((mb * TM) / gpack + (si.sk - si.sq)) + 1.0f) / float(si.sk);
      gw_thr[q] = log2f(g_thr);
    }
  }
  // Next tile below n_prev that at least one group computes; keep[q] says which. `mark`: this thread records the
  // gate-skipped tiles in the tile map (value 3).
  auto walk_next = [&](int n_prev, bool* keep, bool mark) -> int {
    int n = next_tile(n_prev);
    if constexpr (KIND != KIND_GATED) {
      keep[0] = n >= 0 && fsa_fwd_tile_mode(sched[0], n, causal, local) >= 0;
      keep[1] = n >= 0 && fsa_fwd_tile_mode(sched[1], n, causal, local) >= 0;
      return n;
    } else {
    while (n >= 0) {
      const float2 de = __ldg(gw_dext + n);  // (max, min) of delta over the key tile
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        keep[q] = fsa_fwd_tile_mode(sched[q], n, causal, local) >= 0;
        if (keep[q]) {
          const float gmc = fmaxf(fmaxf(gw_amax[q] * de.x, gw_amax[q] * de.y), fmaxf(gw_amin[q] * de.x, gw_amin[q] * de.y));
          const bool skip = (gmc - gw_run[q]) * gw_c < gw_thr[q];
          if (!skip) gw_run[q] = fmaxf(gmc, gw_run[q]);
          keep[q] = !skip;
          if (skip && mark && p.tile_map) {
            const int mb = pair * QT + q;
            p.tile_map[((((long long)si.b * p.hgrid + si.head) * p.num_m_blocks + mb) * p.num_splits + si.split) *
                           p.n_tiles_k + n] = 3;
          }
        }
      }
      if (keep[0] || keep[1]) return n;
      n = next_tile(n);
    }
    keep[0] = keep[1] = false;
    return -1;
    }
  };
  constexpr int WALK_START = 1 << 28;

  // ---- setup ---------------------------------------------------------------------------------
  if (tid == 0) {
    mbar_init(&bars->q_full, 1);
    mbar_init(&bars->k0_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->kv_full[s], 2);
      mbar_init(&bars->kv_empty[s], 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(&bars->s_full[q], 1);
      mbar_init(&bars->p_full[q], RO::GW);  // one arrival per warp of the group
      mbar_init(&bars->p_rest[q], 4);
      mbar_init(&bars->o_final[q], 1);
      mbar_init(&bars->wg_sync[q], RO::GW);
      for (int w = 0; w < 4; ++w) mbar_init(&bars->pair_sync[q][w], 2);
      mbar_init(&bars->d_full[q], 1);
      mbar_init(&bars->d_empty[q], 2 * RO::GW);
    }
    bars->abort_flag = (*reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    mbar_fence_init();
  }
  if (warp == RO::W_PROD) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  [[maybe_unused]] auto cluster_sync = []() { cooperative_groups::this_cluster().sync(); };
  [[maybe_unused]] auto peer = [](auto* ptr, int rank) { return cooperative_groups::this_cluster().map_shared_rank(ptr, rank); };
  const int kv_row_coord_b = (p.flags & (F_VARLEN_K | F_PAGED)) ? 0 : si.b;

  // Register budget: a softmax thread holds a 128-wide fp32 score row (gated: 32 scores at a time) and takes the registers
  // that the last warpgroup does not need: 384 x 168 at launch = 256 x 216 + 128 x 72, gated 640 x 96 = 512 x 104 + 128 x 64.
  if (warp >= RO::W_PROD) {
    // last warpgroup: all four warps release registers at the same instruction
    if constexpr (RO::HALVES == 1)
      asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    else
      asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  if (warp == RO::W_PROD) {
    // =============================== producer ================================================
    if (lane == 0 && !*abort_flag) {
      tma_prefetch_desc(&p.map_q);
      tma_prefetch_desc(&p.map_k);
      tma_prefetch_desc(&p.map_v);
      // Q tiles
      {
        uint32_t bytes = 0;
        for (int q = 0; q < 2; ++q)
          if (q_valid[q]) bytes += SM::kTileBytes;
        if (bytes) {
          mbar_arrive_expect_tx(&bars->q_full, bytes);
          for (int q = 0; q < 2; ++q) {
            if (!q_valid[q]) continue;
            const int mb = pair * QT + q;
            uint8_t* dst = smem + SM::kQ + q * SM::kTileBytes;
            const int row0 = (mb * TM) / gpack;  // token index of the tile's first row
            const int head0 = (p.flags & F_PACK_GQA) ? si.hkv * p.G : si.head;
            const int bq = (p.flags & F_VARLEN_Q) ? 0 : si.b;
            for (int d = 0; d < HD; d += SLAB)
              tma_load_4d(dst + (d / SLAB) * (TM * 128), &p.map_q, &bars->q_full, d, head0, si.off_q + row0, bq);
          }
        }
      }
      auto load_kv = [&](const CUtensorMap* map, uint8_t* dst, uint64_t* bar, int n) {
        // one 128-key tile = HD/64 column slabs x (paged: several pages | one box)
        if (p.flags & F_PAGED) {
          // (shifts and masks: page sizes are powers of two, and two divisions a box cost the one lane that requests the tiles more
          // than a step has to spare. Chunks of 500 queries over four caches of 2000 to 12 000 keys, pages of 256: 237 -> 215 us, of
          // 8000 keys in pages of 64: 371 -> 255.)
          const int page_shift = 31 - __clz(p.page_size), row_shift = min(page_shift, 7);
          const int rows_per_box = 1 << row_shift, nbox = TN >> row_shift;
          uint32_t bytes = 0;
          int pages[4];
          for (int i = 0; i < nbox; ++i) {
            const int r0 = n * TN + i * rows_per_box;
            pages[i] = (r0 < si.sk) ? p.page_table[(long long)si.b * p.pt_stride + (r0 >> page_shift)] : -1;
            if (pages[i] >= 0) bytes += rows_per_box * HD * ES;
          }
          mbar_arrive_expect_tx(bar, bytes);
          for (int i = 0; i < nbox; ++i) {
            if (pages[i] < 0) continue;
            const int r0 = n * TN + i * rows_per_box;
            for (int d = 0; d < HD; d += SLAB)
              tma_load_4d(dst + (d / SLAB) * (TN * 128) + i * rows_per_box * 128, map, bar, d, si.hkv,
                          r0 & (p.page_size - 1), pages[i]);
          }
        } else {
          mbar_arrive_expect_tx(bar, SM::kTileBytes);
          for (int d = 0; d < HD; d += SLAB)
            tma_load_4d(dst + (d / SLAB) * (TN * 128), map, bar, d, si.hkv, si.off_k + n * TN, kv_row_coord_b);
        }
      };
      int t = 0, seen = 0;
      bool ok = true;
      // Which tile comes next and who takes part in it is worked out here, ahead of time, and handed to the MMA issuer with
      // the barrier that it waits on anyway: on windowed schedules the walk took the issuer 925 of the 4250 cycles of
      // a step, in which the tensor pipe had nothing to do.
      [[maybe_unused]] bool act[2], act_next[2];
      auto take_part = [&](int n_t, bool* a) {  // not gated: the groups whose schedule has tile n_t
#pragma unroll
        for (int q = 0; q < 2; ++q) a[q] = n_t >= 0 && fsa_fwd_tile_mode(sched[q], n_t, causal, local) >= 0;
      };
      auto publish = [&](int slot, int n_t, const bool* a, unsigned last) {
        const unsigned f = (a[0] ? 1u : 0u) | (a[1] ? 2u : 0u) | (last << 2);
        *reinterpret_cast<volatile unsigned long long*>(&bars->step_info[slot]) =
            (unsigned long long)(unsigned)n_t | ((unsigned long long)f << 32);
      };
      int n;
      if constexpr (KIND == KIND_GATED) {
        n = walk_next(WALK_START, act, false);
      } else {
        n = first_tile();
        if constexpr (HANDED) take_part(n, act);
      }
      if constexpr (HANDED) publish(2, n, act, 0u);
      if (n >= 0) {
        load_kv(&p.map_k, smem + SM::kK, &bars->k0_full, n);
      } else {
        mbar_arrive(&bars->k0_full);
        if (q_valid[0] || q_valid[1]) ok = mbar_wait(&bars->q_full, 0, abort_flag);  // nobody else waits for Q to land
      }
      while (n >= 0 && ok) {
        int n_next;
        [[maybe_unused]] unsigned last = 0u;  // gated: not known before the next gate is; its output barriers follow the loop
        if constexpr (KIND == KIND_GATED) {
          n_next = walk_next(n, act_next, false);
        } else {
          n_next = next_tile(n);
          if constexpr (HANDED) {
            take_part(n_next, act_next);
#pragma unroll
            for (int q = 0; q < 2; ++q)
              if (act[q] && fsa_fwd_next_tile_below(sched[q], n, local) < 0) last |= 1u << q;
          }
        }
        // Release signals arrive in order (signal c: K(c) and V(c - 1) consumed). V(t) goes into the slot of
        // V(t - 2) and K(t + 1) into the slot of K(t - 1): both free after signal t - 1.
        auto need_signal = [&](int c) {
          while (ok && seen <= c) {
            ok = mbar_wait(&bars->kv_empty[seen & 1], (seen >> 1) & 1, abort_flag);
            ++seen;
          }
        };
        // V(t) replaces V(t - VSTAGES), K(t + 1) replaces K(t + 1 - KSTAGES): both are free after this signal
        need_signal(t - (KSTAGES < VSTAGES ? KSTAGES : VSTAGES) + 1);
        if (!ok) break;
        // the issuer has read the slot's last word: it came before signal t - 1
        if constexpr (HANDED) publish(t & 1, n_next, act_next, last);
        // V is prefetched like K, before the softmax groups have voted on the tile: waiting for the vote
        // would put a full load latency between every S tile and its P V product, and in this
        // tensor-bound kernel a V tile that ends up unused only costs an L2 read: on inputs where 82 % of the
        // tiles are skipped, leaving ALL V loads out changed the kernel time by 1 % (1.476 -> 1.462 ms at
        // S = 16384), so L2 traffic is not what a skipped tile costs. (The reference skips the load,
        // flash_sparse_fwd.py:60-88; it matters there because its tiles are loaded by the same warps that
        // compute.) A skipped tile still skips the softmax work and the P V product.
        load_kv(&p.map_v, smem + SM::kV + (t % VSTAGES) * SM::kTileBytes, &bars->kv_full[t & 1], n);
        if (n_next >= 0)
          load_kv(&p.map_k, smem + SM::kK + ((t + 1) % KSTAGES) * SM::kTileBytes, &bars->kv_full[t & 1], n_next);
        else
          mbar_arrive(&bars->kv_full[t & 1]);  // the barrier counts two arrivals per step
        n = n_next;
        if constexpr (HANDED) {
          act[0] = act_next[0];
          act[1] = act_next[1];
        }
        ++t;
      }
    }
    __syncwarp();
  } else if (warp == RO::W_STAGE) {
    // =============================== delta stager (gated only) ================================
    // delta of every computed key tile as fp32 in a 2-slot ring, with the tile's index and the groups' mask modes, so
    // that the softmax warps need not walk the schedule (1600 to 2200 cycles a tile on their critical path)
    // (flash_sparse_attn/ops/triton/flash_gated_fwd.py:100-115). Keys past the sequence
    // read as 0, like the reference's masked load (scheduler.py:1674-1691).
    if (KIND == KIND_GATED) {
      bool ok = !*abort_flag;
      const TO* dbase = reinterpret_cast<const TO*>(p.delta);
      int t = 0;
      bool keep[2];
      for (int n = walk_next(WALK_START, keep, lane == 0); ok; n = walk_next(n, keep, lane == 0), ++t) {
        const int s = t & 1, use = t >> 1;
        if (use > 0) ok = mbar_wait(&bars->d_empty[s], (use - 1) & 1, abort_flag);
        if (!ok) break;
        if (n >= 0) {
          float dv[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = n * TN + lane * 4 + j;
            float v = 0.f;
            if (k < si.sk) {
              long long e;
              if (p.flags & F_PAGED) {
                const int page = p.page_table[(long long)si.b * p.pt_stride + k / p.page_size];
                e = (long long)page * p.d_sb + (long long)si.hkv * p.d_sh + (k % p.page_size);
              } else {
                e = (long long)((p.flags & F_VARLEN_K) ? 0 : si.b) * p.d_sb + (long long)si.hkv * p.d_sh + si.off_k + k;
              }
              v = float(dbase[e]);
            }
            dv[j] = v;
          }
          *reinterpret_cast<float4*>(&bars->dl[s][lane * 4]) = make_float4(dv[0], dv[1], dv[2], dv[3]);
        }
        if (lane == 0)
          *reinterpret_cast<int4*>(&bars->dl[s][TN]) =
              make_int4(n, n >= 0 && keep[0] ? fsa_fwd_tile_mode(sched[0], n, causal, local) : -1,
                        n >= 0 && keep[1] ? fsa_fwd_tile_mode(sched[1], n, causal, local) : -1, 0);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->d_full[s]);
        if (n < 0) break;
      }
    }
  } else if (warp == RO::W_MMA) {
    // =============================== MMA issuer ==============================================
    constexpr int F8_FMT = __is_same(T, __nv_fp8_e5m2) ? 1 : 0;
    constexpr uint32_t idesc_s = F8 ? umma_idesc_f8(TM, TN, F8_FMT, F8_FMT, false, false)
                                    : umma_idesc_f16(TM, TN, IS_BF16, false, false);
    constexpr uint32_t idesc_o = F8 ? umma_idesc_f8(TM, HD, F8_FMT, F8_FMT, false, true)
                                    : umma_idesc_f16(TM, HD, IS_BF16, false, true);
    // What this warp branches on is made the same in all lanes in a way that the compiler sees, so that it keeps the MMAs'
    // operands in uniform registers; TMEM starts at 0 because all of it is allocated. Sparse causal S = 16384 1859 -> 1830 us,
    // a 1024-token window (B4 S8192) 1000 -> 970, but the 16-bit dense kind then spills around it (1764 -> 1793) and goes without.
    constexpr bool UNIFORM = KIND != KIND_DENSE || F8;
    auto wait_for = [](uint64_t* bar, uint32_t parity, volatile int* abort) {
      return UNIFORM ? mbar_wait_uniform(bar, parity, abort) : mbar_wait(bar, parity, abort);
    };
    const uint32_t tm = UNIFORM ? 0u : tmem_base;
    const uint32_t sQ = smem_u32(smem + SM::kQ), sK = smem_u32(smem + SM::kK), sV = smem_u32(smem + SM::kV);
    bool ok = UNIFORM ? (bool)__any_sync(0xffffffffu, !*abort_flag) : !*abort_flag;
    int cnt[2] = {0, 0}, cnt_kept[2] = {0, 0};
    bool o_started[2] = {false, false};
    bool act[2] = {false, false}, last[2];
    int n = -1;
    [[maybe_unused]] auto read_info = [&](int slot, int& n_t, unsigned& f) {
      unsigned long long w = *reinterpret_cast<const volatile unsigned long long*>(&bars->step_info[slot]);
      if (UNIFORM) w = __shfl_sync(0xffffffffu, w, 0);
      n_t = (int)(unsigned)w;
      f = (unsigned)(w >> 32);
    };
    // Every lane runs the same (warp-uniform) descriptor arithmetic; the MMA and commit instructions carry the
    // one-lane predicate themselves.
    const uint32_t lead = elect_one();
    const uint32_t dq_lo = umma_desc_lo(sQ, 16), dk_lo = umma_desc_lo(sK, 16), dv_lo = umma_desc_lo(sV, TN * 128);
    // The MMA loops are unrolled in the dense and sparse kinds (rolled: sparse causal S = 16384 1830 -> 2006 us, FP8 472 -> 502)
    // and stay rolled in the gated kind, whose softmax warps carry the gate arithmetic.
    constexpr int ISSUE_UNROLL = (KIND == KIND_GATED) ? 1 : 8;
    auto p_col = [](int kk) {  // where P of the kk-th MMA lies: each thread of a row writes it over the front of its own scores
      return kk * 8 + (RO::HALVES == 2 && kk >= KK_PV / 2 ? TN / 2 - KK_PV / 2 * 8 : 0);
    };
    auto issue_s = [&](int q, int ks) {
      const uint32_t aq = dq_lo + ((q * SM::kTileBytes) >> 4), bk = dk_lo + ((ks * SM::kTileBytes) >> 4);
#pragma unroll ISSUE_UNROLL
      for (int kk = 0; kk < KK_QK; ++kk) {
        const uint32_t koff = (kk >> 2) * (TM * 128) + (kk & 3) * 32;
        if (F8)
          umma_f8_ss_lead(lead, tm + TMEM_S0 + q * 128, umma_desc_at(aq, koff), umma_desc_at(bk, koff), idesc_s,
                          kk > 0);
        else
          umma_ss_lead(lead, tm + TMEM_S0 + q * 128, umma_desc_at(aq, koff), umma_desc_at(bk, koff), idesc_s,
                       kk > 0);
      }
      umma_commit_lead(lead, &bars->s_full[q]);
    };
    if constexpr (!HANDED) {
      n = first_tile();
#pragma unroll
      for (int q = 0; q < 2; ++q) act[q] = n >= 0 && fsa_fwd_tile_mode(sched[q], n, causal, local) >= 0;
    }
    if (ok) ok = wait_for(&bars->k0_full, 0, abort_flag);
    if constexpr (HANDED) {
      if (ok) {
        unsigned f;
        read_info(2, n, f);
        act[0] = f & 1u;
        act[1] = f & 2u;
      }
    }
    if (n >= 0 && ok) {
      ok = wait_for(&bars->q_full, 0, abort_flag);
      tc_fence_after();
      if (ok) {
        for (int q = 0; q < 2; ++q)
          if (act[q]) issue_s(q, 0);
        umma_commit_lead(lead, &bars->kv_empty[0]);
      }
    }
    int t = 0;
    // What this warp does between a group publishing P and the next MMA is time the tensor pipe idles: the producer walks the
    // tiles and says who takes part in the next one, and the K / V arrivals are handled before the wait for P. (One issuer
    // per group was tried: the second polling warp slows the softmax warps of its scheduler more than the overlap gains.)
    while (n >= 0 && ok) {
      bool act_next[2];
      const int vs = t % VSTAGES;
      const int ks_next = (t + 1) % KSTAGES;
      int n_next;
      if constexpr (!HANDED) {
        n_next = next_tile(n);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (!local) {  // one contiguous range of tiles per group
            act_next[q] = n_next >= sched[q].n_min && n_next < sched[q].n_max;
            last[q] = act[q] && n == sched[q].n_min;
          } else {
            act_next[q] = n_next >= 0 && fsa_fwd_tile_mode(sched[q], n_next, causal, local) >= 0;
            last[q] = act[q] && fsa_fwd_next_tile_below(sched[q], n, local) < 0;
          }
        }
      }
      ok = wait_for(&bars->kv_full[t & 1], (t >> 1) & 1, abort_flag);  // V(t) and K(t + 1)
      if (!ok) break;
      if constexpr (HANDED) {
        unsigned f;
        read_info(t & 1, n_next, f);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          act_next[q] = (f >> q) & 1u;
          last[q] = (f >> (2 + q)) & 1u;
        }
      }
      if ((p.flags & F_KV_RAGGED) && (n + 1) * TN > si.sk) {
        // keys past the sequence end carry probability 0 but their V rows may hold
        // anything: clear them so that 0 * garbage cannot produce NaN
        const int r0 = si.sk - n * TN;
        uint8_t* vt = smem + SM::kV + vs * SM::kTileBytes;
        constexpr int CPR = HD * ES / 16;  // 16-byte chunks per row
        for (int i = lane; i < (TN - r0) * CPR; i += 32) {
          const int r = r0 + i / CPR, c = i % CPR;
          *reinterpret_cast<uint4*>(vt + (c >> 3) * (TN * 128) + sw128_offset(r, c & 7)) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
        __syncwarp();
      }
      const uint32_t bv = dv_lo + ((vs * SM::kTileBytes) >> 4);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (act[q]) {
          // A skipped tile is known from the votes, all of which come after their warps have read the scores: the next scores are
          // issued at once, while the group is still finding out. The votes of a kept tile are there long before its P. (Verdict
          // passed on by the group: prompts of S = 16384 with concentrated attention, 8 / 2 heads 346 us, with the votes 304, 6000
          // tokens x 32 heads 225 and 214, without any skips S = 4096 143.0 and 142.0. Looking for P first, after a kept tile: 337, 221, 141.6.)
          bool skip = false;
          if (KIND != KIND_DENSE) {
            ok = wait_for(&bars->wg_sync[q], cnt[q] & 1, abort_flag);
            if (!ok) break;
            int votes = 0;
#pragma unroll
            for (int w = 0; w < RO::GW; w += 4) {
              const int4 v4 = *reinterpret_cast<const int4*>(&bars->vote_any[q][cnt[q] & 1][w]);
              votes |= v4.x | v4.y | v4.z | v4.w;
            }
            // the maximum over rows ignores rows that are not numbers; a tile is skipped iff that maximum is < 0
            skip = __all_sync(0xffffffffu, votes == 2);
          }
          cnt[q]++;
          if (!skip) {
            ok = wait_for(&bars->p_full[q], cnt_kept[q] & 1, abort_flag);
            if (!ok) break;
          }
          tc_fence_after();
          if (!skip) {
#pragma unroll ISSUE_UNROLL
            for (int kk = 0; kk < KK_PV; ++kk) {
              if (HALVES && kk == KK_PV / 2) {
                ok = wait_for(&bars->p_rest[q], cnt_kept[q] & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
              }
              if (F8)
                umma_f8_ts_lead(lead, tm + TMEM_O0 + q * 128, tm + TMEM_S0 + q * 128 + p_col(kk),
                                umma_desc_at(bv, kk * 4096), idesc_o, (kk > 0 || o_started[q]) ? 1u : 0u);
              else
                umma_ts_lead(lead, tm + TMEM_O0 + q * 128, tm + TMEM_S0 + q * 128 + p_col(kk),
                             umma_desc_at(bv, kk * 2048), idesc_o, (kk > 0 || o_started[q]) ? 1u : 0u);
            }
            o_started[q] = true;
            cnt_kept[q]++;
          }
          // last key tile of this group: tell it when its output is complete
          if (last[q]) umma_commit_lead(lead, &bars->o_final[q]);
        }
        if (act_next[q]) {
          if (!act[q]) tc_fence_after();
          issue_s(q, ks_next);
        }
      }
      if (!ok) break;
      // signal t + 1: V(t) and K(t + 1) are free once the MMAs issued so far have completed
      umma_commit_lead(lead, &bars->kv_empty[(t + 1) & 1]);
      n = n_next;
      act[0] = act_next[0];
      act[1] = act_next[1];
      ++t;
    }
    if (KIND == KIND_GATED && ok) {
      // completion of everything issued so far = both outputs are final
      for (int q = 0; q < 2; ++q)
        if (o_started[q]) umma_commit_lead(lead, &bars->o_final[q]);
    }
  }
  if constexpr (CL) {  // the softmax warps merge between the two; these have too few registers to take part
    __syncwarp();
    cluster_sync();
    cluster_sync();
  }
  } else {
    // =============================== softmax groups ==========================================
    if constexpr (RO::HALVES == 1)
      asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    else
      asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    constexpr int NC = TN / RO::HALVES;                    // key columns of a thread
    constexpr int OC = HD / RO::HALVES;                    // output columns of a thread
    const int q = RO::HALVES == 1 ? warp >> 2 : warp >> 3;   // group / query tile (a shift: a signed division costs FP8 1.8 %)
    const int half = RO::HALVES == 1 ? 0 : (warp >> 2) & 1;  // which key (and output) columns
    const int wq = warp & 3;        // warp within group == TMEM lane quadrant
    const int row = wq * 32 + lane; // row within the tile
    const int mb = pair * QT + q;
    const uint32_t lane_addr = uint32_t(wq * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + TMEM_S0 + q * 128 + half * NC;
    const uint32_t tO = tmem_base + lane_addr + TMEM_O0 + q * 128 + half * OC;

    const int offs_m = mb * TM + row;
    const int q_idx = offs_m / gpack;
    const int q_head = (p.flags & F_PACK_GQA) ? si.hkv * p.G + (offs_m - q_idx * gpack) : si.head;
    RowMask rm;
    rm.row_ok = q_idx < si.sq;
    rm.sk = si.sk;
    rm.diag = q_idx + (si.sk - si.sq);
    rm.near_lo = rm.diag - si.w.near_;
    rm.far_hi = rm.diag - si.w.near_ - si.w.right;
    rm.far_lo = rm.far_hi - si.w.left;
    rm.sink_hi = si.w.sink;
    const FsaFwdSched my = sched[q];  // registers, not the indexed copy

    float thr_log2 = 0.f;
    if (KIND != KIND_DENSE) {
      // flash_sparse_attn/ops/triton/seqlen_info.py:118-153
      const float visible = causal ? float(q_idx + (si.sk - si.sq) + 1) : float(si.sk);
      thr_log2 = log2f(fmaxf(fminf(p.softmax_thr / visible, 1.0f), 0.0f));
    }
    // Block-scaled FP8: the scale of the logits changes from key tile to key tile, so the scores are multiplied by it
    // right after they leave TMEM and everything below works on scaled logits (cc = 1). The value block's scale is
    // folded into P relative to a running reference v_run - the largest value scale this row has met so far - and
    // the output accumulator is rescaled when that reference grows (like the running maximum); the output is
    // multiplied by the final reference. Blocks more than 2^9 below the running reference underflow in FP8 P, i.e.
    // contributions that small relative to the largest block a row has seen are dropped.
    constexpr bool bscaled = F8 && BSCALE;
    const float* kbs = bscaled ? p.k_bscale + ((long long)si.b * p.Hkv + si.hkv) * p.n_tiles_k : nullptr;
    const float* vbs = bscaled ? p.v_bscale + ((long long)si.b * p.Hkv + si.hkv) * p.n_tiles_k : nullptr;
    const float c = bscaled ? p.scale_log2 * p.q_bscale[((long long)si.b * p.Hq + q_head) * p.num_m_blocks +
                                                        (mb < p.num_m_blocks ? mb : 0)]
                            : (p.qkv_scale ? p.scale_log2 * p.qkv_scale[0] * p.qkv_scale[1] : p.scale_log2);
    const float cc = bscaled ? 1.0f : c;  // factor between the values held in sr[] and base-2 logits
    float v_run = 0.f;  // block-scaled: running reference of the value scale (uniform over the tile's rows)
    const float v_scale = p.qkv_scale ? p.qkv_scale[2] : p.v_scale;
    float m_ref = -INFINITY;  // reference maximum all stored exponentials are relative to
    float l_ref = 0.f;        // sum of exp2((s - m_ref) * c) over this thread's columns
    float lg_l = -INFINITY;   // log2(l_ref) for the skip test, refreshed at the end of a tile (off the S -> P path)
    bool have_o = false;      // some P V has been issued for this tile
    int cnt_s = 0;
    bool ok = !*abort_flag;
    const bool has_work = q_valid[q] && !fsa_fwd_sched_empty(my);

    // ---- gated: alpha of this row ----------------------------------------------------------------------
    float alpha = 0.f;
    if (KIND == KIND_GATED) {
      if (rm.row_ok && q_valid[q]) {
        const TO* ab = reinterpret_cast<const TO*>(p.alpha);
        alpha = float(ab[(long long)((p.flags & F_VARLEN_Q) ? 0 : si.b) * p.a_sb + (long long)q_head * p.a_sh +
                         si.off_q + q_idx]);
        if (p.flags & F_LOGSIGMOID) alpha *= 1.4426950408889634f;
      }
    }

    int t_merged = -1;
    int n = -1;
    if (KIND != KIND_GATED && has_work) n = first_tile();
    for (; (KIND == KIND_GATED || n >= 0) && ok; n = (KIND == KIND_GATED) ? n : next_tile(n)) {
      ++t_merged;
      int mode;
      const int ds = t_merged & 1;
      if constexpr (KIND == KIND_GATED) {
        // every tile that one of the groups computes was staged by the delta warp, with its index and mask modes
        ok = mbar_wait(&bars->d_full[ds], (t_merged >> 1) & 1, abort_flag);
        if (!ok) break;
        const int4 info = *reinterpret_cast<const int4*>(&bars->dl[ds][TN]);
        n = info.x;
        if (n < 0) break;
        mode = q == 0 ? info.y : info.z;
        if (mode < 0) {  // not in this group's schedule, or skipped by its gate: nothing was issued for it
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->d_empty[ds]);
          continue;
        }
      } else {
        mode = has_work ? fsa_fwd_tile_mode(my, n, causal, local) : -1;
        if (mode < 0) continue;
      }
      const int par = cnt_s & 1;
      if (KIND != KIND_GATED) {
        ok = mbar_wait(&bars->s_full[q], par, abort_flag);
        if (!ok) break;
        tc_fence_after();
      }
      cnt_s++;
      const int k0 = n * TN;

      // ---- scores of this row: TMEM -> registers (warp-collective loads, one wait) ---------------
      // Gated kind: 32 columns at a time, and the gated and masked logits go back to TMEM, from where the exponentials
      // below read them in pieces again: with the whole row in registers beside the gate's arithmetic the softmax
      // warps spill (64 columns in the registers of two threads a row: 200 bytes, 10 % slower). The other
      // kinds hold the row: reading it twice costs them 17 % (dense, S = 16384: 1.93 -> 2.27 ms).
      constexpr bool GATED = KIND == KIND_GATED;
      uint32_t sr[GATED ? 32 : TN];
      float p_mul = 1.0f, o_mul = 1.0f;
      float m_cur;
      if constexpr (GATED) {
        TileMask tm = {{0, 0, 0}, {0u, 0u, 0u}};
        if (mode != FSA_MASK_NONE) tm = make_tile_mask(rm, mode, k0);
        // NaN: the maximum of a row without any number is NaN (it then takes no part in the vote)
        float mx[4] = {__int_as_float(0x7fffffff), __int_as_float(0x7fffffff), __int_as_float(0x7fffffff),
                       __int_as_float(0x7fffffff)};
        const float2 al2 = make_float2(alpha, alpha);  // times log2(e) for the logsigmoid gate, whose exponential is 2^x
        const bool logsig = p.flags & F_LOGSIGMOID;
        // logits = (q.k + g(alpha * delta_j)) * scale, g = logsigmoid or identity (flash_sparse_attn/ops/triton/flash_gated_fwd.py:104-122,
        // activations.py:245-262). Two threads a row work the first 32 gates out before the scores are waited for. One thread a row (head sizes
        // above 128) takes gate and score together: with the gates first head size 192, S = 4096, 16 / 4 heads takes 245 us, so 233; with
        // an identity gate 205 and 189. Both loops are rolled up: unrolled over
        // the row, the gate's code alone is larger than the instruction caches hold beside the other roles', and its 128 columns took 6700 cycles.
        if constexpr (RO::HALVES == 1) {
          ok = mbar_wait(&bars->s_full[q], par, abort_flag);
          if (!ok) break;
          tc_fence_after();
#pragma unroll 1
          for (int ch = 0; ch < TN / 32; ++ch) {
            uint32_t r[32];
            tmem_ld32(tS + ch * 32, r);
            tmem_ld_wait();
            const float4* d4 = reinterpret_cast<const float4*>(&bars->dl[ds][ch * 32]);
            if (logsig) {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 dd = d4[i >> 2];
                const float2 a = add_log_sigmoid2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])),
                                                  mul2(al2, make_float2(dd.x, dd.y)));
                const float2 b = add_log_sigmoid2(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])),
                                                  mul2(al2, make_float2(dd.z, dd.w)));
                r[i] = __float_as_uint(a.x);
                r[i + 1] = __float_as_uint(a.y);
                r[i + 2] = __float_as_uint(b.x);
                r[i + 3] = __float_as_uint(b.y);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                const float4 dd = d4[i >> 2];
                r[i] = __float_as_uint(fmaf(alpha, dd.x, __uint_as_float(r[i])));
                r[i + 1] = __float_as_uint(fmaf(alpha, dd.y, __uint_as_float(r[i + 1])));
                r[i + 2] = __float_as_uint(fmaf(alpha, dd.z, __uint_as_float(r[i + 2])));
                r[i + 3] = __float_as_uint(fmaf(alpha, dd.w, __uint_as_float(r[i + 3])));
              }
            }
            if (mode != FSA_MASK_NONE) {
              mask_cols32(r, tile_bits(tm, ch * 32));
            } else if (!rm.row_ok) {
              // rows past the query length read as zero scores in fully visible tiles
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0u;
            }
            tmem_st32(tS + ch * 32, r);
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mx[j] = max3(mx[j], __uint_as_float(r[i + 2 * j]), __uint_as_float(r[i + 2 * j + 1]));
            }
          }
        } else {
#pragma unroll 1
        for (int ch = 0; ch < NC / 32; ++ch) {
          float2 g[16];
          {
            float4 dd[8];
            const float4* d4 = reinterpret_cast<const float4*>(&bars->dl[ds][half * NC + ch * 32]);
#pragma unroll
            for (int i = 0; i < 8; ++i) dd[i] = d4[i];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              g[2 * i] = mul2(al2, make_float2(dd[i].x, dd[i].y));
              g[2 * i + 1] = mul2(al2, make_float2(dd[i].z, dd[i].w));
            }
          }
          if (logsig) {
#pragma unroll
            for (int i = 0; i < 16; ++i) g[i] = log_sigmoid2(g[i]);
          }
          if (ch == 0) {
            ok = mbar_wait(&bars->s_full[q], par, abort_flag);
            if (!ok) break;
            tc_fence_after();
          }
          const uint32_t bits = mode != FSA_MASK_NONE ? tile_bits(tm, half * NC + ch * 32) : 0u;
#pragma unroll
          for (int h = 0; h < 32; h += 16) {
            uint32_t r[16];
            tmem_ld16(tS + ch * 32 + h, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              const float2 v = add2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), g[(h + i) >> 1]);
              r[i] = __float_as_uint(v.x);
              r[i + 1] = __float_as_uint(v.y);
            }
            if (mode != FSA_MASK_NONE) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (!(bits & (1u << (h + i)))) r[i] = 0xff800000u;
            } else if (!rm.row_ok) {
              // rows past the query length read as zero scores in fully visible tiles
#pragma unroll
              for (int i = 0; i < 16; ++i) r[i] = 0u;
            }
            tmem_st16(tS + ch * 32 + h, r);
#pragma unroll
            for (int i = 0; i < 16; i += 8) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mx[j] = max3(mx[j], __uint_as_float(r[i + 2 * j]), __uint_as_float(r[i + 2 * j + 1]));
            }
          }
        }
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->d_empty[ds]);
        m_cur = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // The other half of the row: its maximum, and its sum up to the tile before. (It has read this thread's values of that tile
        // before it voted, without which this tile's scores were not issued.)
        if constexpr (RO::HALVES == 2) {
          float2* xch = reinterpret_cast<float2*>(smem + SM::kXch) + q * 256;
          xch[half * 128 + row] = make_float2(m_cur, l_ref);
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->pair_sync[q][wq]);
          ok = mbar_wait(&bars->pair_sync[q][wq], par, abort_flag);
          if (!ok) break;
          const float2 other = xch[(half ^ 1) * 128 + row];
          m_cur = fmaxf(m_cur, other.x);
          lg_l = lg2_approx(l_ref + other.y);
        }
      } else {
#pragma unroll
      for (int ch = 0; ch < TN / 32; ++ch) tmem_ld32(tS + ch * 32, &sr[ch * 32]);
      tmem_ld_wait();
      if constexpr (F8) {
        if (bscaled) {
          const float ct = c * kbs[n];
#pragma unroll
          for (int i = 0; i < TN; ++i) sr[i] = __float_as_uint(__uint_as_float(sr[i]) * ct);
        }
      }
      if (mode != FSA_MASK_NONE) {
        const TileMask tm = make_tile_mask(rm, mode, k0);
#pragma unroll
        for (int ch = 0; ch < TN / 32; ++ch) mask_cols32(&sr[ch * 32], tile_bits(tm, ch * 32));
      } else if (!rm.row_ok) {
        // rows past the query length read as zero scores in fully visible tiles
#pragma unroll
        for (int i = 0; i < TN; ++i) sr[i] = 0u;
      }

      // ---- row maximum ------------------------------------------------------------------------------
      float mx[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        mx[j] = fmaxf(__uint_as_float(sr[j * 32]), __uint_as_float(sr[j * 32 + 1]));
#pragma unroll
        for (int i = 2; i < 32; i += 2)
          mx[j] = max3(mx[j], __uint_as_float(sr[j * 32 + i]), __uint_as_float(sr[j * 32 + i + 1]));
      }
      m_cur = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      }

      // ---- tile skip vote (flash_sparse_attn/ops/triton/activations.py:129-138) -----------------
      bool skip = false;
      if (KIND != KIND_DENSE) {
        const float d = (m_cur - m_ref) * cc - lg_l;
        const float val = d - thr_log2;
        const unsigned want = __ballot_sync(0xffffffffu, val >= 0.0f);
        const unsigned drop = __ballot_sync(0xffffffffu, val < 0.0f);
        // group-wide exchange through a (bounded) mbarrier rather than bar.sync, so that an
        // aborting pipeline can never leave part of the group parked on a hardware barrier
        // After the last vote the MMA issuer may write the next scores over these.
        if (GATED) tmem_st_wait();
        tc_fence_before();
        if (lane == 0) {
          bars->vote_any[q][par][half * 4 + wq] = (want ? 1 : 0) | (drop ? 2 : 0);
          mbar_arrive(&bars->wg_sync[q]);
        }
        // a warp holding a row that wants the tile already knows the outcome ("keep") and moves on;
        // only warps whose rows all vote "skip" have to hear from the others. Every warp still
        // arrives once per tile, and none can reach the next tile's vote before all have arrived
        // here (the next S tile is only issued after all have voted).
        if (!want) {
          ok = mbar_wait(&bars->wg_sync[q], par, abort_flag);
          if (!ok) break;
          int v = 0;
#pragma unroll
          for (int w = 0; w < RO::GW; ++w) v |= bars->vote_any[q][par][w];
          // max over rows ignores NaN rows; a tile is skipped iff that max is < 0
          skip = !(v & 1) && (v & 2);
        }
      }
      auto mark_tile = [&](int what) {
        if (KIND != KIND_DENSE && half == 0 && wq == 0 && lane == 0 && p.tile_map)
          p.tile_map[((((long long)si.b * p.hgrid + si.head) * p.num_m_blocks + mb) * p.num_splits + si.split) * p.n_tiles_k + n] = what;
      };
      if (skip) {
        mark_tile(2);
        continue;
      }

      // ---- move the reference maximum only when it lags by more than 2^8 -------------------------
      float m_cand = fmaxf(m_cur, m_ref);
      if (mode != FSA_MASK_NONE) m_cand = fmaxf(m_cand, -1e6f);
      // A share of the keys may begin with tiles that are not masked (whole sequences begin with the diagonal) and where every score of a
      // row is -inf. There is no maximum to refer to yet: the exponentials, all zero, are taken as they are. (Not a finite maximum instead:
      // it would outweigh scores below it in the tiles that follow.)
      const bool none = CL && m_cand == -INFINITY;
      const bool need = !none && !((m_cand - m_ref) * cc <= 8.0f);  // also true on the first tile (m_ref = -inf)
      float scale = 1.0f;
      if (need) {
        scale = ex2_approx((m_ref - m_cand) * cc);
        m_ref = m_cand;
        l_ref *= scale;
      }
      if constexpr (F8) {
        if (bscaled) {  // only for a tile that is kept: a skipped tile must not move the reference
          const float svn = vbs[n];
          if (svn > v_run) {  // the accumulator moves to the larger unit (nothing to move before the first P V)
            o_mul = v_run > 0.f ? __fdividef(v_run, svn) : 1.0f;
            v_run = svn;
          }
          p_mul = v_run > 0.f ? __fdividef(svn, v_run) : 0.0f;
        }
      }
      // s_full for this tile was committed after the previous P V of this group, so O is at rest
      if (have_o && (__any_sync(0xffffffffu, need) || o_mul != 1.0f)) {
        const float o_scale = scale * o_mul;
        // A rolled loop of as many columns as fit beside the row's scores: 32 (head size 256, scores of standard deviation 6, S = 4096:
        // 183.1 us with 16, which spill 272 bytes there, 173.7 with 32, 175.5 with 32 unrolled; head size 128: 77.4 and 76.0), at head
        // size 64 sixteen (dense causal S = 4096, 8 heads: 57.0 us, 59.2 with 32).
        constexpr int RC = HD == 64 ? 16 : 32;
#pragma unroll 1
        for (int ch = 0; ch < OC / RC; ++ch) {
          uint32_t r[RC];
          if constexpr (RC == 32)
            tmem_ld32(tO + ch * RC, r);
          else
            tmem_ld16(tO + ch * RC, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < RC; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * o_scale);
          if constexpr (RC == 32)
            tmem_st32(tO + ch * RC, r);
          else
            tmem_st16(tO + ch * RC, r);
        }
      }

      // ---- P = exp2(S*c - m*c), row sum, publish P (16-bit pairs) over the S columns -----------------
      const float2 c2 = make_float2(cc, cc);
      const float neg_mc = none ? 0.f : -(m_ref * cc);
      const float2 nm2 = make_float2(neg_mc, neg_mc);
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      constexpr int EXP_UNROLL = GATED ? 1 : NC / 32;
#pragma unroll EXP_UNROLL
      for (int ch = 0; ch < NC / 32; ++ch) {
        uint32_t pk[16];
        if constexpr (GATED) {
          tmem_ld32(tS + ch * 32, sr);
          tmem_ld_wait();
        }
        const uint32_t* src = GATED ? sr : &sr[ch * 32];
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float2 ta = fma2(make_float2(__uint_as_float(src[i]), __uint_as_float(src[i + 1])), c2, nm2);
          const float2 tb = fma2(make_float2(__uint_as_float(src[i + 2]), __uint_as_float(src[i + 3])), c2, nm2);
          float2 ea, eb;
          ea.x = ex2_approx(ta.x);
          ea.y = ex2_approx(ta.y);
          eb.x = ex2_approx(tb.x);
          eb.y = ex2_approx(tb.y);
          sum2[0] = add2(sum2[0], ea);
          sum2[1] = add2(sum2[1], eb);
          if constexpr (F8) {
            pk[i >> 2] = bscaled ? pack4_fp8<T>(ea.x * p_mul, ea.y * p_mul, eb.x * p_mul, eb.y * p_mul)
                                 : pack4_fp8<T>(ea.x, ea.y, eb.x, eb.y);
          } else {
            pk[i >> 1] = pack2<T>(ea.x, ea.y);
            pk[(i >> 1) + 1] = pack2<T>(eb.x, eb.y);
          }
        }
        if constexpr (F8)
          tmem_st8(tS + ch * 8, pk);
        else
          tmem_st16(tS + ch * 16, pk);
        if (HALVES && ch == 1) {
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->p_full[q]);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(HALVES ? &bars->p_rest[q] : &bars->p_full[q]);
      l_ref += (sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y);
      mark_tile(1);  // not in front of the exponentials
      if (KIND != KIND_DENSE && RO::HALVES == 1) lg_l = lg2_approx(l_ref);  // two halves: when the other's sum is known
      have_o = true;
    }

    // ---- epilogue (flash_sparse_attn/ops/triton/activations.py:169-203) ---------------------------
    if (ok && have_o) {
      ok = mbar_wait(&bars->o_final[q], 0, abort_flag);
      tc_fence_after();
      if constexpr (RO::HALVES == 2) {  // the row's sum; the last tile's exchange has been read (all votes came before o_final)
        float2* xch = reinterpret_cast<float2*>(smem + SM::kXch) + q * 256;
        xch[half * 128 + row].y = l_ref;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->pair_sync[q][wq]);
        ok = ok && mbar_wait(&bars->pair_sync[q][wq], cnt_s & 1, abort_flag);
        const float other = xch[(half ^ 1) * 128 + row].y;
        l_ref += other;
      }
    }
    if constexpr (CL) {
      // ---- merge: this CTA's rows go to its shared memory, over the K and V ring (all MMAs that read it are done), 16-byte pieces
      // swizzled by the row; then every CTA finishes 256 / cluster of the rows from the shared memory of all. A remote read takes
      // as long as a step's MMAs, so sixteen are under way at a time. (Pushing the rows to their owner, a row a thread: 32 packets of 16
      // bytes a store, S = 1024 at head size 64 16.6 us against 14.3.)
#pragma unroll
      for (int g = 0; g < 2; ++g)
        if (ok && !fsa_fwd_sched_empty(sched[g])) ok = mbar_wait(&bars->o_final[g], 0, abort_flag);
      tc_fence_after();
      float4* const own = reinterpret_cast<float4*>(smem + SM::kK);        // [256 rows][HD / 4]
      float2* const own_ml = reinterpret_cast<float2*>(smem + SM::kXch);   // [256]
      float2* const all_ml = own_ml + 256;                                 // [CTA][row of this CTA's share]
      float* const weight = &bars->dl[0][0];                               // likewise
#pragma unroll
      for (int ch = 0; ch < HD / 32; ++ch) {
        uint32_t r[32];
        if (ok && have_o) {
          tmem_ld32(tO + ch * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          own[(q * TM + row) * (HD / 4) + ((ch * 8 + i) ^ (row & 7))] =
              make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                          __uint_as_float(r[4 * i + 3]));
      }
      own_ml[q * TM + row] = make_float2(m_ref, l_ref);
      cluster_sync();
      const int rows = QT * TM / p.cluster;  // of this CTA's share, a power of two
      // the place of row r of the share in the results, or -1
      auto place = [&](int r, int* head, long long* tok) {
        const int at = share * rows + r, mb_r = pair * QT + at / TM, offs = mb_r * TM + at % TM, qi = offs / gpack;
        *head = (p.flags & F_PACK_GQA) ? si.hkv * p.G + (offs - qi * gpack) : si.head;
        *tok = qi;
        return mb_r < m_blocks_here && qi < si.sq && !*abort_flag;
      };
      const long long b_at = (p.flags & F_VARLEN_Q) ? 0 : si.b;
      int head;
      long long tok;
      {  // weights: a thread for every (CTA, row)
        const int r = tid & (rows - 1), from = tid / rows;
        const float2 e = peer(own_ml, from)[share * rows + r];
        all_ml[tid] = e;
        named_bar_sync(1, 256);
        float m_tot = -INFINITY, l_tot = 0.f;
        for (int i = 0; i < p.cluster; ++i) m_tot = fmaxf(m_tot, all_ml[i * rows + r].x);
        for (int i = 0; i < p.cluster; ++i) {
          const float2 x = all_ml[i * rows + r];
          if (x.y != 0.f) l_tot = fmaf(x.y, ex2_approx((x.x - m_tot) * cc), l_tot);
        }
        const bool dead = (l_tot == 0.0f) || (l_tot != l_tot);
        weight[tid] = e.y != 0.f ? ex2_approx((e.x - m_tot) * cc) * (dead ? 1.0f : v_scale / l_tot) : 0.f;
        if (from == 0 && place(r, &head, &tok))
          p.lse[b_at * p.l_sb + (long long)head * p.l_sh + ((p.flags & F_VARLEN_Q) ? si.off_q + tok : tok)] =
              dead ? -INFINITY : (m_tot * cc + log2f(l_tot)) * 0.6931471805599453f;
        named_bar_sync(1, 256);
      }
      auto merge = [&](auto size) {
        constexpr int C = decltype(size)::value, KB = 16 / C, ITEMS = (HD / 4) / C;  // 16-byte pieces of a thread: at a time, in all
        static_assert(ITEMS % KB == 0, "whole batches");
        const int d4 = tid % (HD / 4), r0 = tid / (HD / 4);
        constexpr int RSTEP = 256 / (HD / 4);  // rows that the threads cover together
#pragma unroll 1
        for (int k0 = 0; k0 < ITEMS; k0 += KB) {
          float4 v[C][KB];
#pragma unroll
          for (int i = 0; i < C; ++i) {
            const float4* src = peer(own, i) + share * rows * (HD / 4);
#pragma unroll
            for (int k = 0; k < KB; ++k) {
              const int r = r0 + (k0 + k) * RSTEP;
              v[i][k] = src[r * (HD / 4) + (d4 ^ (r & 7))];
            }
          }
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            const int r = r0 + (k0 + k) * RSTEP;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < C; ++i) {
              const float w = weight[i * rows + r];
              if (w != 0.f) {
                acc.x = fmaf(v[i][k].x, w, acc.x);
                acc.y = fmaf(v[i][k].y, w, acc.y);
                acc.z = fmaf(v[i][k].z, w, acc.z);
                acc.w = fmaf(v[i][k].w, w, acc.w);
              }
            }
            if (place(r, &head, &tok) && d4 * 4 < p.D)
              *reinterpret_cast<uint2*>(reinterpret_cast<TO*>(p.out) + b_at * p.o_sb + (si.off_q + tok) * p.o_sm +
                                        (long long)head * p.o_sh + d4 * 4) = make_uint2(pack2<TO>(acc.x, acc.y), pack2<TO>(acc.z, acc.w));
          }
        }
      };
      if (p.cluster == 2)
        merge(std::integral_constant<int, 2>());
      else if (p.cluster == 4)
        merge(std::integral_constant<int, 4>());
      else
        merge(std::integral_constant<int, 8>());
      cluster_sync();  // nobody leaves while another CTA may still read its shared memory
    } else if (ok && q_valid[q]) {
      const bool dead = (l_ref == 0.0f) || (l_ref != l_ref);
      const float inv = dead ? 1.0f : (bscaled ? v_run : v_scale) / l_ref;
      float lse = dead ? -INFINITY : m_ref * cc + log2f(l_ref);
      if (!(p.flags & F_LSE_LOG2)) lse *= 0.6931471805599453f;
      const long long tok = si.off_q + q_idx;
      if (rm.row_ok && half == 0)
        p.lse[(long long)((p.flags & F_VARLEN_Q) ? 0 : si.b) * p.l_sb + (long long)q_head * p.l_sh +
              (long long)si.split * p.l_ss + ((p.flags & F_VARLEN_Q) ? tok : q_idx)] = lse;
      const long long obase = (long long)((p.flags & F_VARLEN_Q) ? 0 : si.b) * p.o_sb + tok * p.o_sm +
                              (long long)q_head * p.o_sh + (long long)si.split * p.o_ss + half * OC;
#pragma unroll
      for (int ch = 0; ch < OC / 32; ++ch) {
        uint32_t r[32];
        if (have_o) {
          tmem_ld32(tO + ch * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (rm.row_ok) {
          if (p.flags & F_SPLIT) {
            float* dst = reinterpret_cast<float*>(p.out) + obase + ch * 32;
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              if (half * OC + ch * 32 + i < p.D)
                *reinterpret_cast<float4*>(dst + i) =
                    make_float4(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv,
                                __uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
          } else {
            TO* dst = reinterpret_cast<TO*>(p.out) + obase + ch * 32;
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 v;
              v.x = pack2<TO>(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
              v.y = pack2<TO>(__uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
              v.z = pack2<TO>(__uint_as_float(r[i + 4]) * inv, __uint_as_float(r[i + 5]) * inv);
              v.w = pack2<TO>(__uint_as_float(r[i + 6]) * inv, __uint_as_float(r[i + 7]) * inv);
              if (half * OC + ch * 32 + i < p.D) *reinterpret_cast<uint4*>(dst + i) = v;
            }
          }
        }
      }
    }
  }

  // ---- teardown ------------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag) atomicExch(p.status, 1);
  if (warp == RO::W_PROD) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Calls whose key tiles may be shared inside clusters (fsa_fwd_cluster_size): whole sequences of equal query and key length. Not the
// other kinds: whether a tile is skipped depends on the tiles before it. Windows have few tiles. Not calls with lengths of their own,
// pages or keys in front of the queries: unsplit, those give a sequence the same bits alone as in a batch, at every size.
// `known`: the runtime's answers, per device and for one kernel: resident clusters plus one, 0: not asked yet.
template <typename Kernel>
int fwd_cluster_size(Kernel kern, const FwdKernelParams& p, int threads, int smem, std::atomic<int> (*known)[FSA_FWD_MAX_CLUSTER + 1]) {
  int dev = 0;
  if ((p.flags & (F_SPLIT | F_LOCAL | F_VARLEN_Q | F_VARLEN_K | F_USED_Q | F_USED_K | F_PAGED)) || p.sq != p.sk || p.tile_map || cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 1;
  return fsa_fwd_cluster_size((long long)p.num_pairs * p.hgrid * p.B, p.n_tiles_k, device_sm_count(), [&](int size) {
    int room = known[dev][size].load(std::memory_order_relaxed) - 1;
    if (room < 0) {
      room = resident_clusters(kern, size, threads, smem);
      known[dev][size].store(room + 1, std::memory_order_relaxed);
    }
    return room;
  });
}

template <int HD, typename T, int KIND, bool BSCALE = false, bool CL = false>
cudaError_t launch_one(FwdKernelParams& p, cudaStream_t stream) {
  auto kern = fwd_kernel<HD, T, KIND, BSCALE, CL>;
  constexpr int smem = FwdSmem<HD, sizeof(T), KIND, CL>::kTotal, threads = FwdRoles<HD, KIND>::NTHREADS;
  static std::atomic<unsigned long long> opted_in{0};  // one bit per device: the attribute is per device
  if (cudaError_t e = smem_opt_in(kern, smem, opted_in); e != cudaSuccess) return e;
  const long long grid = (long long)p.num_pairs * p.hgrid * p.B * p.num_splits;
  if (grid <= 0) return cudaSuccess;
  if constexpr (CL) {
    static std::atomic<int> known[64][FSA_FWD_MAX_CLUSTER + 1];
    p.cluster = fwd_cluster_size(kern, p, threads, smem, known);
    if (p.cluster == 1) return launch_one<HD, T, KIND>(p, stream);
    return launch_early(kern, (unsigned)grid * p.cluster, threads, smem, stream, p.cluster, p);
  }
  // Set up while the kernel in front still runs, except one round of equally long CTAs on more than half of the SMs: behind a call that leaves
  // the other half free, more of them come to share a pair of SMs than when all are spread at once. Full attention, 8 heads of 128, 96 CTAs:
  // S = 3000 56.8 us early, 55.4 not, over 6000 keys 101.1 and 98.3, sparse 105.3 and 101.8. Short calls (700 tokens, 32 heads 21.6 and 21.7), head
  // size 64 (5000 tokens, 4 heads 75.4 and 76.7) and the gated kind gain as much as they lose.
  const bool even = KIND != KIND_GATED && HD > 64 && !(p.flags & (F_CAUSAL | F_LOCAL | F_VARLEN_Q | F_VARLEN_K | F_USED_Q | F_USED_K));
  const int sms = device_sm_count();
  return launch_early_if(!(even && 2 * grid > sms && grid <= sms && p.n_tiles_k >= 12), kern, (unsigned)grid, threads, smem, stream, 1, p);
}

}  // namespace

// kind: KIND_*, dtype: DT_BF16 / DT_FP16, head_dim: 64 or 128. Returns cudaErrorInvalidValue for
// unsupported combinations.

cudaError_t launch_fwd(FwdKernelParams& p, int kind, int dtype, int head_dim, cudaStream_t stream) {
  if (p.k_bscale) {  // block-scaled FP8: dense and sparse kinds at head_dim 128
    if (head_dim != 128 || kind == KIND_GATED) return cudaErrorInvalidValue;
    if (dtype == DT_E4M3)
      return kind == KIND_DENSE ? launch_one<128, __nv_fp8_e4m3, KIND_DENSE, true>(p, stream)
                                : launch_one<128, __nv_fp8_e4m3, KIND_SPARSE, true>(p, stream);
    if (dtype == DT_E5M2)
      return kind == KIND_DENSE ? launch_one<128, __nv_fp8_e5m2, KIND_DENSE, true>(p, stream)
                                : launch_one<128, __nv_fp8_e5m2, KIND_SPARSE, true>(p, stream);
    return cudaErrorInvalidValue;
  }
#define FSA_FWD_CASE(HD_, T_, DT_)                                                  \
  if (head_dim == HD_ && dtype == DT_) {                                            \
    if (kind == KIND_DENSE)                                                         \
      return launch_one<HD_, T_, KIND_DENSE, false, (HD_ <= 128 && sizeof(T_) == 2)>(p, stream); \
    if (kind == KIND_SPARSE) return launch_one<HD_, T_, KIND_SPARSE>(p, stream);    \
    if (kind == KIND_GATED) return launch_one<HD_, T_, KIND_GATED>(p, stream);      \
  }
  FSA_FWD_CASE(128, __nv_bfloat16, DT_BF16)
  FSA_FWD_CASE(128, __half, DT_FP16)
  FSA_FWD_CASE(64, __nv_bfloat16, DT_BF16)
  FSA_FWD_CASE(64, __half, DT_FP16)
  FSA_FWD_CASE(192, __nv_bfloat16, DT_BF16)
  FSA_FWD_CASE(192, __half, DT_FP16)
  FSA_FWD_CASE(256, __nv_bfloat16, DT_BF16)
  FSA_FWD_CASE(256, __half, DT_FP16)
  FSA_FWD_CASE(128, __nv_fp8_e4m3, DT_E4M3)
  FSA_FWD_CASE(128, __nv_fp8_e5m2, DT_E5M2)
#undef FSA_FWD_CASE
  return cudaErrorInvalidValue;
}

}  // namespace fsa
