// Top-k position selection for the decode path: per row of scores the k largest entries, returned as
// ascending positions - what `gather_kv_indices` of the decode operators expects. Restates
// flash_sparse_attn/utils/mask.py:20-44 (torch.topk(..., sorted=False) followed by a sort of the indices)
// as one kernel without a sort: a radix select (8 bits per pass) finds the k-th largest key exactly, then one
// ordered compaction pass writes the selected positions in index order. Among equal scores at the
// threshold the lowest positions win (torch leaves that choice unspecified). NaN orders above +inf, as
// in torch.topk. Integer work on L2-resident rows: a cluster of 1 to 8 CTAs of 1024 threads per row (as many as
// keep the grid within the SM count), three (16-bit scores) or five (fp32) passes over the row with 16-byte loads,
// plus a counting pass when the row is shared.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fsa_b200.h"
#include "fsa_params.h"

namespace fsa {

namespace {

constexpr int TK_THREADS = 1024;
constexpr int TK_V = 8;  // consecutive entries per thread and step (one or two 16-byte loads)

// Monotone map to an unsigned key: larger value, larger key (-0 < +0 is harmless for a selection). 16-bit
// inputs keep 16-bit keys (two radix passes instead of four).
template <typename T>
struct KeyOf {
  static constexpr int kBits = 16;
  __device__ static uint32_t key(T v) {
    const uint32_t b = *reinterpret_cast<const unsigned short*>(&v);
    return (b & 0x8000u) ? (~b & 0xffffu) : (b | 0x8000u);
  }
};
template <>
struct KeyOf<float> {
  static constexpr int kBits = 32;
  __device__ static uint32_t key(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  }
};

// Keys of entries [i0, i0 + TK_V) of a row; entries past n get `fill`.
template <typename T>
__device__ __forceinline__ void load_keys(const T* row, bool vec_ok, int i0, int n, uint32_t fill, uint32_t* keys) {
  if (vec_ok && i0 + TK_V <= n) {
    constexpr int NV = TK_V * sizeof(T) / 16;
    uint4 raw[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) raw[v] = __ldg(reinterpret_cast<const uint4*>(row + i0) + v);
    const T* e = reinterpret_cast<const T*>(raw);
#pragma unroll
    for (int j = 0; j < TK_V; ++j) keys[j] = KeyOf<T>::key(e[j]);
  } else {
#pragma unroll
    for (int j = 0; j < TK_V; ++j) keys[j] = (i0 + j < n) ? KeyOf<T>::key(row[i0 + j]) : fill;
  }
}

// Inclusive scan of `v` over the block; returns the inclusive prefix of this thread and the block total.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
    if (lane >= s) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_tot[lane];  // TK_THREADS / 32 == 32 warps
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, s);
      if (lane >= s) w += y;
    }
    warp_tot[lane] = w;  // inclusive totals of the warps
  }
  __syncthreads();
  const uint32_t before = warp == 0 ? 0u : warp_tot[warp - 1];
  *total = warp_tot[TK_THREADS / 32 - 1];
  __syncthreads();  // warp_tot is reused by the next call
  return x + before;
}

constexpr int TK_COPIES = 8;  // copies of the histogram: the lanes of a warp spread over them (see below)
constexpr int TK_PITCH = 257;  // a bin's copies lie in different banks

// One thread-block cluster per row: CTA `rank` of `csize` owns the slice [rank * chunk, (rank + 1) * chunk) of the
// row. The histograms of a radix pass are summed over the cluster through distributed shared memory (every CTA
// reads all of them and finds the bin itself, so all agree without a broadcast); for the compaction every CTA
// takes the counts of the slices before it as its base. With 64 rows one CTA per row would leave more than half of
// a B200's 148 SMs idle.
// What bounds it is the chain of dependent steps of a pass, not the bytes: so the bin is found by a scan over the 256
// bins in parallel, a pass costs one cluster barrier (two sets of sums alternate), lanes spread over eight copies of
// the histogram because scores share their leading bits (a warp's 32 updates would queue on two or three bins), and
// with NC > 0 a thread keeps its 8 * NC consecutive entries in registers for all passes (NC = 0 reads the slice again in
// every pass).
template <typename T, typename I, int NC>
__global__ void __launch_bounds__(TK_THREADS) topk_kernel(const T* __restrict__ scores, long long row_stride, int n, int k,
                                                          I* __restrict__ out, int csize, int chunk) {
  static_assert(TK_THREADS == 1024, "block_scan assumes 32 warps");
  after_previous();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ uint32_t copies[TK_COPIES * TK_PITCH];
  __shared__ uint32_t hist[2][256];
  __shared__ uint32_t warp_tot[TK_THREADS / 32];
  __shared__ uint32_t sel_prefix, sel_remaining;
  __shared__ uint32_t slice_cnt[2];  // greater / equal entries of this CTA's slice
  const int rank = (int)cluster.block_rank();
  const int row_idx = blockIdx.x / csize;
  const T* row = scores + (long long)row_idx * row_stride;
  I* dst = out + (long long)row_idx * k;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool vec_ok = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  constexpr int PASSES = KeyOf<T>::kBits / 8;
  constexpr int STEP = TK_THREADS * TK_V;
  const int lo = rank * chunk < n ? rank * chunk : n;
  const int hi = lo + chunk < n ? lo + chunk : n;  // this CTA's slice [lo, hi); chunk is a multiple of TK_V
  const int mine = lo + tid * (NC * TK_V);         // NC > 0: this thread's first entry
  uint32_t kc[NC > 0 ? NC * TK_V : 1];
  if constexpr (NC > 0) {
#pragma unroll
    for (int c = 0; c < NC; ++c) load_keys(row, vec_ok, mine + c * TK_V, hi, 0u, kc + c * TK_V);
  }
  for (int i = tid; i < TK_COPIES * TK_PITCH; i += TK_THREADS) copies[i] = 0;
  __syncthreads();

  // ---- radix select: after pass d the top 8(d+1) bits of the k-th largest key are known ----------------
  uint32_t prefix = 0, remaining = (uint32_t)k;  // keys above the prefix range so far: k - remaining
  for (int pass = 0; pass < PASSES; ++pass) {
    const int shift = KeyOf<T>::kBits - 8 - 8 * pass;
    const uint32_t mask_hi = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    uint32_t* my_copy = copies + (lane & (TK_COPIES - 1)) * TK_PITCH;
    auto count = [&](uint32_t key) {
      if ((key & mask_hi) == prefix) atomicAdd(my_copy + ((key >> shift) & 255u), 1u);
    };
    if constexpr (NC > 0) {
#pragma unroll
      for (int j = 0; j < NC * TK_V; ++j)
        if (mine + j < hi) count(kc[j]);
    } else {
      for (int start = lo; start < hi; start += STEP) {
        const int i0 = start + tid * TK_V;
        if (i0 < hi) {
          uint32_t keys[TK_V];
          load_keys(row, vec_ok, i0, hi, 0u, keys);
#pragma unroll
          for (int j = 0; j < TK_V; ++j)
            if (i0 + j < hi) count(keys[j]);
        }
      }
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t sum = 0;
#pragma unroll
      for (int r = 0; r < TK_COPIES; ++r) {
        sum += copies[r * TK_PITCH + tid];
        copies[r * TK_PITCH + tid] = 0;  // for the next pass
      }
      hist[pass & 1][tid] = sum;
    }
    cluster.sync();  // every CTA's sums are there, and everybody has read those of the pass before
    if (tid < 256) {
      // thread t takes bin 255 - t: the first bin from the top at which `remaining` keys are covered
      const int bin = 255 - tid;
      uint32_t v = 0;
#pragma unroll
      for (int r = 0; r < 8; ++r)  // unrolled: the remote reads are in flight together
        if (r < csize) v += *cluster.map_shared_rank(&hist[pass & 1][bin], r);
      uint32_t x = v;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += y;
      }
      if (lane == 31) warp_tot[tid >> 5] = x;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      for (int w = 0; w < (tid >> 5); ++w) x += warp_tot[w];
      if (x >= remaining && x - v < remaining) {
        sel_prefix = prefix | ((uint32_t)bin << shift);
        sel_remaining = remaining - (x - v);  // how many keys of this bin (with this prefix) are still needed
      }
    }
    __syncthreads();
    prefix = sel_prefix;
    remaining = sel_remaining;
  }
  const uint32_t thr = prefix;         // key of the k-th largest entry
  const uint32_t need_eq = remaining;  // entries equal to it that belong to the selection (lowest positions)

  if constexpr (NC > 0) {
    // ---- one scan over the slice; positions come out ascending ------------------------------------------
    // (greater in the low half, equal in the high half: a slice has at most 1024 * 8 * NC <= 32768 entries)
    uint32_t cnt = 0, total;
#pragma unroll
    for (int j = 0; j < NC * TK_V; ++j)
      if (mine + j < hi) cnt += (kc[j] > thr ? 1u : 0u) | (kc[j] == thr ? 0x10000u : 0u);
    const uint32_t inc = block_scan(cnt, warp_tot, &total);
    uint32_t gt_before = (inc & 0xffffu) - (cnt & 0xffffu), eq_before = (inc >> 16) - (cnt >> 16);
    if (csize > 1) {
      if (tid == 0) slice_cnt[0] = total;
      cluster.sync();
#pragma unroll
      for (int r = 0; r < 7; ++r) {
        const uint32_t t = r < rank ? *cluster.map_shared_rank(&slice_cnt[0], r) : 0u;
        gt_before += t & 0xffffu;
        eq_before += t >> 16;
      }
    }
    if (cnt != 0u) {
#pragma unroll
      for (int j = 0; j < NC * TK_V; ++j) {
        if (mine + j < hi) {
          const bool gt = kc[j] > thr, eq = kc[j] == thr;
          if (gt || (eq && eq_before < need_eq))
            dst[gt_before + (eq_before < need_eq ? eq_before : need_eq)] = (I)(mine + j);
          gt_before += gt ? 1u : 0u;
          eq_before += eq ? 1u : 0u;
        }
      }
    }
    cluster.sync();  // nobody leaves while another CTA may still read its shared memory
    return;
  }

  // ---- counts of this slice, bases from the slices before it ------------------------------------------
  uint32_t base_gt = 0, base_eq = 0;  // greater / equal entries before the current step of this CTA
  if (csize > 1) {
    uint32_t c_gt = 0, c_eq = 0;
    for (int start = lo; start < hi; start += STEP) {
      const int i0 = start + tid * TK_V;
      if (i0 < hi) {
        uint32_t keys[TK_V];
        load_keys(row, vec_ok, i0, hi, 0u, keys);
#pragma unroll
        for (int j = 0; j < TK_V; ++j)
          if (i0 + j < hi) {
            c_gt += keys[j] > thr ? 1u : 0u;
            c_eq += keys[j] == thr ? 1u : 0u;
          }
      }
    }
    uint32_t tot;
    block_scan(c_gt, warp_tot, &tot);
    if (tid == 0) slice_cnt[0] = tot;
    block_scan(c_eq, warp_tot, &tot);
    if (tid == 0) slice_cnt[1] = tot;
    cluster.sync();
    for (int r = 0; r < rank; ++r) {
      base_gt += *cluster.map_shared_rank(&slice_cnt[0], r);
      base_eq += *cluster.map_shared_rank(&slice_cnt[1], r);
    }
  }

  // ---- ordered compaction: every thread owns TK_V consecutive entries, positions come out ascending ----------
  for (int start = lo; start < hi; start += STEP) {
    const int i0 = start + tid * TK_V;
    uint32_t keys[TK_V];
    uint32_t cnt = 0;  // greater in the low half, equal in the high half (a step has <= 8192 entries)
    if (i0 < hi) {
      load_keys(row, vec_ok, i0, hi, 0u, keys);
#pragma unroll
      for (int j = 0; j < TK_V; ++j)
        if (i0 + j < hi) cnt += (keys[j] > thr ? 1u : 0u) | (keys[j] == thr ? 0x10000u : 0u);
    }
    uint32_t total;
    const uint32_t inc = block_scan(cnt, warp_tot, &total);
    uint32_t gt_before = base_gt + (inc & 0xffffu) - (cnt & 0xffffu);
    uint32_t eq_before = base_eq + (inc >> 16) - (cnt >> 16);
    if (i0 < hi && cnt != 0u) {
#pragma unroll
      for (int j = 0; j < TK_V; ++j) {
        if (i0 + j >= hi) break;
        const bool gt = keys[j] > thr, eq = keys[j] == thr;
        if (gt || (eq && eq_before < need_eq)) dst[gt_before + (eq_before < need_eq ? eq_before : need_eq)] = (I)(i0 + j);
        gt_before += gt ? 1u : 0u;
        eq_before += eq ? 1u : 0u;
      }
    }
    base_gt += total & 0xffffu;
    base_eq += total >> 16;
  }
  cluster.sync();  // nobody leaves while another CTA may still read its shared memory
}

// Entries of a row that a CTA of a cluster of c takes.
inline int topk_chunk(int n, int c) { return ((n + c - 1) / c + TK_V - 1) / TK_V * TK_V; }

// Shared memory that keeps a second CTA off the SM: more than half of what it has. Clusters are launched with it: set up while a call in
// front of them still runs, they would double up on the SMs that it leaves free (32 rows of 131 072 bf16 scores over and over, clusters
// of four: 31.8 us, with an SM to each CTA 25.8, launched behind one another 26.2).
constexpr int LONE_SMEM = 120 * 1024;

// Clusters of c CTAs that the device holds with one CTA per SM, asked once per device.
template <typename Kernel>
int topk_room(Kernel kern, int c, std::atomic<int>& known) {
  int fit = known.load(std::memory_order_relaxed) - 1;
  if (fit < 0) {
    fit = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LONE_SMEM) == cudaSuccess)
      fit = resident_clusters(kern, c, TK_THREADS, LONE_SMEM);
    else
      (void)cudaGetLastError();
    known.store(fit + 1, std::memory_order_relaxed);
  }
  return fit;
}

// Cluster size: the smallest power of two up to 8 that brings a slice down to what TK_V entries a thread hold, or the
// largest below that whose clusters all find room at a time with an SM to each CTA. Smaller slices gain less than the exchange costs
// (one row of 8000 fp32 scores: two CTAs 10.9 us, one 9.5; 32 of 16 000 bf16: four 10.8, two 9.1).
// rows * size <= SMs does not say that: 16 clusters of eight have no room on 148 SMs (16 rows of 32000 fp32 scores: 25.9 us
// with them, 13.1 with clusters of four; bf16, whose CTAs share SMs then, 13.9 and 10.2).
template <typename T, typename I>
int topk_cluster_size(int rows, int n) {
  static std::atomic<int> room[64][3][4];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 1;
  for (int lg = 3; lg > 0; --lg) {
    const int c = 1 << lg, chunk = topk_chunk(n, c);
    if ((long long)rows * c > device_sm_count() || n <= TK_THREADS * TK_V * (c / 2)) continue;
    const int nc = chunk <= TK_THREADS * TK_V ? 1 : chunk <= TK_THREADS * TK_V * 2 ? 2 : 0;
    std::atomic<int>& known = room[dev][nc][lg];
    const int fit = nc == 1 ? topk_room(topk_kernel<T, I, 1>, c, known)
                            : nc == 2 ? topk_room(topk_kernel<T, I, 2>, c, known) : topk_room(topk_kernel<T, I, 0>, c, known);
    if (rows <= fit) return c;
  }
  return 1;
}

template <typename T, typename I>
cudaError_t launch_topk_t(const void* scores, long long row_stride, int rows, int n, int k, void* out, cudaStream_t stream) {
  const int csize = topk_cluster_size<T, I>(rows, n), chunk = topk_chunk(n, csize);
  const T* x = reinterpret_cast<const T*>(scores);
  I* o = reinterpret_cast<I*>(out);
  const int smem = csize > 1 ? LONE_SMEM : 0;  // topk_room has asked for it
  const auto launch = [&](void (*kern)(const T*, long long, int, int, I*, int, int)) {
    return launch_early(kern, (unsigned)(rows * csize), TK_THREADS, smem, stream, csize, x, row_stride, n, k, o, csize, chunk);
  };
  // slices of up to 8192 / 16384 entries stay in registers
  if (chunk <= TK_THREADS * TK_V) return launch(topk_kernel<T, I, 1>);
  if (chunk <= TK_THREADS * TK_V * 2) return launch(topk_kernel<T, I, 2>);
  return launch(topk_kernel<T, I, 0>);
}

template <typename T>
cudaError_t launch_topk(const void* scores, long long row_stride, int rows, int n, int k, void* out, int out64,
                        cudaStream_t stream) {
  if (out64) return launch_topk_t<T, long long>(scores, row_stride, rows, n, k, out, stream);
  return launch_topk_t<T, int>(scores, row_stride, rows, n, k, out, stream);
}

}  // namespace

}  // namespace fsa

extern "C" int fsa_topk_indices(const void* scores, int dtype, int rows, int n, int64_t row_stride, int k, void* out,
                                int out_is_int64, void* stream_) {
  if (!scores || !out || rows < 0 || n <= 0 || k <= 0 || k > n || row_stride < n) return FSA_ERR_INVALID_ARG;
  if (rows == 0) return FSA_OK;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  cudaError_t e;
  switch (dtype) {
    case FSA_DT_BF16:
      e = fsa::launch_topk<__nv_bfloat16>(scores, row_stride, rows, n, k, out, out_is_int64, stream);
      break;
    case FSA_DT_FP16:
      e = fsa::launch_topk<__half>(scores, row_stride, rows, n, k, out, out_is_int64, stream);
      break;
    case FSA_DT_F32:
      e = fsa::launch_topk<float>(scores, row_stride, rows, n, k, out, out_is_int64, stream);
      break;
    default:
      return FSA_ERR_UNSUPPORTED;
  }
  return e == cudaSuccess ? FSA_OK : FSA_ERR_LAUNCH;
}
