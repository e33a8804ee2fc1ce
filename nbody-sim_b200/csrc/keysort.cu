// keysort.cu -- Morton keys and their sort in one launch, for disks of up to
// 65,536 bodies.
//
// At these sizes the key kernel, the clears and the four one-sweep passes of
// sort.cu are latency: 37 us at N = 4096 and 42 us at N = 30011, whatever the
// work.  Here one thread-block cluster holds every (key, index) pair: a block
// owns kThreads x kI consecutive places, in registers while a pass ranks them
// and in its shared memory between passes, and three passes of ten bits sort
// the 30-bit keys.  A pass
//   1. ranks the keys of each warp by digit and turns the warps' counts into
//      prefixes within the block;
//   2. sends the block's 1024 counts to every block of the cluster and meets
//      the others at a cluster barrier: each now has all counts, and with
//      them the place of every digit (the first pass waits before it sends
//      until every block of the cluster has started: until then its shared
//      memory may not be touched);
//   3. scatters its pairs into the blocks that own their places (distributed
//      shared memory; the last pass writes to global memory).
// The order is that of the one-sweep sort (stable, ties by index).
// Sort phase at N = 4096 / 30011 (in the step's graph): 18 / 27 us; a pass
// takes 3 to 4 us, in cluster barriers (0.6 to 1.2 us each, two a pass),
// ranking and the prefixes.  With eight keys a thread (N = 131072) the
// scatter and the ranking in 16 blocks take 52 us against the one-sweep
// sort's 45, so the rule stops at four.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "geom.cuh"
#include "kernels.cuh"

namespace nb {
namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kDigitBits = 10;
constexpr int kDigits = 1 << kDigitBits;
constexpr int kPasses = 3;
constexpr int kMaxBlocks = 16;  // of a cluster (above 8 needs the device's consent)
static_assert(kDigits == kThreads, "one thread per digit");
static_assert(kPasses * kDigitBits == 30, "whole Morton keys");

// Block exclusive scan of one value per thread; s_w: kWarps words.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t inc = warp_incl_scan(v, lane);
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  const uint32_t t = s_w[lane];
  const uint32_t ti = warp_incl_scan(t, lane);
  return inc - v + __shfl_sync(kFull, ti - t, warp);
}

template <int kI>
struct Smem {
  union {
    uint32_t cnt[kWarps][kDigits / 2];  // counts, then prefixes, of each warp's digits (two a word)
    uint2 stage[kThreads * kI];         // the block's pairs by digit, on their way out
  };
  uint32_t tot[kMaxBlocks][kDigits / 2];  // every block's counts
  uint32_t half[2][kDigits / 2];
  uint2 pair[kThreads * kI];  // (key, index) of the block's places
  uint32_t base[kDigits];     // where this block's first key of a digit goes
  uint32_t local[kDigits];    // and where it is staged
  uint32_t scan[kWarps];
  TreeGeom geom;
};

// Lanes whose low ten bits of v equal this lane's.  Ten ballots: one
// __match_any_sync takes some 250 cycles of a scheduler on random digits.
__device__ __forceinline__ unsigned digit_peers(uint32_t v) {
  unsigned peers = kFull;
#pragma unroll
  for (int b = 0; b < kDigitBits; ++b) {
    const bool on = (v >> b) & 1u;
    const unsigned m = __ballot_sync(kFull, on);
    peers &= on ? m : ~m;
  }
  return peers;
}

// kMake: makes the keys; else they are in `keys_in` (body order).
template <typename T, int kI, bool kMake>
__global__ void __launch_bounds__(kThreads)
k_sorted_keys(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ z,
              const uint32_t* __restrict__ keys_in, int n,
              const unsigned long long* __restrict__ enc, TreeGeom* __restrict__ geom_out,
              uint32_t* __restrict__ keys, uint32_t* __restrict__ perm,
              int* __restrict__ status) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char raw[];
  Smem<kI>& sm = *reinterpret_cast<Smem<kI>*>(raw);
  cg::cluster_group cl = cg::this_cluster();
  // Waited for before the first store into another block's shared memory; the
  // keys are made and ranked meanwhile.
  cl.barrier_arrive();
  const int blocks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  constexpr int kOwn = kThreads * kI;
  constexpr bool kStage = kI >= 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int w0 = warp * (32 * kI) + lane;  // the thread's places: w0 + 32 r
  uint32_t key[kI], idx[kI], at[kI];
  if constexpr (kMake) {
    T px[kI], py[kI], pz[kI];
#pragma unroll
    for (int r = 0; r < kI; ++r) {  // in flight while one thread makes the geometry
      const int i = min(rank * kOwn + w0 + 32 * r, n - 1);
      px[r] = x[i];
      py[r] = y[i];
      pz[r] = z[i];
    }
    if (tid == 0) {
      compute_geom(enc, sm.geom);
      if (rank == 0) *geom_out = sm.geom;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kI; ++r)
      key[r] = rank * kOwn + w0 + 32 * r < n
                   ? morton_key(sm.geom, (double)px[r], (double)py[r], (double)pz[r], status)
                   : 0x3fffffffu;
  } else {
#pragma unroll
    for (int r = 0; r < kI; ++r) {
      const int i = rank * kOwn + w0 + 32 * r;
      key[r] = i < n ? __ldg(keys_in + i) : 0x3fffffffu;
    }
  }
  // places past the last body sort behind every body: no key is larger, and
  // bodies of the largest key come first by their index
#pragma unroll
  for (int r = 0; r < kI; ++r) idx[r] = (uint32_t)(rank * kOwn + w0 + 32 * r);
  uint16_t* const mine = reinterpret_cast<uint16_t*>(&sm.cnt[warp][0]);
#pragma unroll 1
  for (int p = 0; p < kPasses; ++p) {
    const int shift = kDigitBits * p;
    uint4* clear = reinterpret_cast<uint4*>(&sm.cnt[0][0]);
#pragma unroll
    for (int i = 0; i < (int)sizeof(sm.cnt) / 16 / kThreads; ++i)
      clear[i * kThreads + tid] = make_uint4(0, 0, 0, 0);
    if (p > 0) {
#pragma unroll
      for (int r = 0; r < kI; ++r) {
        const uint2 q = sm.pair[w0 + 32 * r];
        key[r] = q.x;
        idx[r] = q.y;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kI; ++r) {
      const uint32_t d = (key[r] >> shift) & (kDigits - 1);
      const unsigned peers = digit_peers(d);
      const uint32_t old = mine[d];
      const uint32_t below = __popc(peers & lanemask_lt());
      __syncwarp();
      if (below == 0) mine[d] = (uint16_t)(old + __popc(peers));
      __syncwarp();
      at[r] = old + below;
    }
    __syncthreads();
    // Two digits a word and half of the warps a thread (a block's counts stay
    // below 2^16): prefixes over the warps, then the block's counts.
    {
      const int q = tid & (kDigits / 2 - 1), h = tid >> (kDigitBits - 1);
      constexpr int kRows = kWarps / 2;
      uint32_t c[kRows], sum = 0;
#pragma unroll
      for (int w = 0; w < kRows; ++w) c[w] = sm.cnt[h * kRows + w][q];
#pragma unroll
      for (int w = 0; w < kRows; ++w) {
        const uint32_t v = c[w];
        c[w] = sum;
        sum += v;
      }
      sm.half[h][q] = sum;
      __syncthreads();
      const uint32_t lo = sm.half[0][q], all = lo + sm.half[1][q], add = h ? lo : 0u;
#pragma unroll
      for (int w = 0; w < kRows; ++w) sm.cnt[h * kRows + w][q] = c[w] + add;
      if (p == 0) cl.barrier_wait();  // every block has started
      for (int b = h; b < blocks; b += 2)
        *cl.map_shared_rank(&sm.tot[rank][q], (unsigned)b) = all;
    }
    cl.sync();  // every block's counts are here, and its pairs in registers
    {
      // thread q < 512: digits 2 q and 2 q + 1
      uint32_t before[2] = {0, 0}, all[2] = {0, 0}, own = 0;
      if (tid < kDigits / 2) {
#pragma unroll 4
        for (int b = 0; b < blocks; ++b) {
          const uint32_t c = sm.tot[b][tid], lo = c & 0xffffu, hi = c >> 16;
          if (b < rank) { before[0] += lo; before[1] += hi; }
          if (b == rank) own = c;
          all[0] += lo;
          all[1] += hi;
        }
      }
      // both scans in one word: all of the cluster's keys (2^16), the block's (2^12)
      const uint32_t lo = own & 0xffffu, hi = own >> 16;
      const uint32_t ex = block_excl_scan(((all[0] + all[1]) << 14) | (lo + hi), sm.scan);
      if (tid < kDigits / 2) {
        const uint32_t g = ex >> 14, l = ex & 0x3fffu;
        sm.base[2 * tid] = g + before[0] - (kStage ? l : 0u);
        sm.base[2 * tid + 1] = g + all[0] + before[1] - (kStage ? l + lo : 0u);
        if (kStage) {
          sm.local[2 * tid] = l;
          sm.local[2 * tid + 1] = l + lo;
        }
      }
    }
    __syncthreads();
    if (kStage) {
#pragma unroll
      for (int r = 0; r < kI; ++r) {
        const uint32_t d = (key[r] >> shift) & (kDigits - 1);
        at[r] += sm.local[d] + mine[d];
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kI; ++r) sm.stage[at[r]] = make_uint2(key[r], idx[r]);
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kI; ++r) {
      uint2 q = make_uint2(key[r], idx[r]);
      uint32_t to;
      if (kStage) {  // runs of a digit's pairs go out together
        q = sm.stage[r * kThreads + tid];
        to = sm.base[(q.x >> shift) & (kDigits - 1)] + (uint32_t)(r * kThreads + tid);
      } else {
        const uint32_t d = (q.x >> shift) & (kDigits - 1);
        to = sm.base[d] + mine[d] + at[r];
      }
      if (p + 1 < kPasses) {
        *cl.map_shared_rank(&sm.pair[to % kOwn], to / kOwn) = q;
      } else if (to < (uint32_t)n) {
        keys[to] = q.x;
        perm[to] = q.y;
      }
    }
    if (p + 1 < kPasses) cl.sync();  // the pairs have arrived
  }
}

constexpr int kMaxDevices = 64;

// Blocks a cluster of kernel f may have on the current device (0: unknown
// device), with its dynamic shared memory and cluster size allowed.
template <typename T, int kI, bool kMake>
int cluster_limit() {
  static std::mutex mu;
  static int limit[kMaxDevices] = {0};
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (limit[dev] == 0) {
    auto* f = k_sorted_keys<T, kI, kMake>;
    check(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(Smem<kI>)),
          "sorted keys shared memory");
    check(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
          "sorted keys cluster size");
    int best = -1;
    for (int c = kMaxBlocks; c >= 1 && best < 0; c /= 2) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)c);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = sizeof(Smem<kI>);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim = {(unsigned)c, 1, 1};
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) == cudaSuccess && clusters >= 1)
        best = c;
      else
        (void)cudaGetLastError();
    }
    limit[dev] = best;
  }
  return std::max(limit[dev], 0);
}

// With four keys a thread the keys come from a kernel of their own on the
// whole GPU: in 16 blocks their FP64 quantisation takes 1300 cycles a key of
// each thread.
template <typename T, int kI>
int try_sorted_keys(TreeWork& w, const T* x, const T* y, const T* z, int n, cudaStream_t s) {
  constexpr bool kMake = kI < 4;
  const int need = div_up(n, kThreads * kI);
  if (need > kMaxBlocks) return 0;
  int c = 1;
  while (c < need) c *= 2;
  if (c > cluster_limit<T, kI, kMake>()) return 0;
  if (!kMake) {
    TreeWork to_alt = w;  // unsorted keys to keys_alt
    to_alt.keys = w.keys_alt;
    launch_keys<T>(to_alt, x, y, z, n, s);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)c);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(Smem<kI>);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)c, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  check(cudaLaunchKernelEx(&cfg, k_sorted_keys<T, kI, kMake>, x, y, z,
                           (const uint32_t*)w.keys_alt, n, (const unsigned long long*)w.bbox_enc,
                           w.geom, w.keys, w.perm, w.status),
        "k_sorted_keys launch");
  return kMake ? 1 : 2;
}

}  // namespace

// The cluster sort with the fewest keys a thread that holds n bodies, else
// the key kernel and the one-sweep passes.
template <typename T>
int launch_sorted_keys(TreeWork& w, const T* x, const T* y, const T* z, int n, cudaStream_t s,
                       bool alone) {
  if (alone) {
    int k = try_sorted_keys<T, 1>(w, x, y, z, n, s);
    if (!k) k = try_sorted_keys<T, 2>(w, x, y, z, n, s);
    if (!k) k = try_sorted_keys<T, 4>(w, x, y, z, n, s);
    if (k) return k;
  }
  uint32_t* hist = radix_sort_prepare(w.counts, 30, s);  // counted by the key kernel
  launch_keys<T>(w, x, y, z, n, s, hist);
  radix_sort_pairs(w.keys, w.perm, w.keys_alt, w.perm_alt, w.counts, n, 30, s, w.status, true);
  return 5;
}

template int launch_sorted_keys<float>(TreeWork&, const float*, const float*, const float*, int,
                                       cudaStream_t, bool);
template int launch_sorted_keys<double>(TreeWork&, const double*, const double*, const double*,
                                        int, cudaStream_t, bool);
template int launch_sorted_keys<HiLo>(TreeWork&, const HiLo*, const HiLo*, const HiLo*, int,
                                      cudaStream_t, bool);

}  // namespace nb
