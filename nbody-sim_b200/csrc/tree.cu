// tree.cu -- on-device octree build: bbox, Morton keys, FP64 moments, and the
// compressed octree with contiguous children straight from the sorted keys.
//
// Replaces resetOctree / launchBBoxKernel / launchBuildKernel /
// launchSummarizeKernel of the reference (BHTree.cu:42-317,397-516): no 9N
// node reset, no host round trips for the bbox and the root, no CAS
// insertion, one bottom-up pass instead of 20 summarize launches.
//
// Geometry follows the reference: the bbox is padded x1.001 about its middle
// (BHTree.cu:440-446) and the root half-size pads the largest extent x1.001
// again (BHTree.cu:484-485).  A node at octree level L is the cube of side
// 2*rhs/2^L that the first 3L key bits select; its half-size rhs/2^L is the
// `cell_size` of the reference's opening test (BHTree.cu:577).
#include "common.cuh"
#include "digit_hist.cuh"
#include "geom.cuh"
#include "kernels.cuh"
#include "moments.cuh"

namespace nb {
namespace {

constexpr int kThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kThreads)
k_bbox(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ z, int n,
       unsigned long long* __restrict__ enc) {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double p[3] = {(double)x[i], (double)y[i], (double)z[i]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = fmin(lo[k], p[k]);
      hi[k] = fmax(hi[k], p[k]);
    }
  }
  __shared__ double s[6][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double a = warp_min(lo[k]), b = warp_max(hi[k]);
    if (lane == 0) { s[k][warp] = a; s[3 + k][warp] = b; }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    int k = threadIdx.x;
    double v = s[k][0];
    for (int w = 1; w < kThreads / 32; ++w) v = (k < 3) ? fmin(v, s[k][w]) : fmax(v, s[k][w]);
    if (v == v && fabs(v) != INFINITY) {
      if (k < 3) atomicMin(&enc[k], ordered_bits(v));
      else atomicMax(&enc[k], ordered_bits(v));
    }
  }
}

__global__ void k_bbox_reset(unsigned long long* enc) {
  int k = threadIdx.x;
  if (k < 6) enc[k] = (k < 3) ? ~0ull : 0ull;
}

// The key kernels give each block one contiguous run of keys (a multiple of
// the block size, so every warp's keys are 32 consecutive ones): the keys
// arrive nearly sorted, so a run's high digits take few values, and the
// block adds far fewer non-zero bins to the global histograms than a
// grid-strided block, whose keys span the whole key range, would.
__device__ __forceinline__ long long key_block_span(long long end) {
  const long long per = (end + gridDim.x - 1) / gridDim.x;
  return (per + blockDim.x - 1) / blockDim.x * blockDim.x;
}

// Keys of n positions; hist (optional, 4 x 256 words, cleared) receives the
// digit counts of the four 8-bit passes of the radix sort that follows.
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_keys(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ z, int n,
       const unsigned long long* __restrict__ enc, TreeGeom* __restrict__ geom_out,
       uint32_t* __restrict__ keys, uint32_t* __restrict__ perm, int* __restrict__ status,
       uint32_t* __restrict__ hist) {
  __shared__ TreeGeom g;
  __shared__ uint32_t s_h[4][kHistBins];
  if (threadIdx.x == 0) {
    compute_geom(enc, g);
    if (blockIdx.x == 0) *geom_out = g;
  }
  if (hist)
    for (int i = threadIdx.x; i < 4 * kHistBins; i += blockDim.x) (&s_h[0][0])[i] = 0;
  __syncthreads();
  const long long end = hist ? (n + 31) / 32 * 32 : n;  // whole warps count digits (hist_add)
  const long long span = key_block_span(end);
  const long long stop = min(end, ((long long)blockIdx.x + 1) * span);
  for (long long i = (long long)blockIdx.x * span + threadIdx.x; i < stop; i += blockDim.x) {
    const bool valid = i < n;
    uint32_t key = 0;
    if (valid) {
      key = morton_key(g, (double)x[i], (double)y[i], (double)z[i], status);
      keys[i] = key;
      perm[i] = (uint32_t)i;
    }
    if (hist) hist_add(s_h, key, valid, 4);
  }
  if (hist) {
    __syncthreads();
    hist_flush(s_h, 4, hist);
  }
}

__global__ void k_geoms(const unsigned long long* __restrict__ enc, TreeGeom* __restrict__ geoms,
                        int n_disks) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= n_disks) return;
  TreeGeom g;
  compute_geom(enc + 6 * d, g);
  geoms[d] = g;
}

__global__ void k_bbox_reset_n(unsigned long long* enc, int n_disks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 6 * n_disks) enc[i] = ((i % 6) < 3) ? ~0ull : 0ull;
}

// Ensemble keys: (disk << 30) | Morton key in the disk's own root cube.
template <typename T>
__global__ void __launch_bounds__(kThreads)
k_keys_multi(const T* __restrict__ x, const T* __restrict__ y, const T* __restrict__ z,
             const int* __restrict__ disk, int n, const TreeGeom* __restrict__ geoms,
             uint64_t* __restrict__ keys, uint32_t* __restrict__ perm, int* __restrict__ status,
             uint32_t* __restrict__ hist, int passes) {
  __shared__ uint32_t s_h[kHistMaxPasses][kHistBins];
  if (hist) {
    for (int i = threadIdx.x; i < passes * kHistBins; i += blockDim.x) (&s_h[0][0])[i] = 0;
    __syncthreads();
  }
  const long long end = hist ? (n + 31) / 32 * 32 : n;  // whole warps count digits (hist_add)
  const long long span = key_block_span(end);
  const long long stop = min(end, ((long long)blockIdx.x + 1) * span);
  for (long long i = (long long)blockIdx.x * span + threadIdx.x; i < stop; i += blockDim.x) {
    const bool valid = i < n;
    uint64_t key = 0;
    if (valid) {
      const int d = disk[i];
      const TreeGeom& g = geoms[d];
      key = ((uint64_t)d << 30) |
            (uint64_t)morton_key(g, (double)x[i], (double)y[i], (double)z[i], status);
      keys[i] = key;
      perm[i] = (uint32_t)i;
    }
    if (hist) hist_add(s_h, key, valid, passes);
  }
  if (hist) {
    __syncthreads();
    hist_flush(s_h, passes, hist);
  }
}

__global__ void __launch_bounds__(kThreads)
k_gather_body4(const uint32_t* __restrict__ perm, const float* __restrict__ x,
               const float* __restrict__ y, const float* __restrict__ z,
               const float* __restrict__ m, int n, float4* __restrict__ body4) {
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < n;
       s += (long long)gridDim.x * blockDim.x) {
    uint32_t o = perm[s];
    body4[s] = make_float4(x[o], y[o], z[o], m ? m[o] : 1.f);
  }
}

// ---------------------------------------------------------------- Karras
// delta(i, j): common prefix of keys i and j, with the index as tie-break so
// equal keys still form a valid binary radix tree (Karras 2012, sec. 4).
__device__ __forceinline__ int clz_key(uint32_t v) { return __clz(v); }
__device__ __forceinline__ int clz_key(uint64_t v) { return __clzll((long long)v); }

// ki = keys[i], loaded once by the caller.
template <typename K>
__device__ __forceinline__ int delta(const K* __restrict__ keys, int n, K ki, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const K kj = __ldg(keys + j);
  if (ki != kj) return clz_key(ki ^ kj);
  return 8 * (int)sizeof(K) + __clz((uint32_t)i ^ (uint32_t)j);
}

// The binary radix tree as nbody_radix_tree_u32 hands it out (the octree
// build needs none: k_cells below).  key_bits: the low bits of K the keys use.
// prefix[] stores the common prefix in those bits, key_bits for runs of equal
// keys.  Tried and slower at N = 2^20: staging the block's keys and a halo in
// shared memory (35 -> 39 us), and a bottom-up agglomerative build (Apetrei
// 2014; 130 us: the last climbers' chains of atomics and fences run the depth
// of the tree).

// Writes internal node i: range end j, split offset s along direction d, and
// dnode = delta(i, j).
template <typename K>
__device__ __forceinline__ void karras_write(int i, int j, int d, int s, int dnode, int n,
                                             int key_bits, int* __restrict__ left,
                                             int* __restrict__ right, int* __restrict__ lo_out,
                                             int* __restrict__ hi_out,
                                             uint8_t* __restrict__ prefix) {
  const int gamma = i + s * d + min(d, 0);
  const int lo = min(i, j), hi = max(i, j);
  left[i] = (lo == gamma) ? (n - 1) + gamma : gamma;
  right[i] = (hi == gamma + 1) ? (n - 1) + gamma + 1 : gamma + 1;
  lo_out[i] = lo;
  hi_out[i] = hi;
  constexpr int kW = 8 * (int)sizeof(K);
  prefix[i] = (uint8_t)(dnode >= kW ? key_bits : dnode - (kW - key_bits));
}

// The whole warp narrows [lo, hi) to the last m with delta(i, i + m d) > thr
// (true at lo, false at hi; the predicate only turns false once as m grows,
// Karras 2012 sec. 3): each round every lane tests one of 31 evenly spaced
// points and a ballot keeps the step after the last true one.
template <typename K>
__device__ __forceinline__ long long warp_last_above(const K* __restrict__ keys, int n, K ki,
                                                     int i, int d, int thr, long long lo,
                                                     long long hi, int lane) {
  while (hi - lo > 1) {
    const long long step = (hi - lo + 31) / 32;
    const long long m = lo + (long long)(lane + 1) * step;
    const bool q = m < hi && delta(keys, n, ki, i, i + (int)m * d) > thr;
    const long long nlo = lo + (long long)__popc(__ballot_sync(kFull, q)) * step;
    hi = min(hi, nlo + step);
    lo = nlo;
  }
  return lo;
}

// One thread per internal node (Karras 2012, Fig. 4): direction, range end
// by an exponential then a binary search, split by a binary search.  A warp
// runs each search as many steps as its widest node needs, so a node whose
// range reaches kKarrasCap bodies is handed to the whole warp instead, which
// searches 32 points a step: the lanes' own searches stop at kKarrasCap.
constexpr int kKarrasCap = 1024;

template <typename K>
__global__ void __launch_bounds__(kThreads)
k_karras(const K* __restrict__ keys, int n, int key_bits, int* __restrict__ left,
         int* __restrict__ right, int* __restrict__ lo_out, int* __restrict__ hi_out,
         uint8_t* __restrict__ prefix) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool act = i < n - 1;  // every lane stays for the warp's ballots
  K ki = 0;
  int d = 1, dmin = 0;
  bool wide = false;
  if (act) {
    ki = __ldg(keys + i);
    d = (delta(keys, n, ki, i, i + 1) - delta(keys, n, ki, i, i - 1)) > 0 ? 1 : -1;
    dmin = delta(keys, n, ki, i, i - d);
    int lmax = 2;
    while (lmax <= kKarrasCap && delta(keys, n, ki, i, i + lmax * d) > dmin) lmax <<= 1;
    wide = lmax > kKarrasCap;
    if (!wide) {
      int l = 0;
      for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, ki, i, i + (l + t) * d) > dmin) l += t;
      const int j = i + l * d;
      const int dnode = delta(keys, n, ki, i, j);
      int s = 0, t = l;
      do {
        t = (t + 1) >> 1;
        if (delta(keys, n, ki, i, i + (s + t) * d) > dnode) s += t;
      } while (t > 1);
      karras_write<K>(i, j, d, s, dnode, n, key_bits, left, right, lo_out, hi_out, prefix);
    }
  }
  // wide nodes, one at a time: delta(i, i + kKarrasCap d) > dmin holds, and
  // nothing lies beyond n - 1 steps
  unsigned todo = __ballot_sync(kFull, wide);
  while (todo) {
    const int b = __ffs(todo) - 1;
    todo &= todo - 1;
    const int bi = __shfl_sync(kFull, i, b), bd = __shfl_sync(kFull, d, b);
    const int bmin = __shfl_sync(kFull, dmin, b);
    const K bk = __shfl_sync(kFull, ki, b);
    // the power of two the range end lies below: lane k tests kKarrasCap << k
    const long long mk = (long long)kKarrasCap << lane;
    const bool p = mk < n && delta(keys, n, bk, bi, bi + (int)mk * bd) > bmin;
    const int top = 31 - __clz(__ballot_sync(kFull, p) | 1u);
    const long long lo = (long long)kKarrasCap << top;
    const int l = (int)warp_last_above(keys, n, bk, bi, bd, bmin, lo, min(2 * lo, (long long)n),
                                       lane);
    const int j = bi + l * bd;
    const int dnode = delta(keys, n, bk, bi, j);
    const int s = (int)warp_last_above(keys, n, bk, bi, bd, dnode, 0ll, (long long)l, lane);
    if (lane == b)
      karras_write<K>(bi, j, bd, s, dnode, n, key_bits, left, right, lo_out, hi_out, prefix);
  }
}

// ------------------------------------------------------------- moments
// FP64 prefix sums of (m, m x, m y, m z) over the bodies in key order, kept
// tile-local: ploc[k] sums the bodies of k's tile before k, tpre[t] sums the
// tiles before t.  A node's moments over [lo, end) are then
//   (ploc[end] - ploc[lo]) + (tpre[tile(end)] - tpre[tile(lo)]),
// two differences of partial sums no larger than the node's own tiles, so
// cancellation stays at the level of a tile (~1e-13 relative) rather than of
// the whole disk.  Fixed tiling: the sums are the same on every run.
constexpr int kMomThreads = kMomentThreads;
constexpr int kTileM = kMomentTile;

// Two bodies per thread keep the registers low and the loads and stores
// nearly contiguous (8 bodies per thread needed 93 registers and ran at 21%
// warp occupancy).
__global__ void __launch_bounds__(kMomThreads)
k_moment_tiles(const float4* __restrict__ body4, const double* __restrict__ xd,
               const double* __restrict__ yd, const double* __restrict__ zd, int n,
               double4* __restrict__ ploc, double4* __restrict__ tile_sum) {
  const long long base = (long long)blockIdx.x * kTileM + 2ll * threadIdx.x;
  double4 v[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long i = base + k;
    v[k] = make_double4(0, 0, 0, 0);
    if (i < n) {
      const float4 b = body4[i];
      v[k] = body_moment((double)b.w, xd ? xd[i] : (double)b.x, yd ? yd[i] : (double)b.y,
                         zd ? zd[i] : (double)b.z);
    }
  }
  moment_tile_scan(v[0], v[1], base, n, ploc, tile_sum);
}

// Exclusive scan of the tile sums into tpre[0..ntiles] by one block of kT
// threads (chunks of kT tiles, a fixed order of additions).
template <int kT>
__device__ __forceinline__ void tile_scan(const double4* __restrict__ tile_sum, int ntiles,
                                          double4* __restrict__ tpre) {
  constexpr int kWarps = kT / 32;
  __shared__ double4 s_w[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double4 carry = make_double4(0, 0, 0, 0);
  for (int c0 = 0; c0 < ntiles; c0 += kT) {
    const int t = c0 + tid;
    const double4 x = (t < ntiles) ? tile_sum[t] : make_double4(0, 0, 0, 0);
    const double4 inc = d4warp_incl_scan(x, lane);
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    double4 run = carry;
    for (int w = 0; w < kWarps; ++w) {
      if (w == warp) run = carry;
      carry = d4add(carry, s_w[w]);
    }
    run = d4add(run, d4sub(inc, x));
    if (t < ntiles) tpre[t] = run;
    if (t == ntiles - 1) tpre[ntiles] = d4add(run, x);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_tile_scan(const double4* __restrict__ tile_sum,
                                                   int ntiles, double4* __restrict__ tpre) {
  tile_scan<256>(tile_sum, ntiles, tpre);
}

// ------------------------------------------------- octree cells + groups
// The compressed octree straight from the sorted keys, with no binary tree
// between them.  Let lev(a, b) be the octree level two keys share (0 .. 10;
// -1: different disks).  Body k starts a cell at level L when lev(k-1, k) < L,
// and that cell has more than P bodies when lev(k, k+P) >= L: two key reads
// tell a body that it starts no cell which needs child records, and at
// N = 2^20 nine bodies in ten stop there.  The others list their (body,
// level) candidates, and eight lanes take each: lane o finds the end of
// octant o by a search of the keys.  A candidate with bodies in two or more
// octants is a node of the compressed octree; its children are those octants.
//
// Child slots come from one counter (a block takes the slots of all its
// nodes with one atomic), so siblings stay contiguous and no pass scans the
// node counts.  Which slots a node's children hold is kept under the node's
// first body, or, for a node that is its parent's first child (and so starts
// where its parent does), under its last body: no two nodes share an entry.
// k_emit then writes one record per slot.
//
// Target groups: a maximal binary node (bodies sharing a key prefix, the
// index breaking ties) of <= gspan bodies is cut into the fewest equal runs
// of <= gmax.  Groups partition the bodies into contiguous key ranges inside
// one node's cell, so a group never straddles a jump of the space-filling
// curve (a fixed run of 32 consecutive bodies can: its box then spans most of
// the domain and its walk degenerates to O(N) work on one warp).  gspan =
// gmax gives the maximal nodes of <= gmax bodies themselves; a larger gspan
// fills the warps better (a node of 40 bodies is two runs of 20, not a binary
// split such as 5 + 30 + 5) at the price of larger boxes.  Bodies i-1 and i
// are in different group nodes exactly when the smallest node holding both,
// the run sharing delta(i-1, i) bits, has more than gspan bodies.  Groups
// never span disks.
//
// One launch instead of five (Karras tree, child counts, scan, slots, and
// the scan of the moment tiles, which block 0 does here) and a search per
// octree child instead of two per binary node: the tree phase takes 14 / 17 /
// 19 / 39 / 111 us at N = 4096 / 30011 / 131072 / 2^20 / 2^22, against 31 /
// 35 / 38 / 86 / 318 us.  What bounds it is a block's chain of dependent key
// reads (group search, octant search, the atomic), 3 us long, with issue
// slots 40% used.  Measured slower at 2^20: keys and a halo of 256 staged in
// shared memory (46 against 41 us, one body a thread), the searches run by
// every body's own thread instead of from the lists (45 against 28 us), and
// the groups listed in body order (31 against 27 us; the walk is the same).
constexpr int kMaxLevel = 10;
// From here on two bodies a thread (2^20: 27 against 30 us with one); below,
// one, so that there are blocks for more SMs (131072: 11 against 15.5 us).
constexpr int kCellLargeBodies = 1 << 18;

__device__ __forceinline__ int level_of_diff(uint32_t x) {  // x: differing Morton bits
  return x ? (__clz(x) - 2) / 3 : kMaxLevel;
}
__device__ __forceinline__ int oct_level(uint32_t a, uint32_t b) { return level_of_diff(a ^ b); }
__device__ __forceinline__ int oct_level(uint64_t a, uint64_t b) {
  const uint64_t x = a ^ b;
  return (x >> 30) ? -1 : level_of_diff((uint32_t)x);
}

// Disk index of a key (the bits above the 30 Morton bits).
template <typename K>
__device__ __forceinline__ int key_disk(K k) { return sizeof(K) == 4 ? 0 : (int)(k >> 30); }

// A cell's child slots as kept per body: first slot - n_roots << 4 | children.
__device__ __forceinline__ uint32_t pack_cell(uint32_t first, uint32_t nch) {
  return (first << 4) | nch;
}

template <typename K>
struct CellArgs {
  int n, n_roots, gmax, gshift, gspan, prune;  // gmax = 1 << gshift
  const K* keys;
  int2* slot;         // slot -> (first body, bodies << 1 | is its parent's first child)
  uint32_t* cell_lo;  // pack_cell of the node whose first body this is
  uint32_t* cell_hi;  // the same for first children, under their last body
  unsigned long long* alloc;  // child slots << 32 | groups (zeroed)
  int2* groups;
  int* group_disk;    // optional: disk of each group
  int2* group_span;   // optional: (first group of the span node, its bodies)
  const double4* tile_sum;  // moment tiles for block 0 to scan into tpre (optional)
  double4* tpre;
  int ntiles;
};

// A key prefix, the index extending equal keys: body j shares it with body i
// when key_i ^ key_j <= key and i ^ j <= index.
template <typename K>
struct Prefix {
  K key;
  uint32_t index;
};

// The longest prefix two bodies share: x their keys' difference, ix their
// indices'.
template <typename K>
__device__ __forceinline__ Prefix<K> shared_prefix(K x, uint32_t ix) {
  if (x) return {(K)(~(K)0 >> clz_key(x)), ~0u};
  return {(K)0, ~0u >> __clz((int)ix)};
}

template <typename K>
__device__ __forceinline__ bool shares(const K* __restrict__ keys, int n, K ki, int i, int j,
                                       const Prefix<K> p) {
  return (unsigned)j < (unsigned)n && (K)(ki ^ __ldg(keys + j)) <= p.key &&
         (uint32_t)(i ^ j) <= p.index;
}

// Whether neither half of a span still shares the prefix of bodies i-1 and i:
// the smallest node that holds both is then within a span.
template <typename K>
__device__ __forceinline__ bool within_span(const K* __restrict__ keys, int n, K ki, int i,
                                            int gspan, const Prefix<K> p) {
  const int h = (gspan + 1) / 2;
  return !shares(keys, n, ki, i, i - h, p) && !shares(keys, n, ki, i, i + h, p);
}

// Bodies of the group node that starts at body i (0: none does).
template <typename K>
__device__ __forceinline__ int group_node(const K* __restrict__ keys, int n, int i, int gspan) {
  const int top = 1 << (31 - __clz(gspan));
  const K ki = __ldg(keys + i);
  Prefix<K> p = {(K)0x3fffffffu, ~0u};  // any body of the disk
  bool inside = false;
  if (i > 0) {
    const K x = ki ^ __ldg(keys + i - 1);
    inside = (x >> 30) == 0;
    if (inside) p = shared_prefix<K>(x, (uint32_t)(i ^ (i - 1)));
  }
  if (inside) {
    int x = 0;  // bodies of the node of i-1 and i before i, at most gspan
    for (int step = top; step > 0; step >>= 1)
      if (x + step <= gspan && shares(keys, n, ki, i, i - x - step, p)) x += step;
    if (x < gspan && !shares(keys, n, ki, i, i - x + gspan, p)) return 0;
  }
  // the node: the longest run within gspan bodies that shares one bit more
  // than bodies i-1 and i, and than bodies i and i + gspan, do
  const int e = i + gspan;
  Prefix<K> q = p;
  if (inside) q = {(K)(p.key >> 1), p.key ? ~0u : p.index >> 1};
  if (e < n) {
    const Prefix<K> r = shared_prefix<K>((K)(ki ^ __ldg(keys + e)), (uint32_t)(i ^ e));
    const Prefix<K> d = {(K)(r.key >> 1), r.key ? ~0u : r.index >> 1};
    if (d.key < q.key) q = d;
    else if (d.key == q.key) q.index = min(q.index, d.index);
  }
  int t = 0;
  for (int step = top; step > 0; step >>= 1)
    if (t + step < gspan && shares(keys, n, ki, i, i + t + step, q)) t += step;
  return t + 1;
}

// First body j > k whose key is at least `target` (n if none), keys[k] < target.
template <typename K>
__device__ __forceinline__ int first_at_least(const K* __restrict__ keys, int n, int k,
                                              K target) {
  int lo = k, step = 8;
  while (step < n - k && __ldg(keys + k + step) < target) {
    lo = k + step;
    step <<= 2;
  }
  int hi = (step < n - k) ? k + step : n;
  while (hi - lo > 1) {
    const int mid = lo + ((hi - lo) >> 1);
    if (__ldg(keys + mid) < target) lo = mid;
    else hi = mid;
  }
  return hi;
}

template <typename K, int kT, int kItems>
__global__ void __launch_bounds__(kT, 2048 / kT) k_cells(const CellArgs<K> a) {
  constexpr int kBodies = kT * kItems;
  constexpr int kSubs = kT / 8;  // candidates in flight
  constexpr int kPer = kSubs / 32;
  static_assert(kSubs % 32 == 0 && kBodies <= 4096, "one warp scans a round's child counts");
  if (a.ntiles > 0 && blockIdx.x == 0) {
    tile_scan<kT>(a.tile_sum, a.ntiles, a.tpre);
    return;
  }
  __shared__ uint16_t s_task[kBodies * kMaxLevel];  // candidates: body << 4 | level
  __shared__ uint16_t s_grp[kBodies];   // bodies that may start a group node
  __shared__ uint16_t s_size[kBodies];  // their nodes' bodies
  __shared__ uint16_t s_run[kBodies];   // and first runs
  __shared__ uint32_t s_cnt[kSubs];
  __shared__ int s_ntask, s_ngrp, s_nrun;
  __shared__ unsigned long long s_base;
  const int tid = threadIdx.x, lane = tid & 31;
  const int n = a.n;
  const K* __restrict__ keys = a.keys;
  const int b0 = (blockIdx.x - (a.ntiles > 0 ? 1 : 0)) * kBodies;
  if (tid == 0) s_ntask = s_ngrp = s_nrun = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int k = b0 + j * kT + tid;
    if (k >= n) break;
    const int ahead = min(k + max(a.prune, 1), n);
    const K key = __ldg(keys + k);
    const K kl = __ldg(keys + max(k - 1, 0));
    const K kp = __ldg(keys + min(ahead, n - 1));
    const int l = k > 0 ? oct_level(kl, key) : -1;
    const int q = ahead < n ? min(kMaxLevel - 1, oct_level(key, kp)) : -1;
    if (q > l) {
      const int at = atomicAdd(&s_ntask, q - l);
      for (int t = 0; t < q - l; ++t)
        s_task[at + t] = (uint16_t)(((j * kT + tid) << 4) | (l + 1 + t));
    }
    if (l < 0 || !within_span<K>(keys, n, key, k, a.gspan,
                                 shared_prefix<K>((K)(kl ^ key), (uint32_t)((k - 1) ^ k))))
      s_grp[atomicAdd(&s_ngrp, 1)] = (uint16_t)(j * kT + tid);
    if (l < 0) {  // a disk's root: slot = the disk index
      int end = n;
      if constexpr (sizeof(K) == 8)
        if (a.n_roots > 1) end = first_at_least<K>(keys, n, k, (K)(key_disk(key) + 1) << 30);
      a.slot[key_disk(key)] = make_int2(k, (end - k) << 1);
    }
  }
  __syncthreads();
  const int ntasks = s_ntask, ngrp = s_ngrp;
  // group nodes: from the block's last thread down, as the candidates start
  // from its first
  for (int i = kT - 1 - tid; i < ngrp; i += kT) {
    const int size = group_node<K>(keys, n, b0 + s_grp[i], a.gspan);
    s_size[i] = (uint16_t)size;
    if (size) s_run[i] = (uint16_t)atomicAdd(&s_nrun, (size + a.gmax - 1) >> a.gshift);
  }
  const int sub = tid >> 3, o = tid & 7;
  uint32_t gbase = 0;
  for (int t0 = 0; t0 < max(ntasks, 1); t0 += kSubs) {
    const int t = t0 + sub;
    int end = 0, first = 0;
    bool is_first = false;
    if (t < ntasks) {
      first = b0 + (s_task[t] >> 4);
      const K fk = __ldg(keys + first);
      const int shift = 3 * (kMaxLevel - 1 - (s_task[t] & 15));
      const K target = (K)(((fk >> (shift + 3)) << 3) + (K)(o + 1)) << shift;
      end = (fk >= target) ? first : first_at_least<K>(keys, n, first, target);
      // its parent starts with it too when the level on its other side is
      // deeper than lev(first - 1, first)
      if (o == 7 && end < n) {
        const int le = oct_level(__ldg(keys + end - 1), __ldg(keys + end));
        is_first = le > (first > 0 ? oct_level(__ldg(keys + first - 1), fk) : -1);
      }
    }
    const int before = __shfl_up_sync(kFull, end, 1, 8);
    const int s = o == 0 ? first : before;
    const int count = end - s;
    const unsigned kids = (__ballot_sync(kFull, count > 0) >> (lane & 24)) & 0xffu;
    int nch = __popc(kids);
    if (nch < 2) nch = 0;  // one octant: the same bodies as a deeper cell
    if (o == 0) s_cnt[sub] = (uint32_t)nch;
    __syncthreads();
    if (tid < 32) {  // exclusive scan of the round's child counts, one atomic for its slots
      uint32_t c[kPer], sum = 0;
#pragma unroll
      for (int r = 0; r < kPer; ++r) {
        c[r] = sum;
        sum += s_cnt[kPer * lane + r];
      }
      const uint32_t ci = warp_incl_scan(sum, lane);
#pragma unroll
      for (int r = 0; r < kPer; ++r) s_cnt[kPer * lane + r] = ci - sum + c[r];
      if (lane == 31) {
        const unsigned long long add =
            ((unsigned long long)ci << 32) | (unsigned long long)(t0 == 0 ? s_nrun : 0);
        s_base = add ? atomicAdd(a.alloc, add) : 0ull;
      }
    }
    __syncthreads();
    if (t0 == 0) gbase = (uint32_t)s_base;
    if (nch > 0) {
      const uint32_t slot0 = (uint32_t)(s_base >> 32) + s_cnt[sub];
      if (count > 0)
        a.slot[a.n_roots + (int)slot0 + __popc(kids & ((1u << o) - 1u))] =
            make_int2(s, (count << 1) | (s == first ? 1 : 0));
      if (o == 7) {
        if (is_first) a.cell_hi[end - 1] = pack_cell(slot0, (uint32_t)nch);
        else a.cell_lo[first] = pack_cell(slot0, (uint32_t)nch);
      }
    }
    if (t0 + kSubs < ntasks) __syncthreads();  // s_cnt and s_base are rewritten
  }
  for (int i = kT - 1 - tid; i < ngrp; i += kT) {
    const int size = s_size[i];
    if (size == 0) continue;
    // runs of size / runs or size / runs + 1 consecutive bodies
    const int k = b0 + s_grp[i], runs = (size + a.gmax - 1) >> a.gshift;
    const int g0 = (int)gbase + s_run[i], q = size / runs, r = size % runs;
    const int disk = a.group_disk ? key_disk(__ldg(keys + k)) : 0;
    for (int j = 0, s = k; j < runs; ++j) {
      const int sz = q + (j < r ? 1 : 0);
      a.groups[g0 + j] = make_int2(s, sz);
      if (a.group_disk) a.group_disk[g0 + j] = disk;
      if (a.group_span) a.group_span[g0 + j] = make_int2(g0, size);
      s += sz;
    }
  }
}

__device__ __forceinline__ uint32_t compact3(uint32_t v) {
  v &= 0x09249249u;
  v = (v ^ (v >> 2)) & 0x030c30c3u;
  v = (v ^ (v >> 4)) & 0x0300f00fu;
  v = (v ^ (v >> 8)) & 0x030000ffu;
  v = (v ^ (v >> 16)) & 0x000003ffu;
  return v;
}

template <typename K>
struct EmitArgs {
  int n, n_roots, prune;
  const K* keys;
  const int2* slot;
  const uint32_t* cell_lo;
  const uint32_t* cell_hi;
  const unsigned long long* alloc;
  int* n_nodes;
  const float4* body4;
  const double4* ploc;  // nullptr: no centres of mass (a neighbour search reads none)
  const double4* tpre;
  const TreeGeom* geom;
  OctNodes oct;
  bool boxes;  // also the records' boxes (the neighbour search reads them)
};

// A node's cube: the level L cell of its first key (side 2 rhs / 2^L, exact
// power-of-two scaling), grown by a margin for float positions that sit an
// ulp outside their FP64-quantised cell, and its centre.
struct NodeCube {
  float lo[3], hi[3], mid[3];
};
template <typename K>
__device__ __forceinline__ NodeCube node_cube(const TreeGeom* __restrict__ geom, K klo, int L) {
  const uint32_t kl = (uint32_t)(klo & (K)0x3fffffffu) >> (3 * (kMaxLevel - L));
  const uint32_t cc[3] = {compact3(kl), compact3(kl >> 1), compact3(kl >> 2)};
  const double side = (double)geom->rhs * (double)(2.0f / (float)(1u << L));
  NodeCube c;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double l0 = geom->lo[k] + (double)cc[k] * side;
    const float fl = (float)l0, fs = (float)side;
    const float margin = 1e-6f * (fabsf(fl) + fs) + 1e-30f;
    c.lo[k] = fl - margin;
    c.hi[k] = fl + fs + margin;
    c.mid[k] = fl + 0.5f * fs;
  }
  return c;
}

// Writes the octree record of slot f.
template <typename K>
__device__ void write_node(const EmitArgs<K>& a, int f) {
  const int2 sl = a.slot[f];
  const int lo = sl.x, cnt = sl.y >> 1;
  const K klo = a.keys[lo];
  const TreeGeom* geom = a.geom + key_disk(klo);
  const float rhs = geom->rhs;
  if (cnt == 1) {  // single-body leaf
    const float4 p = a.body4[lo];
    a.oct.com[f] = p;
    a.oct.info[f] = make_int4(-1, lo, (1 << 4), __float_as_int(ldexpf(rhs, -kMaxLevel)));
    if (a.boxes) {
      a.oct.box_lo[f] = make_float4(p.x, p.y, p.z, 0.f);
      a.oct.box_hi[f] = make_float4(p.x, p.y, p.z, 0.f);
    }
    return;
  }
  // loaded before the record's stores (the arrays carry no restrict)
  const int L = oct_level(klo, a.keys[lo + cnt - 1]);
  uint32_t cell = 0;
  const bool open = cnt > a.prune && L < kMaxLevel;
  if (open) cell = (sl.y & 1) ? a.cell_hi[lo + cnt - 1] : a.cell_lo[lo];
  const int nch = (int)(cell & 15u);
  const int first_child = open ? a.n_roots + (int)(cell >> 4) : -1;
  double4 s = make_double4(0, 0, 0, 0);
  if (a.ploc) s = range_moments(a.ploc, a.tpre, lo, lo + cnt);
  const NodeCube c = node_cube<K>(geom, klo, L);
  a.oct.com[f] = com_of(s, c.mid[0], c.mid[1], c.mid[2]);
  a.oct.info[f] = make_int4(first_child, lo, (cnt << 4) | nch, __float_as_int(ldexpf(rhs, -L)));
  if (a.boxes) {
    a.oct.box_lo[f] = make_float4(c.lo[0], c.lo[1], c.lo[2], 0.f);
    a.oct.box_hi[f] = make_float4(c.hi[0], c.hi[1], c.hi[2], 0.f);
  }
}

// One thread per record; consecutive slots are siblings, so the record
// stores coalesce.  The record count is read on the device (a grid-stride
// loop over it).
template <typename K>
__global__ void __launch_bounds__(kThreads) k_emit(const EmitArgs<K> a) {
  const int total = a.n_roots + (int)(*a.alloc >> 32);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.n_nodes = total;
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < total; f += gridDim.x * blockDim.x)
    write_node(a, f);
}

// The boxes alone of the records there are (one disk), for a search of `radius`:
// none when it goes by cells.
__global__ void __launch_bounds__(kThreads)
k_boxes(const uint32_t* __restrict__ keys, const int2* __restrict__ slot,
        const float4* __restrict__ body4, const TreeGeom* __restrict__ geom,
        const unsigned long long* __restrict__ alloc, float radius,
        float4* __restrict__ box_lo, float4* __restrict__ box_hi) {
  if (by_cells(*geom, radius)) return;
  const int total = 1 + (int)(*alloc >> 32);
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < total; f += gridDim.x * blockDim.x) {
    const int2 sl = slot[f];
    const int lo = sl.x, cnt = sl.y >> 1;
    float4 b0 = body4[lo], b1 = b0;
    if (cnt > 1) {
      const uint32_t klo = keys[lo];
      const NodeCube c = node_cube<uint32_t>(geom, klo, oct_level(klo, keys[lo + cnt - 1]));
      b0 = make_float4(c.lo[0], c.lo[1], c.lo[2], 0.f);
      b1 = make_float4(c.hi[0], c.hi[1], c.hi[2], 0.f);
    }
    box_lo[f] = make_float4(b0.x, b0.y, b0.z, 0.f);
    box_hi[f] = make_float4(b1.x, b1.y, b1.z, 0.f);
  }
}

// N == 1: the root is the single body and the only group.
__global__ void k_single(const float4* __restrict__ body4, const TreeGeom* __restrict__ geom,
                         OctNodes oct, int* __restrict__ n_nodes, int2* __restrict__ groups,
                         int* __restrict__ n_groups) {
  float4 p = body4[0];
  oct.com[0] = p;
  oct.info[0] = make_int4(-1, 0, (1 << 4), __float_as_int(geom->rhs));
  oct.box_lo[0] = make_float4(p.x, p.y, p.z, 0.f);
  oct.box_hi[0] = make_float4(p.x, p.y, p.z, 0.f);
  *n_nodes = 1;
  groups[0] = make_int2(0, 1);
  *n_groups = 1;
}

template <typename T>
T* dalloc(size_t count, const char* what) {
  T* p = nullptr;
  check(cudaMalloc(&p, sizeof(T) * (count ? count : 1)), what);
  return p;
}

int grid_for(long long n) { return (int)((n + kThreads - 1) / kThreads); }

}  // namespace

void tree_alloc(TreeWork& w, int cap) {
  tree_free(w);
  if (cap < 1) cap = 1;
  w.cap = cap;
  const size_t n = (size_t)cap, nb = 2 * n;
  w.keys = dalloc<uint32_t>(n, "keys");
  w.perm = dalloc<uint32_t>(n, "perm");
  w.keys_alt = dalloc<uint32_t>(n, "keys_alt");
  w.perm_alt = dalloc<uint32_t>(n, "perm_alt");
  w.counts = dalloc<uint32_t>(radix_sort_count_words(cap), "sort counts");
  w.body4 = dalloc<float4>(n, "body4");
  w.mom_ploc = dalloc<double4>(n + 1, "moment prefix");
  w.mom_tiles = dalloc<double4>(2 * ((n + 1) / kTileM + 2), "moment tiles");
  w.oct_slot = dalloc<int2>(nb, "octree slots");
  w.cell_lo = dalloc<uint32_t>(n, "octree cells");
  w.cell_hi = dalloc<uint32_t>(n, "octree cells");
  w.oct.com = dalloc<float4>(nb, "oct com");
  w.oct.info = dalloc<int4>(nb, "oct info");
  w.oct.box_lo = dalloc<float4>(nb, "oct box_lo");
  w.oct.box_hi = dalloc<float4>(nb, "oct box_hi");
  w.bbox_enc = dalloc<unsigned long long>(6, "bbox");
  w.geom = dalloc<TreeGeom>(1, "geom");
  w.n_nodes = dalloc<int>(1, "n_nodes");
  w.groups = dalloc<int2>(n, "groups");
  w.alloc = dalloc<unsigned long long>(1, "octree counter");
  w.n_groups = (int*)w.alloc;
  w.status = dalloc<int>(1, "status");
  check(cudaMemset(w.status, 0, sizeof(int)), "status init");
  check(cudaMemset(w.n_nodes, 0, sizeof(int)), "n_nodes init");
}

void tree_free(TreeWork& w) {
  void* ptrs[] = {w.keys,    w.perm,     w.keys_alt, w.perm_alt,   w.counts,     w.body4,
                  w.mom_ploc, w.mom_tiles, w.oct_slot, w.cell_lo,  w.cell_hi,    w.oct.com,
                  w.oct.info, w.oct.box_lo, w.oct.box_hi, w.bbox_enc, w.geom,    w.n_nodes,
                  w.status,  w.groups,   w.alloc};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (w.side) cudaStreamDestroy(w.side);
  w = TreeWork();
}

void tree_enable_overlap(TreeWork& w) {
  if (w.side) return;
  check(cudaStreamCreateWithFlags(&w.side, cudaStreamNonBlocking), "tree side stream");
}

void launch_bbox_reset(TreeWork& w, cudaStream_t s) {
  k_bbox_reset<<<1, 32, 0, s>>>(w.bbox_enc);
}

template <typename T>
void launch_bbox(TreeWork& w, const T* x, const T* y, const T* z, int n, cudaStream_t s) {
  launch_bbox_reset(w, s);
  int g = std::min(grid_for(n), 148 * 8);
  if (g < 1) g = 1;
  k_bbox<T><<<g, kThreads, 0, s>>>(x, y, z, n, w.bbox_enc);
  check(cudaGetLastError(), "k_bbox launch");
}

template <typename T>
void launch_keys(TreeWork& w, const T* x, const T* y, const T* z, int n, cudaStream_t s,
                 uint32_t* hist) {
  // with histograms: fewer blocks, so fewer block histograms to add up
  int g = hist ? std::min(div_up(n, kThreads * 8), 148 * 4) : std::min(grid_for(n), 148 * 16);
  if (g < 1) g = 1;
  k_keys<T><<<g, kThreads, 0, s>>>(x, y, z, n, w.bbox_enc, w.geom, w.keys, w.perm, w.status,
                                   hist);
  check(cudaGetLastError(), "k_keys launch");
}

template void launch_bbox<float>(TreeWork&, const float*, const float*, const float*, int,
                                 cudaStream_t);
template void launch_bbox<double>(TreeWork&, const double*, const double*, const double*, int,
                                  cudaStream_t);
template void launch_keys<float>(TreeWork&, const float*, const float*, const float*, int,
                                 cudaStream_t, uint32_t*);
template void launch_keys<double>(TreeWork&, const double*, const double*, const double*, int,
                                  cudaStream_t, uint32_t*);
template void launch_bbox<HiLo>(TreeWork&, const HiLo*, const HiLo*, const HiLo*, int,
                                cudaStream_t);
template void launch_keys<HiLo>(TreeWork&, const HiLo*, const HiLo*, const HiLo*, int,
                                cudaStream_t, uint32_t*);

void launch_gather_body4(TreeWork& w, const float* x, const float* y, const float* z,
                         const float* m, int n, cudaStream_t s) {
  int g = std::min(grid_for(n), 148 * 16);
  if (g < 1) g = 1;
  k_gather_body4<<<g, kThreads, 0, s>>>(w.perm, x, y, z, m, n, w.body4);
  check(cudaGetLastError(), "k_gather_body4 launch");
}

void launch_geoms(const unsigned long long* enc, TreeGeom* geoms, int n_disks, cudaStream_t s) {
  k_geoms<<<div_up(n_disks, 64), 64, 0, s>>>(enc, geoms, n_disks);
  check(cudaGetLastError(), "k_geoms launch");
}

void launch_bbox_reset_n(unsigned long long* enc, int n_disks, cudaStream_t s) {
  k_bbox_reset_n<<<div_up(6 * n_disks, 256), 256, 0, s>>>(enc, n_disks);
  check(cudaGetLastError(), "k_bbox_reset_n launch");
}

template <typename T>
void launch_keys_multi(const T* x, const T* y, const T* z, const int* disk, int n,
                       const TreeGeom* geoms, uint64_t* keys, uint32_t* perm, int* status,
                       cudaStream_t s, uint32_t* hist, int key_bits) {
  int g = hist ? std::min(div_up(n, kThreads * 8), 148 * 4) : std::min(grid_for(n), 148 * 16);
  if (g < 1) g = 1;
  k_keys_multi<T><<<g, kThreads, 0, s>>>(x, y, z, disk, n, geoms, keys, perm, status, hist,
                                         (key_bits + 7) / 8);
  check(cudaGetLastError(), "k_keys_multi launch");
}

template void launch_keys_multi<float>(const float*, const float*, const float*, const int*, int,
                                       const TreeGeom*, uint64_t*, uint32_t*, int*, cudaStream_t,
                                       uint32_t*, int);
template void launch_keys_multi<double>(const double*, const double*, const double*, const int*,
                                        int, const TreeGeom*, uint64_t*, uint32_t*, int*,
                                        cudaStream_t, uint32_t*, int);
template void launch_keys_multi<HiLo>(const HiLo*, const HiLo*, const HiLo*, const int*, int,
                                      const TreeGeom*, uint64_t*, uint32_t*, int*, cudaStream_t,
                                      uint32_t*, int);

template <typename K>
void emit_records(TreeWork& w, const K* keys, int n, int n_roots, const TreeGeom* geoms,
                  cudaStream_t s) {
  EmitArgs<K> e{n,          n_roots,   w.prune_max, keys,
                w.oct_slot, w.cell_lo, w.cell_hi,   w.alloc,
                w.n_nodes,  w.body4,   w.moments ? w.mom_ploc : nullptr,
                moment_tile_prefix(w, n), geoms, w.oct, w.boxes};
  // one thread per record for up to n / 2 records (about 0.35 n with leaves of
  // eight bodies); the loop covers any more
  k_emit<K><<<std::max(1, div_up(n, 2 * kThreads)), kThreads, 0, s>>>(e);
  check(cudaGetLastError(), "octree launch");
}

template <typename K>
int launch_tree(TreeWork& w, const K* keys, int n, int n_roots, const TreeGeom* geoms,
                int* group_disk, const double* xd, const double* yd, const double* zd,
                cudaStream_t s, bool tiles_done) {
  if (n < 1) return 0;
  if (n == 1) {
    k_single<<<1, 1, 0, s>>>(w.body4, geoms, w.oct, w.n_nodes, w.groups, w.n_groups);
    if (group_disk) check(cudaMemsetAsync(group_disk, 0, sizeof(int), s), "group disk");
    check(cudaGetLastError(), "k_single launch");
    return 1;
  }
  const int ntiles = w.moments ? moment_tiles(n) : 0;
  double4* tpre = moment_tile_prefix(w, n);
  if (!tiles_done) {
    check(cudaMemsetAsync(w.alloc, 0, sizeof(unsigned long long), s), "octree counter reset");
    if (w.moments)
      k_moment_tiles<<<ntiles, kMomThreads, 0, s>>>(w.body4, xd, yd, zd, n, w.mom_ploc,
                                                    w.mom_tiles);
  }
  const int gspan = w.group_max * std::max(1, w.group_span);
  int gshift = 0;
  while ((1 << gshift) < w.group_max) ++gshift;
  CellArgs<K> c{n,          n_roots,   w.group_max, gshift,   gspan,    w.prune_max,
                keys,       w.oct_slot, w.cell_lo,  w.cell_hi, w.alloc,  w.groups,
                group_disk, w.group_spans, w.mom_tiles, tpre,  ntiles};
  const int extra = ntiles > 0 ? 1 : 0;
  if (n < kCellLargeBodies)
    k_cells<K, 512, 1><<<div_up(n, 512) + extra, 512, 0, s>>>(c);
  else
    k_cells<K, 512, 2><<<div_up(n, 1024) + extra, 512, 0, s>>>(c);
  emit_records<K>(w, keys, n, n_roots, geoms, s);
  return (!tiles_done && w.moments ? 1 : 0) + 2;
}

void launch_boxes(const TreeWork& w, int n, float radius, cudaStream_t s) {
  if (n < 2) return;  // one body: k_single wrote its box
  k_boxes<<<std::max(1, div_up(n, 2 * kThreads)), kThreads, 0, s>>>(
      w.keys, w.oct_slot, w.body4, w.geom, w.alloc, radius, w.oct.box_lo, w.oct.box_hi);
  check(cudaGetLastError(), "k_boxes launch");
}

template int launch_tree<uint32_t>(TreeWork&, const uint32_t*, int, int, const TreeGeom*, int*,
                                   const double*, const double*, const double*, cudaStream_t,
                                   bool);
template int launch_tree<uint64_t>(TreeWork&, const uint64_t*, int, int, const TreeGeom*, int*,
                                   const double*, const double*, const double*, cudaStream_t,
                                   bool);

void radix_tree_u32(const uint32_t* keys, int n, int key_bits, int* left, int* right, int* lo,
                    int* hi, uint8_t* prefix) {
  if (n >= 2) {
    k_karras<uint32_t><<<grid_for(n - 1), kThreads>>>(keys, n, key_bits, left, right, lo, hi,
                                                      prefix);
    check(cudaGetLastError(), "k_karras launch");
  }
  check(cudaDeviceSynchronize(), "radix tree");
}

void launch_moment_prefix(TreeWork& w, int n, const double* xd, const double* yd,
                          const double* zd, cudaStream_t s) {
  if (n < 1) return;
  const int ntiles = moment_tiles(n);
  k_moment_tiles<<<ntiles, kMomThreads, 0, s>>>(w.body4, xd, yd, zd, n, w.mom_ploc, w.mom_tiles);
  check(cudaGetLastError(), "moment prefix launch");
  launch_tile_scan(w.mom_tiles, ntiles, moment_tile_prefix(w, n), s);
}

void launch_tile_scan(const double4* tile_sum, int ntiles, double4* tpre, cudaStream_t s) {
  k_tile_scan<<<1, 256, 0, s>>>(tile_sum, ntiles, tpre);
  check(cudaGetLastError(), "tile scan launch");
}

double4* moment_tile_prefix(TreeWork& w, int n) { return w.mom_tiles + (n / kTileM + 2); }

}  // namespace nb
