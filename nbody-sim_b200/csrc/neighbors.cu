// neighbors.cu -- fixed-radius neighbour search over the octree: the
// two-pass collision impulse and the FoF links + union-find.
//
// Radii below half a level-10 cell are searched by cells (k_cell_neighbors
// below), larger ones through the tree (k_neighbors).
//
// Collision replaces bhtree_collisionKernel (BHTree.cu:620-673).  The
// reference prunes a cell when |x - com| - 1.732 half >= r_coll, which can
// skip pairs whose cell COM is off-centre; here a warp group of 32 targets
// descends every node whose tight AABB overlaps the group box grown by the
// radius, so every pair with dist2 < r_coll^2 is found.  The per-pair
// impulse is the reference's (BHTree.cu:650-660): dv_i -= J n with
// J = -(1+e) dvn / 2 for approaching pairs, computed from pre-collision
// velocities (two-pass semantics).
//
// FoF links use the exact test of detectAggregates (Aggregate.cpp:36-42),
// ((dx*dx + dy*dy) + dz*dz) < ll*ll in FP32 without contraction, so the
// linked pair set, the components and their smallest-index labels are
// bit-identical to the host O(N^2) loop.  Union-find always hooks the larger
// root under the smaller one, so every root is its component's smallest
// original index; every loop is bounded and reports kStatusUnionFindLimit.
#include <algorithm>

#include "collide_math.cuh"
#include "common.cuh"
#include "geom.cuh"
#include "kernels.cuh"

namespace nb {
namespace {

constexpr int kNbWarps = 4;
constexpr int kStk = 384;

struct NbSmem {
  float4 pos[64];
  int idx[64];
  int stk[kStk];
  int sc[32];
  int slo[32];
};

__device__ __forceinline__ int uf_find(int* parent, int x) {
  for (int guard = 0; guard < (1 << 26); ++guard) {
    int p = __ldcg(parent + x);
    if (p == x) return x;
    int gp = __ldcg(parent + p);
    if (gp != p) atomicCAS(parent + x, p, gp);  // path halving; parents only decrease
    x = p;
  }
  return -1;
}

__device__ void uf_union(int* parent, int a, int b, int* status) {
  for (int guard = 0; guard < (1 << 20); ++guard) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a < 0 || b < 0) break;
    if (a == b) return;
    if (a > b) { int t = a; a = b; b = t; }
    int old = atomicCAS(parent + b, b, a);
    if (old == b) return;
    b = old;
  }
  atomicOr(status, kStatusUnionFindLimit);
}

struct CollideOut {
  const void* vx;   // velocities in the state's storage type (vtype)
  const void* vy;
  const void* vz;
  int vtype;        // 0 float, 1 double, 2 hi/lo float pairs
  const uint32_t* vmap;
  float rc2;
  float e;
  float* dvx;
  float* dvy;
  float* dvz;
  // report mode: the octree's centres of mass, r_coll and the two counters
  // (pairs, pairs the reference's cell prune would skip)
  const float4* com;
  unsigned long long* report;
};

// Whether bhtree_collisionKernel would skip the pair (target at xi, sorted
// body j): descending the octree cells that contain j, the first whose
// |com - x_i| - 1.732 half is not below r_coll is pruned (BHTree.cu:663-665;
// the same float operations, without contraction).  A chain of single-child
// cells shares one centre of mass, so testing its smallest cell, the one the
// compressed octree keeps, decides the whole chain.  Cells below the tenth
// level (inside a bucket of equal keys) are not modelled.
__device__ bool ref_prunes(const float4* __restrict__ com, const int4* __restrict__ info,
                           float4 xi, int j, float r) {
  int node = 0;
  for (int depth = 0; depth < 64; ++depth) {
    const int4 inf = __ldg(info + node);
    const int nch = inf.z & 15;
    if (nch == 0) return false;  // a leaf: the reference tests the bodies themselves
    const float4 c = __ldg(com + node);
    const float dx = c.x - xi.x, dy = c.y - xi.y, dz = c.z - xi.z;
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    const float half = __int_as_float(inf.w);
    if (!(__fsub_rn(sqrtf(d2), __fmul_rn(half, 1.732f)) < r)) return true;
    int next = -1;
    for (int k = 0; k < nch; ++k) {
      const int4 ci = __ldg(info + inf.x + k);
      if (j >= ci.y && j < ci.y + (ci.z >> 4)) {
        next = inf.x + k;
        break;
      }
    }
    if (next < 0) return false;
    node = next;
  }
  return false;
}

struct FofOut {
  const uint32_t* ids;
  float ll2;
  int* parent;
};

// ---------------------------------------------------- the search by cells
// When the radius is below half the side of a level-10 cell, the bodies
// within it lie in at most two cells along each axis.  The sorted keys are
// the index of those cells: a body's own cell is the run of equal keys around
// it, another is found by a binary search.  One thread a body (a warp together
// where cells hold many), no tree: at the full-physics radius (0.4% of a cell)
// nearly every body looks at its own cell alone.  Which of the two searches a disk takes is decided on the
// device, from its root cube, by each kernel for itself; the tree search
// leaves the disks the cells served (by_cells in geom.cuh).
//
// The pairs are the tree search's: every pair that passes the FP32 test is
// within reach on each axis, with the margin for float positions an ulp off
// the FP64 ones the keys were made from (as the records' boxes have it), and
// the quantisation is monotone, so the partner's cell is among those searched.
__device__ __forceinline__ uint32_t cell_of(double p, double lo, double scale) {
  const double q = fmin(fmax((p - lo) * scale, 0.0), 1023.0);
  return (uint32_t)q;
}

template <typename K>
__device__ __forceinline__ int first_key(const K* __restrict__ keys, int lo, int hi, K target) {
  while (lo < hi) {  // first index in [lo, hi) with a key of at least target
    const int mid = lo + ((hi - lo) >> 1);
    if (__ldg(keys + mid) < target) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Bodies of a cell that a thread looks at by itself, on each side of its own
// body or from another cell's first on; the warp goes through the rest of a
// longer run together (search_rest).  A collision pass over 524,288 bodies, a
// far body stretching the cube 1 / 4 / 10 / 40 times, with 16 / 32 / 64 and
// without a limit: 123 / 123 / 122 / 123, 144 / 142 / 131 / 130, 178 / 180 /
// 188 / 202 and 442 / 450 / 455 / 1060 us.
constexpr int kOwnRun = 64;

// A body and what its search finds.
template <int kMode>  // 0: collision impulse, 1: FoF links
struct CellTarget {
  float4 me;
  int s;
  bool have_v;  // velocities are read with the first pair
  float vx, vy, vz;
  float dvx, dvy, dvz;

  __device__ __forceinline__ CellTarget(float4 body, int slot)
      : me(body), s(slot), have_v(false), vx(0.f), vy(0.f), vz(0.f), dvx(0.f), dvy(0.f),
        dvz(0.f) {}

  __device__ __forceinline__ bool near(const float4 q, const CollideOut& co,
                                       const FofOut& fo) const {
    if (kMode == 0) return coll_dist2(q.x - me.x, q.y - me.y, q.z - me.z) < co.rc2;
    const float dx = __fsub_rn(me.x, q.x), dy = __fsub_rn(me.y, q.y), dz = __fsub_rn(me.z, q.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)) <
           fo.ll2;
  }

  __device__ __forceinline__ void pair(const float4 q, int j, const CollideOut& co,
                                       const FofOut& fo, int* status) {
    if (!near(q, co, fo)) return;
    if (kMode == 1) {
      uf_union(fo.parent, (int)fo.ids[s], (int)fo.ids[j], status);
      return;
    }
    if (!have_v) {
      const uint32_t vi = co.vmap ? co.vmap[s] : (uint32_t)s;
      vx = coll_vel(co.vx, co.vtype, vi);
      vy = coll_vel(co.vy, co.vtype, vi);
      vz = coll_vel(co.vz, co.vtype, vi);
      have_v = true;
    }
    const float dx = q.x - me.x, dy = q.y - me.y, dz = q.z - me.z;
    const uint32_t vj = co.vmap ? co.vmap[j] : (uint32_t)j;
    coll_impulse(dx, dy, dz, coll_dist2(dx, dy, dz), coll_vel(co.vx, co.vtype, vj) - vx,
                 coll_vel(co.vy, co.vtype, vj) - vy, coll_vel(co.vz, co.vtype, vj) - vz, co.e,
                 dvx, dvy, dvz);
  }
};

// The cells within reach of a body (the own one among them).
struct CellsAround {
  uint32_t c[3][2];
  __device__ __forceinline__ CellsAround(const TreeGeom& g, const float4 me, float radius) {
    const float p[3] = {me.x, me.y, me.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double r = (double)cell_reach(p[k], radius);
      c[k][0] = cell_of((double)p[k] - r, g.lo[k], g.scale);
      c[k][1] = cell_of((double)p[k] + r, g.lo[k], g.scale);
    }
  }
  __device__ __forceinline__ bool several() const {
    return c[0][0] != c[0][1] || c[1][0] != c[1][1] || c[2][0] != c[2][1];
  }
  // Whether cell q of the eight is to be searched, and its key.  Links look at
  // later bodies alone: each pair once.
  template <int kMode, typename K>
  __device__ __forceinline__ bool other(int q, K key, K& cell) const {
    if ((q & 1) && c[0][0] == c[0][1]) return false;
    if ((q & 2) && c[1][0] == c[1][1]) return false;
    if ((q & 4) && c[2][0] == c[2][1]) return false;
    cell = (key >> 30 << 30) | (K)morton30(c[0][q & 1], c[1][(q >> 1) & 1], c[2][q >> 2]);
    return cell != key && !(kMode == 1 && cell < key);
  }
};

// First body of another cell (of the next key there is, if it is empty).
template <typename K>
__device__ __forceinline__ int first_of(const K* __restrict__ keys, int n, int s, K key, K cell) {
  return cell > key ? first_key<K>(keys, s + 1, n, cell) : first_key<K>(keys, 0, s, cell);
}

// What the lanes of a warp left of their runs.  Lanes in one run read its
// bodies together, 32 at a time through shared memory, and test four of them
// before they branch.  A body far off stretches the root cube until a few
// cells hold the disk; a thread on its own then waits for a key and a body of
// global memory at each pair (a collision pass over 30,011 bodies, all but one
// in one cell: 6.2 ms each for itself, 1.1 ms this way, 2.1 ms through the
// tree).
template <typename K, int kMode>
__device__ __forceinline__ void search_rest(const NeighborArgs& a, const K* __restrict__ keys,
                                         float radius, const CollideOut& co, const FofOut& fo,
                                         bool mine, K key, CellTarget<kMode>& t, float4* sm) {
  const int lane = threadIdx.x & 31;
  const CellsAround around(a.geom[sizeof(K) == 8 ? (int)(key >> 30) : 0], t.me, radius);
  for (int q = kMode == 0 ? -2 : -1; q < 8; ++q) {
    int b0 = 0, b1 = 0;  // the rest of the lane's run (empty: b0 >= b1)
    if (mine && q == -2) {
      b0 = first_key<K>(keys, 0, t.s, key);
      b1 = t.s - kOwnRun;
    } else if (mine) {
      K cell = key;
      if (q < 0 || around.template other<kMode>(q, key, cell)) {
        b0 = (q < 0 ? t.s + 1 : first_of<K>(keys, a.n, t.s, key, cell)) + kOwnRun;
        if (b0 < a.n && __ldg(keys + b0) == cell) b1 = first_key<K>(keys, b0, a.n, cell + 1);
      }
    }
    unsigned todo = __ballot_sync(kFull, b0 < b1);
    while (todo) {
      const int from = __ffs(todo) - 1;
      const int l0 = __shfl_sync(kFull, b0, from), l1 = __shfl_sync(kFull, b1, from);
      const bool in = b0 < b1 && b0 < l1 && b1 > l0;  // meets that lane's
      const int lo = __reduce_min_sync(kFull, in ? b0 : l0);
      const int hi = __reduce_max_sync(kFull, in ? b1 : l1);
      float4 next = __ldg(a.body + min(lo + lane, hi - 1));
      for (int j0 = lo; j0 < hi; j0 += 32) {
        sm[lane] = next;
        __syncwarp();
        next = __ldg(a.body + min(j0 + 32 + lane, hi - 1));
        const int k0 = in ? max(b0 - j0, 0) : 32, k1 = min(b1 - j0, 32);
#pragma unroll 2
        for (int k = 0; k < 32; k += 4) {
          unsigned hit = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (t.near(sm[k + i], co, fo) && k + i >= k0 && k + i < k1) hit |= 1u << i;
          for (; hit; hit &= hit - 1) {
            const int i = k + __ffs(hit) - 1;
            t.pair(sm[i], j0 + i, co, fo, a.status);
          }
        }
        __syncwarp();
      }
      todo &= ~__ballot_sync(kFull, in);
    }
  }
}

// Five blocks per SM (48 registers): left to itself the compiler takes 32 for
// the links and spills (links at 2e-3 AU among 524,288 bodies: 334 against
// 318 us).
template <typename K, int kMode>
__global__ void __launch_bounds__(256, 5)
k_cell_neighbors(const NeighborArgs a, const K* __restrict__ keys, float radius, CollideOut co,
                 FofOut fo) {
  __shared__ float4 s_body[8][32];
  const int lane = threadIdx.x & 31;
  for (int base = blockIdx.x * blockDim.x + threadIdx.x - lane; base < a.n;
       base += gridDim.x * blockDim.x) {
    const int s = min(base + lane, a.n - 1);
    const K key = __ldg(keys + s);
    const TreeGeom& g = a.geom[sizeof(K) == 8 ? (int)(key >> 30) : 0];
    const bool mine = base + lane < a.n && by_cells(g, radius);
    CellTarget<kMode> t(__ldg(a.body + s), s);
    bool more = false;  // runs longer than kOwnRun
    if (mine) {
      const CellsAround around(g, t.me, radius);
      auto ahead = [&](int j, K cell) {  // bodies from j on in the cell
        const int stop = min(a.n, j + kOwnRun);
        for (; j < stop && __ldg(keys + j) == cell; ++j)
          t.pair(__ldg(a.body + j), j, co, fo, a.status);
        more |= j == stop;
      };
      if (kMode == 0) {
        int j = s - 1;
        const int stop = max(-1, j - kOwnRun);
        for (; j > stop && __ldg(keys + j) == key; --j)
          t.pair(__ldg(a.body + j), j, co, fo, a.status);
        more |= j == stop;
      }
      ahead(s + 1, key);
      if (around.several())
        for (int q = 0; q < 8; ++q) {
          K cell;
          if (around.template other<kMode>(q, key, cell))
            ahead(first_of<K>(keys, a.n, s, key, cell), cell);
        }
    }
    if (__any_sync(kFull, more)) {
      CellTarget<kMode> u = t;
      search_rest<K, kMode>(a, keys, radius, co, fo, mine, key, u, s_body[threadIdx.x >> 5]);
      t.dvx = u.dvx;
      t.dvy = u.dvy;
      t.dvz = u.dvz;
    }
    if (kMode == 0 && mine) {
      co.dvx[s] = t.dvx;
      co.dvy[s] = t.dvy;
      co.dvz[s] = t.dvz;
    }
  }
}

template <int kMode>
void launch_cell_neighbors(const NeighborArgs& a, float radius, const CollideOut& co,
                           const FofOut& fo, cudaStream_t s) {
  const int grid = std::min(div_up(a.n, 256), 148 * 16);
  if (a.keys)
    k_cell_neighbors<uint32_t, kMode><<<grid, 256, 0, s>>>(a, a.keys, radius, co, fo);
  else
    k_cell_neighbors<uint64_t, kMode><<<grid, 256, 0, s>>>(a, a.keys64, radius, co, fo);
  check(cudaGetLastError(), "k_cell_neighbors launch");
}

template <int kMode>  // 0: collision impulse, 1: FoF links, 2: collision pair report
__global__ void __launch_bounds__(kNbWarps * 32)
k_neighbors(const NeighborArgs a, float radius, CollideOut co, FofOut fo) {
  __shared__ NbSmem smem[kNbWarps];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  NbSmem& w = smem[wib];
  int* spill = a.spill + (size_t)(blockIdx.x * kNbWarps + wib) * (size_t)a.spill_cap;
  const int n_groups = *a.n_groups;
  // conservative per-axis reach: a pair that passes the FP32 test is closer
  // than radius (1 + 2^-20) on every axis
  const float reach = radius * 1.00001f + 1e-30f;
  const bool cells = kMode != 2 && (a.keys || a.keys64);
  if (cells) {  // nothing left for this search?
    bool mine = true;
    for (int d = threadIdx.x; d < a.n_disks; d += blockDim.x)
      mine = mine && by_cells(a.geom[d], radius);
    if (__syncthreads_and(mine)) return;
  }

  while (true) {
    int g = 0;
    if (lane == 0) g = atomicAdd(a.work, 1);
    g = __shfl_sync(kFull, g, 0);
    if (g >= n_groups) break;
    const int2 grp = a.groups[g];
    const int disk = a.group_disk ? a.group_disk[g] : 0;
    if (cells && by_cells(a.geom[disk], radius)) continue;
    // groups hold up to 64 bodies; search them 32 (one per lane) at a time
    for (int c0 = 0; c0 < grp.y; c0 += 32) {
    const int2 gr = make_int2(grp.x + c0, min(32, grp.y - c0));
    const int s = gr.x + lane;
    const bool valid = lane < gr.y;
    const float4 me = a.body[valid ? s : gr.x];
    const float gx0 = warp_min(me.x) - reach, gx1 = warp_max(me.x) + reach;
    const float gy0 = warp_min(me.y) - reach, gy1 = warp_max(me.y) + reach;
    const float gz0 = warp_min(me.z) - reach, gz1 = warp_max(me.z) + reach;

    float vix = 0.f, viy = 0.f, viz = 0.f;
    if (kMode == 0 && valid) {
      const uint32_t vi = co.vmap ? co.vmap[s] : (uint32_t)s;
      vix = coll_vel(co.vx, co.vtype, vi);
      viy = coll_vel(co.vy, co.vtype, vi);
      viz = coll_vel(co.vz, co.vtype, vi);
    }
    float dvx = 0.f, dvy = 0.f, dvz = 0.f;
    unsigned long long npairs = 0, nmissed = 0;
    const int my_id = (kMode == 1 && valid) ? (int)fo.ids[s] : 0;

    int top = 1, spilled = 0;
    bool overflow = false;
    if (lane == 0) w.stk[0] = disk;  // root slot of the group's disk
    __syncwarp();
    while (true) {
      if (top == 0) {
        if (spilled == 0) break;
        const int cnt = min(spilled, kStk / 2);
        for (int k = lane; k < cnt; k += 32) w.stk[k] = __ldcg(spill + (spilled - cnt) + k);
        spilled -= cnt;
        top = cnt;
        __syncwarp();
      }
      const int take = min(top, 32);
      top -= take;
      const int node = (lane < take) ? w.stk[top + lane] : -1;
      __syncwarp();
      int act = 0, first = 0, cnt = 0;
      if (node >= 0) {
        const float4 lo = __ldg(a.box_lo + node), hi = __ldg(a.box_hi + node);
        const bool overlap = lo.x <= gx1 && hi.x >= gx0 && lo.y <= gy1 && hi.y >= gy0 &&
                             lo.z <= gz1 && hi.z >= gz0;
        if (overlap) {
          const int4 inf = __ldg(a.info + node);
          cnt = inf.z >> 4;
          const int nch = inf.z & 15;
          if (nch == 0 || cnt <= a.leaf_max) {
            act = 2;
            first = inf.y;
          } else {
            act = 3;
            first = inf.x;
            cnt = nch;
          }
        }
      }
      const int pc = (act == 3) ? cnt : 0;
      const int pincl = warp_incl_scan(pc, lane);
      const int ptotal = __shfl_sync(kFull, pincl, 31);
      if (ptotal > 0) {
        if (top + ptotal > kStk) {
          if (spilled + top > a.spill_cap) { overflow = true; break; }
          for (int k = lane; k < top; k += 32) __stcg(spill + spilled + k, w.stk[k]);
          spilled += top;
          top = 0;
          __syncwarp();
        }
        const int base = top + pincl - pc;
        for (int k = 0; k < pc; ++k) w.stk[base + k] = first + k;
        top += ptotal;
        __syncwarp();
      }
      const int bc = (act == 2) ? cnt : 0;
      const int bincl = warp_incl_scan(bc, lane);
      const int btotal = __shfl_sync(kFull, bincl, 31);
      if (btotal == 0) continue;
      w.sc[lane] = bincl;
      w.slo[lane] = first;
      __syncwarp();
      for (int base = 0; base < btotal; base += 32) {
        const int gi = base + lane;
        if (gi < btotal) {
          int o = 0;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (w.sc[o + step - 1] <= gi) o += step;
          const int prev = (o > 0) ? w.sc[o - 1] : 0;
          const int j = w.slo[o] + (gi - prev);
          w.pos[lane] = __ldg(a.body + j);
          w.idx[lane] = j;
        }
        const int chunk = min(32, btotal - base);
        __syncwarp();
        if (valid) {
          for (int k = 0; k < chunk; ++k) {
            const float4 q = w.pos[k];
            const int j = w.idx[k];
            if (kMode == 0) {
              // BHTree.cu:642-660 (leaf branch), j != i
              const float dx = q.x - me.x, dy = q.y - me.y, dz = q.z - me.z;
              const float dist2 = coll_dist2(dx, dy, dz);
              if (j != s && dist2 < co.rc2) {
                const uint32_t vj = co.vmap ? co.vmap[j] : (uint32_t)j;
                coll_impulse(dx, dy, dz, dist2, coll_vel(co.vx, co.vtype, vj) - vix,
                             coll_vel(co.vy, co.vtype, vj) - viy,
                             coll_vel(co.vz, co.vtype, vj) - viz, co.e, dvx, dvy, dvz);
              }
            } else if (kMode == 2) {
              const float dx = q.x - me.x, dy = q.y - me.y, dz = q.z - me.z;
              if (j != s && coll_dist2(dx, dy, dz) < co.rc2) {
                ++npairs;
                if (ref_prunes(co.com, a.info, me, j, radius)) ++nmissed;
              }
            } else if (j > s) {
              // Aggregate.cpp:38-40, no FMA contraction
              float dx = __fsub_rn(me.x, q.x), dy = __fsub_rn(me.y, q.y),
                    dz = __fsub_rn(me.z, q.z);
              float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)),
                                   __fmul_rn(dz, dz));
              if (d2 < fo.ll2) uf_union(fo.parent, my_id, (int)fo.ids[j], a.status);
            }
          }
        }
        __syncwarp();
      }
    }
    if (kMode == 0 && valid) {
      co.dvx[s] = dvx;
      co.dvy[s] = dvy;
      co.dvz[s] = dvz;
    }
    if (kMode == 2) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        npairs += __shfl_xor_sync(kFull, npairs, o);
        nmissed += __shfl_xor_sync(kFull, nmissed, o);
      }
      if (lane == 0 && npairs) atomicAdd(co.report, npairs);
      if (lane == 0 && nmissed) atomicAdd(co.report + 1, nmissed);
    }
    if (lane == 0 && overflow) atomicOr(a.status, kStatusStackOverflow);
    }  // chunks of the group
  }
}

__global__ void k_fof_init(int* parent, int n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    parent[i] = (int)i;
}

__global__ void k_fof_labels(int* parent, int n, int* labels, int* sizes, int* status) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int r = uf_find(parent, (int)i);
    if (r < 0) { atomicOr(status, kStatusUnionFindLimit); r = (int)i; }
    labels[i] = r;
    atomicAdd(sizes + r, 1);
  }
}

__global__ void k_fof_sizes(const int* labels, const int* sizes, int n, uint16_t* agg_size,
                            int* n_groups) {
  int local = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int c = sizes[labels[i]];
    agg_size[i] = (uint16_t)(c >= 2 ? (c < 65535 ? c : 65535) : 1);
    if (labels[i] == (int)i && c >= 2) ++local;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(kFull, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(n_groups, local);
}

int g_nb_blocks_per_sm[3] = {0, 0, 0};

template <int kMode>
int nb_blocks_per_sm() {
  int& b = g_nb_blocks_per_sm[kMode];
  if (b == 0) {
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_neighbors<kMode>, kNbWarps * 32, 0),
          "neighbors occupancy");
    if (b < 1) b = 1;
  }
  return b;
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  }
  return sms;
}

template <int kMode>
int launch_nb(const NeighborArgs& a, float radius, const CollideOut& co, const FofOut& fo,
              cudaStream_t s) {
  if (a.n <= 0) return 0;
  const int groups = a.n;  // upper bound on the group count
  int grid = sm_count() * nb_blocks_per_sm<kMode>();
  // the spill area is sized for the walk's slot count; never exceed it
  grid = std::min(grid, walk_spill_slots(0) / kNbWarps);
  grid = std::min(grid, (groups + kNbWarps - 1) / kNbWarps);
  if (grid < 1) grid = 1;
  int launches = 1;
  if constexpr (kMode != 2)
    if (a.keys || a.keys64) {
      launch_cell_neighbors<kMode>(a, radius, co, fo, s);
      launches = 2;
    }
  check(cudaMemsetAsync(a.work, 0, sizeof(int), s), "neighbors work reset");
  k_neighbors<kMode><<<grid, kNbWarps * 32, 0, s>>>(a, radius, co, fo);
  check(cudaGetLastError(), "k_neighbors launch");
  return launches;
}

}  // namespace

int launch_collide_v(const NeighborArgs& a, const void* vx, const void* vy, const void* vz,
                     int vtype, const uint32_t* vmap, float r_coll, float restitution,
                     float* dvx, float* dvy, float* dvz, cudaStream_t s) {
  CollideOut co{vx, vy, vz, vtype, vmap, r_coll * r_coll, restitution, dvx, dvy, dvz, nullptr,
                nullptr};
  FofOut fo{nullptr, 0.f, nullptr};
  return launch_nb<0>(a, r_coll, co, fo, s);
}

void launch_collide(const NeighborArgs& a, const float* vx, const float* vy, const float* vz,
                    const uint32_t* vmap, float r_coll, float restitution, float* dvx,
                    float* dvy, float* dvz, cudaStream_t s) {
  launch_collide_v(a, vx, vy, vz, 0, vmap, r_coll, restitution, dvx, dvy, dvz, s);
}

void launch_collision_report(const NeighborArgs& a, const float4* com, float r_coll,
                             unsigned long long* report, cudaStream_t s) {
  check(cudaMemsetAsync(report, 0, 2 * sizeof(unsigned long long), s), "report reset");
  CollideOut co{nullptr, nullptr, nullptr, 0, nullptr, r_coll * r_coll, 0.f,
                nullptr, nullptr, nullptr, com, report};
  FofOut fo{nullptr, 0.f, nullptr};
  launch_nb<2>(a, r_coll, co, fo, s);
}

void launch_fof_link(const NeighborArgs& a, const uint32_t* ids, float link_length, int* parent,
                     cudaStream_t s) {
  if (a.n <= 0) return;
  k_fof_init<<<div_up(a.n, 256), 256, 0, s>>>(parent, a.n);
  CollideOut co{nullptr, nullptr, nullptr, 0, nullptr, 0.f, 0.f, nullptr, nullptr, nullptr, nullptr, nullptr};
  const float ll2 = link_length * link_length;  // Aggregate.cpp:30
  FofOut fo{ids, ll2, parent};
  launch_nb<1>(a, link_length, co, fo, s);
}

void launch_fof_finish(int* parent, int n, int* labels, int* sizes, uint16_t* agg_size,
                       int* n_groups, int* status, cudaStream_t s) {
  if (n <= 0) return;
  check(cudaMemsetAsync(sizes, 0, sizeof(int) * (size_t)n, s), "fof sizes reset");
  check(cudaMemsetAsync(n_groups, 0, sizeof(int), s), "fof groups reset");
  const int g = std::min(div_up(n, 256), 148 * 16);
  k_fof_labels<<<g, 256, 0, s>>>(parent, n, labels, sizes, status);
  k_fof_sizes<<<g, 256, 0, s>>>(labels, sizes, n, agg_size, n_groups);
  check(cudaGetLastError(), "fof finish launch");
}

// FoF links with the warp count capped at max_warps, for a caller whose stack
// spill area holds max_warps slots of a.spill_cap entries (the allocation-free
// FoF entry point sizes its static area this way).
void launch_fof_link_capped(const NeighborArgs& a, const uint32_t* ids, float link_length,
                            int* parent, int max_warps, cudaStream_t s) {
  if (a.n <= 0) return;
  k_fof_init<<<div_up(a.n, 256), 256, 0, s>>>(parent, a.n);
  CollideOut co{nullptr, nullptr, nullptr, 0, nullptr, 0.f, 0.f, nullptr, nullptr, nullptr, nullptr, nullptr};
  const float ll2 = link_length * link_length;  // Aggregate.cpp:30
  FofOut fo{ids, ll2, parent};
  int grid = sm_count() * nb_blocks_per_sm<1>();
  grid = std::min(grid, max_warps / kNbWarps);
  grid = std::min(grid, (a.n + kNbWarps - 1) / kNbWarps);
  if (grid < 1) grid = 1;
  if (a.keys || a.keys64) launch_cell_neighbors<1>(a, link_length, co, fo, s);
  check(cudaMemsetAsync(a.work, 0, sizeof(int), s), "neighbors work reset");
  k_neighbors<1><<<grid, kNbWarps * 32, 0, s>>>(a, link_length, co, fo);
  check(cudaGetLastError(), "k_neighbors launch");
}

}  // namespace nb
