// walk.cu -- warp-cooperative Barnes-Hut force walk (FP32 SIMT).
//
// Replaces bhtree_forceKernel (BHTree.cu:530-598; one thread per body, a
// 256-entry local-memory stack) and fuses perturber_forceKernel
// (Perturber.cu:13-35) into its epilogue.
//
// A warp owns a group of 32 targets that are consecutive in Morton order.
// Traversal is shared: the warp pops up to 32 nodes from a per-warp stack in
// shared memory and each lane tests one node against the group's bounding
// box.  A node is accepted when half^2 < theta^2 d^2 with d the distance from
// the group box to the node's centre of mass: every target in the group is
// at least d away, so each target's own reference test half/|x - com| <
// theta (BHTree.cu:577) would accept it too.  A node the box rejects is
// still accepted when every target's own test accepts it (a warp vote).
// Accepted nodes (and single bodies) are appended to a shared-memory source
// list; nodes that must be opened either push their contiguous children or,
// when they hold at most leaf_max bodies, append those bodies.  Each full batch of 32 sources is
// evaluated by all 32 lanes for their own target, reading four sources at a
// time from shared memory as broadcasts and computing in packed FP32
// (f32x2): 6 packed instructions + 1 MUFU.RSQ per interaction.  The softened
// self term is exactly zero (d = 0), so no self-skip test is needed when
// softening > 0.
//
// The stack spills to a per-warp global area when it would overflow; a
// spill area that runs out raises kStatusStackOverflow instead of hanging.
#include "collide_math.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "walk_math.cuh"

namespace nb {
namespace {

constexpr int kWalkWarps = 4;
// What a second warp of a walk's block does (k_walk): there is none; it sums
// the sources and writes them to the tape; it sums them.
enum SecondWarp { kNone = 0, kTape = 1, kSums = 2 };
// Vote walks of up to kBlockWalk2 bodies whose sums keep the list's order
// (WalkArgs::list_order): two warps to a group, 16 blocks per SM (one warp /
// two: N = 4096 31 / 28 us, 20,000 48 / 42, 70,000 66 / 62; from 95,000 on one
// warp is faster, 57 / 67).
constexpr int kSumBlocks = 16;
// Recording walks: blocks of one group (two warps) per SM, up to 80 registers
// (20,011 / 65,536 bodies, a gradient of 20 levels: 4027 / 5773 us, with 16
// blocks 4101 / 5865, with 18 4292 / 5853).
constexpr int kRecBlocks = 12;
// Walk modes (WalkArgs::walk_mode), a trade-off that depends on the disk:
//   0: acceptance vote, 5 resident blocks per SM (up to 96 registers);
//   1: acceptance vote, 8 blocks per SM (64 registers) -- the default: at
//      N = 2^20 over r in [0.3, 30] AU (groups of span 8) the step takes
//      0.641 ms, against 0.667 ms with mode 0 and 0.645 / 0.652 ms with 7 / 6
//      blocks per SM;
//   2: no vote, 8 blocks per SM -- the fastest on small compact disks (the
//      64-disk ensemble), where the vote rarely pays and occupancy matters.
template <int kRec, int kMode>
constexpr int walk_min_blocks() {
  return kRec == kSums ? kSumBlocks : kRec == kTape ? kRecBlocks : kMode == 0 ? 5 : 8;
}
template <int kRec>
constexpr int walk_threads() { return kRec ? 64 : kWalkWarps * 32; }
template <int kMode>
constexpr bool walk_vote() { return kMode != 2; }
constexpr int kStk = 384;
// Other vote walks (modes 0 and 1, which differ in their register budget alone)
// of up to this many bodies run k_walk_block with four, then two warps a group.
// A disk has a group for every 22 bodies, for the GPU's 4,736 warp slots.  While
// they do not fill those, the heaviest group's chain is what ends the walk; it
// depends on where the walls of the cells fall, so the times fall and rise with
// N, and no count that the host has tells it.  The lines lie where neither of
// two disks loses more than a tenth (us with one / two / four warps a group; r
// in [0.5, 5] AU, and in [0.3, 30]): N = 20,000 48.2 / 32.3 / 28.2 (55 / 35 /
// 29), 24,000 54 / 36.6 / 31.2 (60 / 39 / 32), 28,000 44.5 / 30.6 / 34.6 (50 /
// 36 / 39), 65,536 49.5 / 46.6 / 59.8 (78 / 59 / 66), 90,000 75.9 / 68.0 / 83
// (74 / 65 / 82), 95,000 56.6 / 62.1 (76 / 69: here the wide disk would do
// better with two warps), 100,003 51.6 / 61.9 (56 / 66).
constexpr int kBlockWalk4 = 25600;
constexpr int kBlockWalk2 = 92160;
constexpr int kList = 64;

// A batch of a recording walk's source list, with each source's sorted body
// range.
struct RecBatch {
  float lsrc[4][32];
  int2 lent[32];
};

template <int kRec>
struct WarpSmem {
  // source list, one row per component (x, y, z, mass): four consecutive
  // sources of a row are one 16-byte broadcast holding two register pairs
  float lsrc[4][kRec ? 4 : kList];
  int lidx[kRec ? 1 : kList];  // fused collisions: body index of each single-body source, else -1
  float4 ext[6];  // the group's targets of least / greatest x, y, z (vote prefilter)
  int stk[kStk];
  int slo[32];    // opened leaves: first body less the bodies of those before it
  // recording walks: the list as a ring of batches -- one being evaluated, two
  // being filled -- and what each published batch is: (sources, group, is its
  // first, is its last)
  static constexpr bool kTaped = kRec == kTape;
  RecBatch rec[kRec ? 4 : 1];
  int4 what[kRec ? 2 : 1];
};

// Squared distance in one fixed rounding, so that the vote and its
// prefilter test a target identically.
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
  return fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
}

// Drops the first 32 entries of the list (and of their body indices with
// fused collisions): each lane moves one 16-byte piece of one row; the entries
// past the list's end that move with them are never read.
template <bool kColl>
__device__ __forceinline__ void list_shift(WarpSmem<0>& w, int lane) {
  const int row = lane >> 3, q = (lane & 7) * 4;
  const float4 t = lst_row4(w, row, 32 + q);
  int b = -1;
  if (kColl) b = w.lidx[32 + lane];
  __syncwarp();
  *reinterpret_cast<float4*>(&w.lsrc[row][q]) = t;
  if (kColl) w.lidx[lane] = b;
  __syncwarp();
}

// Fused collisions: a lane's target (index, half-step velocity) and its
// accumulated impulse.
struct CollLane {
  int self;
  float vx, vy, vz;
  float dvx, dvy, dvz;
};

// Collision sweep of a batch 0 .. cnt of the list: every single-body source
// closer than r_coll to the lane's target adds its impulse (coll_dist2 and
// coll_impulse, as the stand-alone neighbour search).
__device__ __forceinline__ void coll_batch(const WalkArgs& a, const WarpSmem<0>& w, int cnt,
                                           const float4 me, bool valid, float rc2,
                                           CollLane& cl) {
  for (int j = 0; j < cnt; ++j) {
    const int b = w.lidx[j];
    if (b < 0) continue;
    const float4 s = lst_get(w, j);
    const float dx = s.x - me.x, dy = s.y - me.y, dz = s.z - me.z;
    const float d2 = coll_dist2(dx, dy, dz);
    if (valid && b != cl.self && d2 < rc2)
      coll_impulse(dx, dy, dz, d2, coll_vel(a.coll_v[0], a.coll_vtype, b) - cl.vx,
                   coll_vel(a.coll_v[1], a.coll_vtype, b) - cl.vy,
                   coll_vel(a.coll_v[2], a.coll_vtype, b) - cl.vz, a.coll_e, cl.dvx, cl.dvy,
                   cl.dvz);
  }
}

// Tape of a group's source list (recording walks): the sources, in the order
// the walk evaluates them, as sorted body ranges (first, count) in chunks of
// 32 from a pool -- a node's centre of mass is recomputed from its range on
// replay, a count of 1 is the body itself.  A group's chunks are chained;
// each also has its owner (group, its number in the chain) -- (-1, 0) when it
// holds nothing -- so that a pass over the chunks needs no chains.  A pool
// that runs dry raises kStatusTapeFull and the group is not recorded (forces
// are still computed).  The first lane takes the next chunk while the current
// batch is evaluated.
struct TapeCursor {
  int head = -1, cur = -1;
  bool ok = true;
};

__device__ __forceinline__ int tape_take(const WalkArgs& a, TapeCursor& t) {
  if (!t.ok) return -1;
  const int c = atomicAdd(a.tape_used, 1);
  if (c < 0 || c >= a.tape_cap) {
    atomicOr(a.status, kStatusTapeFull);
    t.ok = false;
    return -1;
  }
  if (t.cur >= 0) a.tape_next[t.cur] = c;
  else t.head = c;
  t.cur = c;
  return c;
}

// Writes chunk `index` of group g, k sources of `ent`, as chunk c of the pool.
__device__ __forceinline__ void tape_write(const WalkArgs& a, int c, int g, int index,
                                           const int2* ent, int k, int lane) {
  if (c < 0) return;
  if (lane < k) a.tape[(size_t)c * 32 + lane] = ent[lane];
  if (lane == 0) a.tape_owner[c] = k > 0 ? make_int2(g, index) : make_int2(-1, 0);
}

// Squared distance from a box to a point (0 inside) and to the box's
// farthest corner, in one fixed rounding shared by the walk and the span
// walk: both are monotone in the box bounds, so a box inside another is
// never nearer in FP32 either.
__device__ __forceinline__ float box_d2(float4 c, float x0, float x1, float y0, float y1,
                                        float z0, float z1) {
  const float dx = fmaxf(fmaxf(x0 - c.x, c.x - x1), 0.f);
  const float dy = fmaxf(fmaxf(y0 - c.y, c.y - y1), 0.f);
  const float dz = fmaxf(fmaxf(z0 - c.z, c.z - z1), 0.f);
  return dist2(dx, dy, dz);
}

__device__ __forceinline__ float box_far2(float4 c, float x0, float x1, float y0, float y1,
                                          float z0, float z1) {
  const float fx = fmaxf(fabsf(c.x - x0), fabsf(c.x - x1));
  const float fy = fmaxf(fabsf(c.y - y0), fabsf(c.y - y1));
  const float fz = fmaxf(fabsf(c.z - z0), fabsf(c.z - z1));
  return dist2(fx, fy, fz);
}

// Span-walk list entries: a node index, with kSpanLeafFlag for "the bodies
// of this leaf" (shared list only).
constexpr int kSpanLeafFlag = 1 << 30;
constexpr int kSpanNodeMask = kSpanLeafFlag - 1;

// A chain of 32-entry chunks of ints taken from a pool (the span walk's
// lists): entries fill each chunk before the next is taken.
struct Chain {
  int head = -1, cur = -1, count = 0;
  bool ok = true;
};

// Appends k <= 32 entries; lane l with `on` writes entry e at offset o.  A
// pool that runs dry marks the chain as failed.
__device__ __forceinline__ void chain_append(const SpanArgs& a, Chain& t, bool on, int o, int k,
                                             int e, int lane) {
  if (k <= 0 || !t.ok) return;
  const int used = t.count & 31;
  int c1 = t.cur, c2 = -1;
  if (lane == 0) {
    if (used == 0) {
      c1 = atomicAdd(a.used, 1);
      if (c1 >= a.cap) c1 = -1;
      if (c1 >= 0) {
        if (t.cur >= 0) a.next[t.cur] = c1;
        else t.head = c1;
      }
    }
    if (c1 >= 0 && used + k > 32) {
      c2 = atomicAdd(a.used, 1);
      if (c2 >= a.cap) c2 = -1;
      if (c2 >= 0) a.next[c1] = c2;
    }
  }
  c1 = __shfl_sync(kFull, c1, 0);
  c2 = __shfl_sync(kFull, c2, 0);
  t.head = __shfl_sync(kFull, t.head, 0);
  if (c1 < 0 || (used + k > 32 && c2 < 0)) {
    t.ok = false;
    return;
  }
  if (on) {
    const int q = used + o;
    a.pool[(size_t)((q < 32) ? c1 : c2) * 32 + (q & 31)] = e;
  }
  t.count += k;
  t.cur = (used + k > 32) ? c2 : c1;
}

// The span walk (the shared walk's first traversal): one warp per span node,
// the maximal tree node of <= span x 32 bodies that target groups were cut
// from.  It traverses the tree with the span's bounding box B_S -- the union
// of its groups' boxes -- and files each node it meets by what every group
// of the span would do with it:
//  - a single body, or a node that B_S accepts (half^2 < theta^2 d^2, d from
//    B_S to the centre of mass): every group box lies inside B_S, so is at
//    least as far, and accepts it too -> a shared source;
//  - a node that fails even against B_S's farthest corner (half^2 >= theta^2
//    far^2): every group box, and every target in it, is nearer, so no box
//    test and no acceptance vote can accept it and every group opens it ->
//    its children are traversed here, a leaf's bodies become shared sources;
//  - anything else -> the span's frontier, decided group by group.
// box_d2 and box_far2 are monotone in the box bounds in FP32 too, so the
// shared decisions are exactly the groups' own.  A group's walk evaluates the
// shared sources and starts from the frontier instead of the root: each
// target gets the interactions of a walk from the root, in another order.
// Children that would overflow the stack go to the frontier (deferring a node
// is always exact); a pool that runs dry leaves the span without lists, and
// its groups walk from the root.
__global__ void __launch_bounds__(kWalkWarps * 32) k_span_walk(const SpanArgs a) {
  __shared__ int s_stk[kWalkWarps][kStk];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int* stk = s_stk[wib];
  const int n_groups = *a.n_groups;
  while (true) {
    int g = 0;
    if (lane == 0) g = atomicAdd(a.work, 1);
    g = __shfl_sync(kFull, g, 0);
    if (g >= n_groups) break;
    const int2 sp = __ldg(a.group_span + g);
    if (sp.x != g) continue;  // not the first group of its span
    const int lo = __ldg(a.groups + g).x;
    float x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY, z0 = INFINITY,
          z1 = -INFINITY;
    for (int i = lane; i < sp.y; i += 32) {
      const float4 b = __ldg(a.body + lo + i);
      x0 = fminf(x0, b.x); x1 = fmaxf(x1, b.x);
      y0 = fminf(y0, b.y); y1 = fmaxf(y1, b.y);
      z0 = fminf(z0, b.z); z1 = fmaxf(z1, b.z);
    }
    x0 = warp_min(x0); x1 = warp_max(x1);
    y0 = warp_min(y0); y1 = warp_max(y1);
    z0 = warp_min(z0); z1 = warp_max(z1);
    Chain sh, fr;
    int top = 1;
    if (lane == 0) stk[0] = 0;  // the root
    __syncwarp();
    while (top > 0) {
      const int take = min(top, 32);
      top -= take;
      const int node = (lane < take) ? stk[top + lane] : -1;
      __syncwarp();
      int cls = 0, first = 0, nch = 0;  // 1 shared node, 2 shared leaf, 3 open, 4 frontier
      if (node >= 0) {
        const float4 c = __ldg(a.com + node);
        const int4 inf = __ldg(a.info + node);
        const int cnt = inf.z >> 4;
        nch = inf.z & 15;
        first = inf.x;
        const float half = __int_as_float(inf.w);
        const float h2 = half * half;
        if (cnt == 1 || h2 < a.theta2 * box_d2(c, x0, x1, y0, y1, z0, z1)) cls = 1;
        else if (!(h2 < a.theta2 * box_far2(c, x0, x1, y0, y1, z0, z1)))
          cls = (nch == 0 || cnt <= a.leaf_max) ? 2 : 3;
        else cls = 4;
      }
      unsigned m = __ballot_sync(kFull, cls == 1 || cls == 2);
      chain_append(a, sh, cls == 1 || cls == 2, __popc(m & lanemask_lt()), __popc(m),
                   node | (cls == 2 ? kSpanLeafFlag : 0), lane);
      m = __ballot_sync(kFull, cls == 4);
      chain_append(a, fr, cls == 4, __popc(m & lanemask_lt()), __popc(m), node, lane);
      const int pc = (cls == 3) ? nch : 0;
      const int pincl = warp_incl_scan(pc, lane);
      const int ptotal = __shfl_sync(kFull, pincl, 31);
      if (ptotal > 0) {
        if (top + ptotal <= kStk) {
          const int base = top + pincl - pc;
          for (int k = 0; k < pc; ++k) stk[base + k] = first + k;
          top += ptotal;
        } else {  // no room: the children are decided group by group
          for (int k = 0; k < 8; ++k) {
            const bool on = k < pc;
            const unsigned mk = __ballot_sync(kFull, on);
            chain_append(a, fr, on, __popc(mk & lanemask_lt()), __popc(mk), first + k, lane);
          }
        }
      }
      __syncwarp();
    }
    if (lane == 0) {
      const bool ok = sh.ok && fr.ok;
      if (ok && sh.cur >= 0) a.next[sh.cur] = -1;
      if (ok && fr.cur >= 0) a.next[fr.cur] = -1;
      a.span_lists[g] = ok ? make_int4(sh.head, sh.count, fr.head, fr.count)
                           : make_int4(-1, -1, -1, -1);
      if (a.counters) {
        atomicAdd(a.counters + 0, (unsigned long long)(ok ? sh.count : 0));
        atomicAdd(a.counters + 1, (unsigned long long)(ok ? fr.count : 0));
        atomicAdd(a.counters + 2, ok ? 1ull : 0ull);
      }
    }
  }
}

// Starts a group's stack: the children of its disk's root when the box test
// rejects it and no target can accept it either (not even against the box's
// farthest corner), else the root itself.  It spares the walk a round with one
// node in 32 lanes, of the twelve or so that a group takes (1.5% of the walk
// at N = 2^20 and 2^22; k_walk_block, whose rounds are longer chains, gained
// nothing and starts from the root).  Returns the nodes on the stack.
__device__ __forceinline__ int open_root(const WalkArgs& a, int root, float x0, float x1,
                                         float y0, float y1, float z0, float z1, int* stk,
                                         int lane) {
  const float4 c = __ldg(a.com + root);
  const int4 inf = __ldg(a.info + root);
  const float half = __int_as_float(inf.w), h2 = half * half;
  const int nch = inf.z & 15;
  if (nch > 0 && (inf.z >> 4) > a.leaf_max &&
      !(h2 < a.theta2 * box_d2(c, x0, x1, y0, y1, z0, z1)) &&
      !(h2 < a.theta2 * box_far2(c, x0, x1, y0, y1, z0, z1))) {
    if (lane < nch) stk[lane] = inf.x + lane;
    return nch;
  }
  if (lane == 0) stk[0] = root;
  return 1;
}

// The star's and the perturber's pull, added to a target's tree sum.
__device__ __forceinline__ void add_central(const WalkArgs& a, const float4 me, const float4 p,
                                            float& ax, float& ay, float& az) {
  if (a.star_in_walk) {  // softened star term, BHTree.cu:547-553
    float dx = -me.x, dy = -me.y, dz = -me.z;
    float r2 = dx * dx + dy * dy + dz * dz + a.eps * a.eps;
    float r = sqrtf(r2);
    float f = a.star_mass / (r2 * r);
    ax += f * dx; ay += f * dy; az += f * dz;
  }
  if (a.pert) {  // perturber_forceKernel, Perturber.cu:20-34 (adds)
    float dx = p.x - me.x, dy = p.y - me.y, dz = p.z - me.z;
    float r2 = dx * dx + dy * dy + dz * dz + a.eps * a.eps;
    float r = sqrtf(r2);
    float f = p.w / (r2 * r);
    ax += f * dx; ay += f * dy; az += f * dz;
  }
}

// Entry `pos` of the list that starts with batch `batch`.
template <typename W>
__device__ __forceinline__ void rec_put(W& w, unsigned batch, int pos,
                                        const float4 c, int2 range) {
  RecBatch& r = w.rec[(batch + (pos >> 5)) & 3];
  lst_put(r, pos & 31, c);
  if (W::kTaped) r.lent[pos & 31] = range;
}

__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

// Hands the batch over (k sources; -1: no more groups) and goes on to the next.
template <typename W>
__device__ __forceinline__ void rec_publish(W& w, unsigned& batch, int k, int g,
                                            bool first, bool last, int lane) {
  if (lane == 0) w.what[batch & 1] = make_int4(k, g, first, last);
  __syncwarp();
  pair_sync();
  ++batch;
}

// Recording walks: two warps to a group, for one group's chain is what bounds
// them at the sizes a gradient is taken of (twelve rounds of loads, votes and
// scans, and the sums, which a tape needs in list order).  One warp walks the
// tree and files the sources; this one adds up each batch of 32 and writes it
// to the tape.  One barrier a batch hands it over: whoever passes it has done
// with the batch before, and the first warp goes on filling the ring, into the
// next group too, while the second works.  Lists, chunks and sums are those of
// one warp doing both in turn.  A gradient of 20 levels (us), one warp / two:
// 4096 bodies 3150 / 3000, 20,011 4300 / 4030, 65,536 5930 / 5770, 131,072
// 8400 / 8280, 400,000 19,400 / 19,100; at 10^6 they are even.  Plain walks
// whose sums keep their order run it without a tape (kSums).
template <bool kSoft, bool kTaped, typename W>
__device__ __forceinline__ void record_batches(const WalkArgs& a, W& w, int lane) {
  const float eps2 = a.eps * a.eps;
  const float2 e2 = make_float2(eps2, eps2);
  int2 gr = make_int2(0, 0);
  float4 me[1] = {};
  PairAcc acc[1] = {};
  PairTgt pt[1] = {};
  TapeCursor tc;
  int tape_at = -1, evaluated = 0;
  for (int k = 0;; ++k) {
    pair_sync();
    const int4 b = w.what[k & 1];
    if (b.x < 0) return;  // no more groups
    const int g = b.y;
    if (b.z) {
      gr = a.groups[g];
      me[0] = a.body[lane < gr.y ? gr.x + lane : gr.x];
      acc[0].x = acc[0].y = acc[0].z = make_float2(0.f, 0.f);
      pt[0].x = make_float2(-me[0].x, -me[0].x);
      pt[0].y = make_float2(-me[0].y, -me[0].y);
      pt[0].z = make_float2(-me[0].z, -me[0].z);
      evaluated = 0;
      tc = TapeCursor();
      if (kTaped && lane == 0) tape_at = tape_take(a, tc);  // the chunk of the next batch
    }
    const RecBatch& r = w.rec[k & 3];
    if (kTaped)
      tape_write(a, __shfl_sync(kFull, tape_at, 0), g, evaluated / 32, r.lent, b.x, lane);
    evaluated += b.x;
    if (!b.w) {
      if (kTaped && lane == 0) tape_at = tape_take(a, tc);
      eval_list<kSoft, 1, 32, false, kTaped>(r, 32, me, pt, eps2, e2, acc);
      continue;
    }
    eval_list<kSoft, 1, 0, false, kTaped>(r, b.x, me, pt, eps2, e2, acc);
    // summed in the .x halves alone, in list order
    float ax = kTaped ? acc[0].x.x : acc[0].x.x + acc[0].x.y;
    float ay = kTaped ? acc[0].y.x : acc[0].y.x + acc[0].y.y;
    float az = kTaped ? acc[0].z.x : acc[0].z.x + acc[0].z.y;
    const int disk = a.group_disk ? a.group_disk[g] : 0;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.pert) p = a.pert[(a.pert_step ? *a.pert_step * a.n_disks : 0) + disk];
    add_central(a, me[0], p, ax, ay, az);
    if (lane < gr.y) {
      const int s = gr.x + lane;
      const uint32_t o = a.scatter ? a.scatter[s] : (uint32_t)s;
      a.ax[o] = ax;
      a.ay[o] = ay;
      a.az[o] = az;
    }
    if (kTaped && lane == 0) a.group_tape[g] = tc.ok ? make_int2(tc.head, evaluated) : make_int2(-1, 0);
  }
}

// kT targets per lane: a group of up to 32 kT bodies per warp.  kRec (kT == 1):
// a SecondWarp evaluates the group's source list, and with kTape records it (a
// block walks one group).  kColl (kT == 1): fused
// collisions.  A multi-body node whose box comes within r_coll of the group
// box is opened even when the opening test would accept it, so every body
// that can touch a target reaches the source list as a single body; each
// evaluated batch whose least distance is inside r_coll is then swept for
// collision pairs.  The pairs are those of the stand-alone search: the same
// squared distance and impulse arithmetic (collide_math.cuh); only the order
// in which a target's impulses are summed differs.
template <bool kSoft, int kT, int kRec, int kMode, bool kColl = false, bool kSpan = false>
__global__ void __launch_bounds__(walk_threads<kRec>(), walk_min_blocks<kRec, kMode>())
    k_walk(const WalkArgs a) {
  constexpr int kWalkers = kRec ? 1 : kWalkWarps;
  __shared__ __align__(16) WarpSmem<kRec> smem[kWalkers];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if constexpr (kRec != 0) {
    if (wib == 1) {
      record_batches<kSoft, kRec == kTape>(a, smem[0], lane);
      return;
    }
  }
  WarpSmem<kRec>& w = smem[wib];
  int* spill = a.spill + (size_t)(blockIdx.x * kWalkers + wib) * (size_t)a.spill_cap;
  unsigned batch = 0;  // recording: batches published
  const int n_groups = *a.n_groups;
  const float eps2 = a.eps * a.eps;

  while (true) {
    int g = 0;
    if (lane == 0) g = atomicAdd(a.work, 1);
    g = __shfl_sync(kFull, g, 0);
    if (g >= n_groups) break;
    const int2 gr = a.groups[g];
    const int disk = a.group_disk ? a.group_disk[g] : 0;
    float4 me[kT];
    bool valid[kT];
    float gx0 = INFINITY, gx1 = -INFINITY, gy0 = INFINITY, gy1 = -INFINITY, gz0 = INFINITY,
          gz1 = -INFINITY;
#pragma unroll
    for (int t = 0; t < kT; ++t) {
      valid[t] = lane + 32 * t < gr.y;
      me[t] = a.body[valid[t] ? gr.x + lane + 32 * t : gr.x];
      gx0 = fminf(gx0, me[t].x); gx1 = fmaxf(gx1, me[t].x);
      gy0 = fminf(gy0, me[t].y); gy1 = fmaxf(gy1, me[t].y);
      gz0 = fminf(gz0, me[t].z); gz1 = fmaxf(gz1, me[t].z);
    }
    gx0 = warp_min(gx0); gx1 = warp_max(gx1);
    gy0 = warp_min(gy0); gy1 = warp_max(gy1);
    gz0 = warp_min(gz0); gz1 = warp_max(gz1);
    if (walk_vote<kMode>()) {
      // a target that attains each extreme (invalid lanes hold target 0)
      const float ev[6] = {gx0, gx1, gy0, gy1, gz0, gz1};
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        int ts = -1;
#pragma unroll
        for (int t = kT - 1; t >= 0; --t) {
          const float cv = (e < 2) ? me[t].x : (e < 4) ? me[t].y : me[t].z;
          if (cv == ev[e]) ts = t;
        }
        const unsigned m = __ballot_sync(kFull, ts >= 0);
        if (m == 0u) {  // non-finite positions: a point that rejects nothing
          if (lane == 0) w.ext[e] = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
        } else if (lane == __ffs(m) - 1) {
          w.ext[e] = (ts <= 0) ? me[0] : me[kT - 1];
        }
      }
      __syncwarp();
    }
    CollLane cl{-1, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float rc2 = 0.f, reach = 0.f, rthr = 0.f;
    if (kColl) {
      const int s0 = valid[0] ? gr.x + lane : gr.x;
      cl.self = valid[0] ? s0 : -1;
      cl.vx = coll_vel(a.coll_v[0], a.coll_vtype, s0);
      cl.vy = coll_vel(a.coll_v[1], a.coll_vtype, s0);
      cl.vz = coll_vel(a.coll_v[2], a.coll_vtype, s0);
      rc2 = a.coll_r * a.coll_r;
      reach = a.coll_r * 1.00001f + 1e-30f;  // a pair inside r_coll is inside this on each axis
      // softened squared distances carry eps^2 and a few roundings: a batch
      // whose least one is above this holds no pair inside r_coll
      rthr = (rc2 + eps2) * 1.00002f + 1e-37f;
    }

    // The tree sum starts from zero: adding ~10^3 terms into an accumulator
    // that already holds the star pull (10^3-10^5 times larger) would round
    // every term at the star's ulp.  Star and perturber are added at the end.
    PairAcc acc[kT];
    PairTgt pt[kT];
#pragma unroll
    for (int t = 0; t < kT; ++t) {
      acc[t].x = acc[t].y = acc[t].z = make_float2(0.f, 0.f);
      pt[t].x = make_float2(-me[t].x, -me[t].x);
      pt[t].y = make_float2(-me[t].y, -me[t].y);
      pt[t].z = make_float2(-me[t].z, -me[t].z);
    }
    const float2 e2 = make_float2(eps2, eps2);
    unsigned long long visited = 0, spills = 0, evaluated = 0;
    int top = 1, spilled = 0, nlist = 0;
    bool overflow = false;
    // shared walk: the span's shared sources first (decided by the span
    // walk), then its frontier in place of the root
    int sh_chunk = -1, sh_left = 0, fr_chunk = -1, fr_left = 0;
    if (kSpan) {
      const int4 sl = __ldg(a.span_lists + __ldg(a.group_span + g).x);
      if (sl.y >= 0) {
        sh_chunk = sl.x; sh_left = sl.y;
        fr_chunk = sl.z; fr_left = sl.w;
        top = 0;
      }
    }
    if (top == 1) {
      top = open_root(a, disk, gx0, gx1, gy0, gy1, gz0, gz1, w.stk, lane);
      visited += top > 1 ? 1 : 0;
    }
    __syncwarp();

    while (true) {
      int node = -1, forced = 0;  // forced: 1 source, 2 bodies of a leaf (shared list)
      if (kSpan && sh_left > 0) {
        const int k = min(sh_left, 32);
        const int e = (lane < k) ? __ldg(a.span_pool + (size_t)sh_chunk * 32 + lane) : -1;
        sh_left -= k;
        if (sh_left > 0) sh_chunk = __ldg(a.span_next + sh_chunk);
        node = (e >= 0) ? (e & kSpanNodeMask) : -1;
        forced = (e >= 0) ? ((e & kSpanLeafFlag) ? 2 : 1) : 0;
        visited += k;
      } else {
        if (top == 0) {
          if (spilled == 0) {
            if (!kSpan || fr_left == 0) break;
            const int k = min(fr_left, 32);
            if (lane < k) w.stk[lane] = __ldg(a.span_pool + (size_t)fr_chunk * 32 + lane);
            fr_left -= k;
            if (fr_left > 0) fr_chunk = __ldg(a.span_next + fr_chunk);
            top = k;
          } else {
            const int cnt = min(spilled, kStk / 2);
            for (int k = lane; k < cnt; k += 32) w.stk[k] = __ldcg(spill + (spilled - cnt) + k);
            spilled -= cnt;
            top = cnt;
          }
          __syncwarp();
        }
        const int take = min(top, 32);
        top -= take;
        visited += take;
        node = (lane < take) ? w.stk[top + lane] : -1;
        __syncwarp();
      }

      int act = 0;  // 1: source, 2: bodies of a leaf, 3: open children
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      int first = 0, cnt = 0;
      float h2 = 0.f, d2 = 0.f, far2 = 0.f;
      int4 ninf = make_int4(0, 0, 0, 0);
      if (node >= 0) {
        c = __ldg(a.com + node);
        const int4 inf = __ldg(a.info + node);
        ninf = inf;
        cnt = inf.z >> 4;
        const int nch = inf.z & 15;
        const float half = __int_as_float(inf.w);
        h2 = half * half;
        if (forced == 1 || cnt == 1) {
          act = 1;
        } else if (forced == 2) {
          act = 2;
          first = inf.y;
        } else {
          d2 = box_d2(c, gx0, gx1, gy0, gy1, gz0, gz1);
          // farthest point of the box: no target is farther than this
          if (walk_vote<kMode>()) far2 = box_far2(c, gx0, gx1, gy0, gy1, gz0, gz1);
          if (h2 < a.theta2 * d2) {
            act = 1;
          } else if (nch == 0 || cnt <= a.leaf_max) {
            act = 2;
            first = inf.y;
          } else {
            act = 3;
            first = inf.x;
            cnt = nch;
          }
        }
      }

      // Second chance for the nodes the group box rejects: the box test uses
      // the box's nearest point, a lower bound on every target's distance.
      // Such a node is still accepted when each target's own reference test
      // (half < theta |x_i - com|, BHTree.cu:577) accepts it -- one vote per
      // candidate, all lanes testing their own targets.  At N = 2^20 this
      // opens 11% fewer interactions and makes the walk 25% faster, at
      // unchanged force error.  Two candidates are put to the vote at a time:
      // one at a time is a chain of some 250 cycles each, and the groups
      // whose boxes are large for their surroundings (a few hundred votes
      // against 23 on average) are what the walk ends on at 130,000 to
      // 500,000 bodies (N = 262,144: 158 -> 147 us; 2^20 and 2^22: 0.5%).
      // Candidates in shared memory, one 16-byte broadcast for the four
      // shuffles, were 2% slower at 2^22.
      if (walk_vote<kMode>()) {
        // Necessary conditions first: the far corner, then the extreme
        // target on the node's side along each axis must accept it.
        bool cnd = act >= 2 && d2 > 0.f && h2 < a.theta2 * far2;
        if (cnd) {
          const float4 ex = w.ext[c.x > 0.5f * (gx0 + gx1) ? 1 : 0];
          cnd = h2 < a.theta2 * dist2(c.x - ex.x, c.y - ex.y, c.z - ex.z);
        }
        if (cnd) {
          const float4 ey = w.ext[c.y > 0.5f * (gy0 + gy1) ? 3 : 2];
          cnd = h2 < a.theta2 * dist2(c.x - ey.x, c.y - ey.y, c.z - ey.z);
        }
        if (cnd) {
          const float4 ez = w.ext[c.z > 0.5f * (gz0 + gz1) ? 5 : 4];
          cnd = h2 < a.theta2 * dist2(c.x - ez.x, c.y - ez.y, c.z - ez.z);
        }
        unsigned cand = __ballot_sync(kFull, cnd);
        while (cand) {
          const int j = __ffs(cand) - 1;
          cand &= cand - 1;
          const int k = cand ? __ffs(cand) - 1 : j;
          cand &= cand - 1;
          const float cx = __shfl_sync(kFull, c.x, j), cy = __shfl_sync(kFull, c.y, j);
          const float cz = __shfl_sync(kFull, c.z, j), hh = __shfl_sync(kFull, h2, j);
          const float ex = __shfl_sync(kFull, c.x, k), ey = __shfl_sync(kFull, c.y, k);
          const float ez = __shfl_sync(kFull, c.z, k), eh = __shfl_sync(kFull, h2, k);
          bool ok = true, ek = true;
#pragma unroll
          for (int t = 0; t < kT; ++t) {
            ok = ok && (!valid[t] || hh < a.theta2 * dist2(cx - me[t].x, cy - me[t].y,
                                                           cz - me[t].z));
            ek = ek && (!valid[t] || eh < a.theta2 * dist2(ex - me[t].x, ey - me[t].y,
                                                           ez - me[t].z));
          }
          const bool aj = __all_sync(kFull, ok), ak = __all_sync(kFull, ek);
          if ((aj && lane == j) || (ak && lane == k)) act = 1;
        }
      }
      if (kColl) {  // an accepted node within reach of the group stays open
        const int cntb = ninf.z >> 4;
        if (act == 1 && cntb > 1) {
          const float4 lo = __ldg(a.box_lo + node), hi = __ldg(a.box_hi + node);
          if (lo.x <= gx1 + reach && hi.x >= gx0 - reach && lo.y <= gy1 + reach &&
              hi.y >= gy0 - reach && lo.z <= gz1 + reach && hi.z >= gz0 - reach) {
            const int nch = ninf.z & 15;
            if (nch == 0 || cntb <= a.leaf_max) {
              act = 2;
              first = ninf.y;
              cnt = cntb;
            } else {
              act = 3;
              first = ninf.x;
              cnt = nch;
            }
          }
        }
      }
      // accepted sources -> list
      const unsigned m1 = __ballot_sync(kFull, act == 1);
      if (act == 1) {
        const int pos = nlist + __popc(m1 & lanemask_lt());
        if constexpr (kRec != 0) rec_put(w, batch, pos, c, make_int2(ninf.y, ninf.z >> 4));
        else lst_put(w, pos, c);
        if (kColl) w.lidx[pos] = ((ninf.z >> 4) == 1) ? ninf.y : -1;
      }
      nlist += __popc(m1);
      __syncwarp();
      if (nlist >= 32) {
        if constexpr (kRec != 0) {
          rec_publish(w, batch, 32, g, evaluated == 0, false, lane);
        } else {
          const float rmin = eval_list<kSoft, kT, 32, kColl>(w, 32, me, pt, eps2, e2, acc);
          if constexpr (kColl)
            if (__any_sync(kFull, rmin < rthr))
              coll_batch(a, w, 32, me[0], valid[0], rc2, cl);
          list_shift<kColl>(w, lane);
        }
        evaluated += 32;
        nlist -= 32;
      }

      // Opened nodes -> children on the stack, leaves -> their bodies into
      // the list.  One scan counts both: children (<= 8 a lane, <= 256 a
      // pop) in the top 9 bits, bodies in the low 23; a leaf of >= 2^18
      // bodies (that many on one key) takes a scan of its own.
      const int pc = (act == 3) ? cnt : 0;
      const int bc = (act == 2) ? cnt : 0;
      int pincl, bincl, ptotal, btotal;
      if (__any_sync(kFull, bc >= (1 << 18))) {
        pincl = warp_incl_scan(pc, lane);
        bincl = warp_incl_scan(bc, lane);
        ptotal = __shfl_sync(kFull, pincl, 31);
        btotal = __shfl_sync(kFull, bincl, 31);
      } else {
        const unsigned incl = warp_incl_scan(((unsigned)pc << 23) | (unsigned)bc, lane);
        const unsigned tot = __shfl_sync(kFull, incl, 31);
        pincl = (int)(incl >> 23);
        bincl = (int)(incl & 0x7fffffu);
        ptotal = (int)(tot >> 23);
        btotal = (int)(tot & 0x7fffffu);
      }
      if (ptotal > 0) {
        if (top + ptotal > kStk) {
          if (spilled + top > a.spill_cap) { overflow = true; break; }
          ++spills;
          for (int k = lane; k < top; k += 32) __stcg(spill + spilled + k, w.stk[k]);
          spilled += top;
          top = 0;
          __syncwarp();
        }
        const int base = top + pincl - pc;
#pragma unroll
        for (int k = 0; k < 8; ++k)  // a node has at most 8 children
          if (k < pc) w.stk[base + k] = first + k;
        top += ptotal;
        __syncwarp();
      }

      // leaves to open -> their bodies into the list, 32 at a time: a lane
      // finds its leaf by counting the starts up to its own place (N = 2^22,
      // 24 batches a group: 2573 -> 2503 us against a search of the scan)
      if (btotal > 0) {
        // the leaves in order, each as its first body less the bodies before it
        const int start = bincl - bc;
        const unsigned leaves = __ballot_sync(kFull, bc > 0);
        if (bc > 0) w.slo[__popc(leaves & lanemask_lt())] = first - start;
        __syncwarp();
        for (int base = 0; base < btotal; base += 32) {
          const int gi = base + lane;
          const unsigned before = __ballot_sync(kFull, bc > 0 && start <= base);
          const unsigned starts = __reduce_or_sync(
              kFull, (bc > 0 && start > base && start < base + 32) ? 1u << (start - base) : 0u);
          if (gi < btotal) {
            const int o = __popc(before) - 1 + __popc(starts & (lanemask_lt() | (1u << lane)));
            const int b = w.slo[o] + gi;
            if constexpr (kRec != 0)
              rec_put(w, batch, nlist + lane, __ldg(a.body + b), make_int2(b, 1));
            else
              lst_put(w, nlist + lane, __ldg(a.body + b));
            if (kColl) w.lidx[nlist + lane] = b;
          }
          nlist += min(32, btotal - base);
          __syncwarp();
          if (nlist >= 32) {
            if constexpr (kRec != 0) {
              rec_publish(w, batch, 32, g, evaluated == 0, false, lane);
            } else {
              const float rmin = eval_list<kSoft, kT, 32, kColl>(w, 32, me, pt, eps2, e2, acc);
              if constexpr (kColl)
                if (__any_sync(kFull, rmin < rthr))
                  coll_batch(a, w, 32, me[0], valid[0], rc2, cl);
              list_shift<kColl>(w, lane);
            }
            evaluated += 32;
            nlist -= 32;
          }
        }
      }
    }

    if constexpr (kRec != 0) rec_publish(w, batch, nlist, g, evaluated == 0, true, lane);
    float rmin = 0.f;
    if constexpr (kRec == kNone)
      rmin = eval_list<kSoft, kT, 0, kColl>(w, nlist, me, pt, eps2, e2, acc);
    if constexpr (kColl) {
      if (__any_sync(kFull, rmin < rthr)) coll_batch(a, w, nlist, me[0], valid[0], rc2, cl);
      if (valid[0]) {
        const int s = gr.x + lane;
        a.coll_dv[0][s] = cl.dvx;
        a.coll_dv[1][s] = cl.dvy;
        a.coll_dv[2][s] = cl.dvz;
      }
    }
    evaluated += nlist;
    __syncwarp();

    if constexpr (kRec == kNone) {
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.pert) p = a.pert[(a.pert_step ? *a.pert_step * a.n_disks : 0) + disk];
#pragma unroll
      for (int t = 0; t < kT; ++t) {
        float ax = acc[t].x.x + acc[t].x.y;
        float ay = acc[t].y.x + acc[t].y.y;
        float az = acc[t].z.x + acc[t].z.y;
        add_central(a, me[t], p, ax, ay, az);
        if (valid[t]) {
          const int s = gr.x + lane + 32 * t;
          const uint32_t o = a.scatter ? a.scatter[s] : (uint32_t)s;
          a.ax[o] = ax;
          a.ay[o] = ay;
          a.az[o] = az;
        }
      }
    }
    if (lane == 0) {
      if (overflow) atomicOr(a.status, kStatusStackOverflow);
      atomicAdd(a.inter, evaluated * (unsigned long long)gr.y);
      if (a.counters) {
        atomicAdd(a.counters + 0, visited);
        atomicAdd(a.counters + 1, spills);
        atomicAdd(a.counters + 2, 1ull);
      }
    }
  }
  if constexpr (kRec != 0) rec_publish(w, batch, -1, 0, false, true, lane);
}

// The walk for disks too small to fill the GPU with one warp per group: a
// block of kW warps walks one group.  Every lane l of every warp holds target
// l.  The warps share one node stack and one source list; a round pops up to
// 32 kW nodes, dealt out one to each warp in turn, each warp tests and votes
// on its own nodes as k_walk does, and each evaluates 32 of every 32 kW
// sources, so a group's serial chain (node loads, votes, evaluation) is some
// kW times shorter.  The accepted nodes, opened leaves and counters are
// k_walk's; only the order in which a target's terms are summed differs (kW
// partial sums, added in the order of the warps; the same on every run).
// What bounds it is the heaviest group's chain, ten to twelve rounds of some
// 3000 cycles: at N = 4096 the walk takes 20 us against 31 with one warp a
// group, which ran its heaviest group for 53,000 cycles on an idle SM.
template <int kW>
struct BlockSmem {
  static constexpr int kBatch = 32 * kW;
  static constexpr int kRing = 4 * kBatch;  // a batch read while the next two are written
  static constexpr int kStkB = 12 * kBatch; // a round pushes up to 8 kBatch nodes
  float lsrc[4][kRing];
  float4 ext[kW][6];
  int stk[kStkB];
  int sc[kBatch];   // opened leaves: bodies up to each, within its warp
  int slo[kBatch];  // and their first bodies
  int3 tot[kW];     // a round's sources, children and bodies of each warp
  float part[kW][3][32];
  int group;
};

template <bool kSoft, int kW>
__global__ void __launch_bounds__(kW * 32, 32 / kW) k_walk_block(const WalkArgs a) {
  using Smem = BlockSmem<kW>;
  constexpr int kBatch = Smem::kBatch, kRing = Smem::kRing, kStkB = Smem::kStkB;
  __shared__ __align__(16) Smem w;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, tid = threadIdx.x;
  int* spill = a.spill + (size_t)blockIdx.x * kW * (size_t)a.spill_cap;
  const int spill_cap = kW * a.spill_cap;
  const int n_groups = *a.n_groups;
  const float eps2 = a.eps * a.eps;
  const float2 e2 = make_float2(eps2, eps2);
  int g = blockIdx.x;
  while (g < n_groups) {
    const int2 gr = a.groups[g];
    const bool valid = lane < gr.y;
    const float4 me = a.body[valid ? gr.x + lane : gr.x];
    const float gx0 = warp_min(me.x), gx1 = warp_max(me.x);
    const float gy0 = warp_min(me.y), gy1 = warp_max(me.y);
    const float gz0 = warp_min(me.z), gz1 = warp_max(me.z);
    const float ev[6] = {gx0, gx1, gy0, gy1, gz0, gz1};
#pragma unroll
    for (int e = 0; e < 6; ++e) {  // a target that attains each extreme
      const float cv = (e < 2) ? me.x : (e < 4) ? me.y : me.z;
      const unsigned m = __ballot_sync(kFull, cv == ev[e]);
      if (m == 0u) {  // non-finite positions: a point that rejects nothing
        if (lane == 0) w.ext[wib][e] = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
      } else if (lane == __ffs(m) - 1) {
        w.ext[wib][e] = me;
      }
    }
    PairAcc acc[1];
    PairTgt pt[1];
    acc[0].x = acc[0].y = acc[0].z = make_float2(0.f, 0.f);
    pt[0].x = make_float2(-me.x, -me.x);
    pt[0].y = make_float2(-me.y, -me.y);
    pt[0].z = make_float2(-me.z, -me.z);
    float rmin = 0.f;
    unsigned long long visited = 0, spills = 0, evaluated = 0;
    int top = 1, spilled = 0, head = 0, nlist = 0;
    bool overflow = false;
    auto eval_full = [&]() {  // the list's full batches, 32 sources a warp
      while (nlist >= kBatch) {
        const int at = (head + 32 * wib) & (kRing - 1);
#pragma unroll
        for (int j = 0; j < 32; j += 4) eval_quad<kSoft, 1, false>(w, at + j, pt, e2, acc, rmin);
        head = (head + kBatch) & (kRing - 1);
        nlist -= kBatch;
        evaluated += kBatch;
      }
    };
    if (tid == 0) w.stk[0] = a.group_disk ? a.group_disk[g] : 0;  // root slot of its disk
    __syncthreads();
    while (true) {
      if (top == 0) {
        if (spilled == 0) break;
        const int cnt = min(spilled, kStkB / 2);
        for (int k = tid; k < cnt; k += kBatch) w.stk[k] = __ldcg(spill + (spilled - cnt) + k);
        spilled -= cnt;
        top = cnt;
        __syncthreads();
      }
      const int take = min(top, kBatch);
      top -= take;
      visited += take;
      const int mine = lane * kW + wib;  // nodes dealt out to the warps in turn
      int act = 0;  // 1: source, 2: bodies of a leaf, 3: open children
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
      int first = 0, cnt = 0;
      float h2 = 0.f;
      bool cnd = false;
      int4 inf = make_int4(0, 0, 0, 0);
      if (mine < take) {
        const int node = w.stk[top + mine];
        c = __ldg(a.com + node);
        inf = __ldg(a.info + node);
      }
      // the list's full batches, while the nodes arrive
      eval_full();
      if (mine < take) {
        cnt = inf.z >> 4;
        const int nch = inf.z & 15;
        const float half = __int_as_float(inf.w);
        h2 = half * half;
        if (cnt == 1) {
          act = 1;
        } else {
          const float d2 = box_d2(c, gx0, gx1, gy0, gy1, gz0, gz1);
          if (h2 < a.theta2 * d2) {
            act = 1;
          } else {
            if (nch == 0 || cnt <= a.leaf_max) {
              act = 2;
              first = inf.y;
            } else {
              act = 3;
              first = inf.x;
              cnt = nch;
            }
            // the conditions of k_walk for a vote of the targets
            cnd = d2 > 0.f && h2 < a.theta2 * box_far2(c, gx0, gx1, gy0, gy1, gz0, gz1);
            if (cnd) {
              const float4 ex = w.ext[wib][c.x > 0.5f * (gx0 + gx1) ? 1 : 0];
              cnd = h2 < a.theta2 * dist2(c.x - ex.x, c.y - ex.y, c.z - ex.z);
            }
            if (cnd) {
              const float4 ey = w.ext[wib][c.y > 0.5f * (gy0 + gy1) ? 3 : 2];
              cnd = h2 < a.theta2 * dist2(c.x - ey.x, c.y - ey.y, c.z - ey.z);
            }
            if (cnd) {
              const float4 ez = w.ext[wib][c.z > 0.5f * (gz0 + gz1) ? 5 : 4];
              cnd = h2 < a.theta2 * dist2(c.x - ez.x, c.y - ez.y, c.z - ez.z);
            }
          }
        }
      }
      unsigned cand = __ballot_sync(kFull, cnd);
      while (cand) {
        const int j = __ffs(cand) - 1;
        cand &= cand - 1;
        const int k = cand ? __ffs(cand) - 1 : j;
        cand &= cand - 1;
        const float cx = __shfl_sync(kFull, c.x, j), cy = __shfl_sync(kFull, c.y, j);
        const float cz = __shfl_sync(kFull, c.z, j), hh = __shfl_sync(kFull, h2, j);
        const float ex = __shfl_sync(kFull, c.x, k), ey = __shfl_sync(kFull, c.y, k);
        const float ez = __shfl_sync(kFull, c.z, k), eh = __shfl_sync(kFull, h2, k);
        const bool aj = __all_sync(
            kFull, !valid || hh < a.theta2 * dist2(cx - me.x, cy - me.y, cz - me.z));
        const bool ak = __all_sync(
            kFull, !valid || eh < a.theta2 * dist2(ex - me.x, ey - me.y, ez - me.z));
        if ((aj && lane == j) || (ak && lane == k)) act = 1;
      }
      const unsigned m1 = __ballot_sync(kFull, act == 1);
      const int pc = (act == 3) ? cnt : 0, bc = (act == 2) ? cnt : 0;
      int pincl, bincl;  // one scan for both, as in k_walk
      if (__any_sync(kFull, bc >= (1 << 18))) {
        pincl = warp_incl_scan(pc, lane);
        bincl = warp_incl_scan(bc, lane);
      } else {
        const unsigned incl = warp_incl_scan(((unsigned)pc << 23) | (unsigned)bc, lane);
        pincl = (int)(incl >> 23);
        bincl = (int)(incl & 0x7fffffu);
      }
      w.sc[tid] = bincl;
      w.slo[tid] = first;
      if (lane == 31) w.tot[wib] = make_int3(__popc(m1), pincl, bincl);
      __syncthreads();  // every warp has read its nodes and counted
      int apre = 0, atotal = 0, ppre = 0, ptotal = 0, btotal = 0;
#pragma unroll
      for (int v = 0; v < kW; ++v) {
        const int3 t = w.tot[v];
        if (v < wib) {
          apre += t.x;
          ppre += t.y;
        }
        atotal += t.x;
        ptotal += t.y;
        btotal += t.z;
      }
      if (act == 1)
        lst_put(w, (head + nlist + apre + __popc(m1 & lanemask_lt())) & (kRing - 1), c);
      nlist += atotal;
      if (top + ptotal > kStkB) {
        if (spilled + top > spill_cap) { overflow = true; break; }
        ++spills;
        for (int k = tid; k < top; k += kBatch) __stcg(spill + spilled + k, w.stk[k]);
        spilled += top;
        top = 0;
        __syncthreads();
      }
      const int base = top + ppre + pincl - pc;
#pragma unroll
      for (int k = 0; k < 8; ++k)  // a node has at most 8 children
        if (k < pc) w.stk[base + k] = first + k;
      top += ptotal;
      // the opened leaves' bodies, a batch at a time
      int b0 = 0;
      while (true) {
        const int room = min(btotal - b0, kBatch);
        if (tid < room) {
          int q = b0 + tid, v = 0;
          while (q >= w.tot[v].z) q -= w.tot[v++].z;
          int o = 32 * v;
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (w.sc[o + step - 1] <= q) o += step;
          const int prev = (o & 31) ? w.sc[o - 1] : 0;
          lst_put(w, (head + nlist + tid) & (kRing - 1), __ldg(a.body + w.slo[o] + (q - prev)));
        }
        nlist += room;
        b0 += kBatch;
        __syncthreads();  // the batch is in the list, the children on the stack
        if (b0 >= btotal) break;
        eval_full();
      }
    }
    // the rest of the list, whole quads dealt out to the warps
    const int quads = (nlist + 3) / 4;
    for (int k = wib; k < quads; k += kW) {
      const int at = (head + 4 * k) & (kRing - 1);
      if (4 * k + 4 <= nlist) {
        eval_quad<kSoft, 1, false>(w, at, pt, e2, acc, rmin);
      } else {
        const float4 mv[1] = {me};
        for (int j = 4 * k; j < nlist; ++j)
          eval_one<kSoft, 1, false>(lst_get(w, (head + j) & (kRing - 1)), mv, eps2, acc, rmin);
      }
    }
    evaluated += nlist;
    w.part[wib][0][lane] = acc[0].x.x + acc[0].x.y;
    w.part[wib][1][lane] = acc[0].y.x + acc[0].y.y;
    w.part[wib][2][lane] = acc[0].z.x + acc[0].z.y;
    if (tid == 0) w.group = gridDim.x + atomicAdd(a.work, 1);
    __syncthreads();
    if (wib == 0) {
      float ax = 0.f, ay = 0.f, az = 0.f;
#pragma unroll
      for (int v = 0; v < kW; ++v) {
        ax += w.part[v][0][lane];
        ay += w.part[v][1][lane];
        az += w.part[v][2][lane];
      }
      const int disk = a.group_disk ? a.group_disk[g] : 0;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (a.pert) p = a.pert[(a.pert_step ? *a.pert_step * a.n_disks : 0) + disk];
      add_central(a, me, p, ax, ay, az);
      if (valid) {
        const int s = gr.x + lane;
        const uint32_t o = a.scatter ? a.scatter[s] : (uint32_t)s;
        a.ax[o] = ax;
        a.ay[o] = ay;
        a.az[o] = az;
      }
      if (lane == 0) {
        if (overflow) atomicOr(a.status, kStatusStackOverflow);
        atomicAdd(a.inter, evaluated * (unsigned long long)gr.y);
        if (a.counters) {
          atomicAdd(a.counters + 0, visited);
          atomicAdd(a.counters + 1, spills);
          atomicAdd(a.counters + 2, 1ull);
        }
      }
    }
    g = w.group;
    __syncthreads();  // before the next group's sums and stack
  }
}

template <bool kSoft, int kT, int kRec = kNone, int kMode = 0, bool kColl = false,
          bool kSpan = false>
int walk_blocks_per_sm() {
  static int b = 0;
  if (b == 0) {
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
              &b, k_walk<kSoft, kT, kRec, kMode, kColl, kSpan>, walk_threads<kRec>(), 0),
          "walk occupancy");
    if (b < 1) b = 1;
  }
  return b;
}

int num_sms() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  }
  return sms;
}

template <bool kSoft, int kT, int kRec = kNone, int kMode = 0, bool kColl = false,
          bool kSpan = false>
void launch_variant(const WalkArgs& a, cudaStream_t s) {
  int grid = num_sms() * walk_blocks_per_sm<kSoft, kT, kRec, kMode, kColl, kSpan>();
  const int walkers = kRec ? 1 : kWalkWarps;
  grid = std::min(grid, (a.n + walkers - 1) / walkers);  // groups <= n
  if (kRec) grid = std::min(grid, walk_spill_slots(0));
  if (grid < 1) grid = 1;
  k_walk<kSoft, kT, kRec, kMode, kColl, kSpan><<<grid, walk_threads<kRec>(), 0, s>>>(a);
}

template <bool kSoft, int kW>
void launch_block(const WalkArgs& a, cudaStream_t s) {
  // no more warps than the spill area holds slots for
  const int grid = std::min(num_sms() * (32 / kW), walk_spill_slots(0) / kW);
  k_walk_block<kSoft, kW><<<std::max(1, std::min(grid, a.n)), kW * 32, 0, s>>>(a);
}

template <bool kSoft, bool kColl, bool kSpan = false>
void launch_mode(const WalkArgs& a, cudaStream_t s) {
  if (a.walk_mode == 1) launch_variant<kSoft, 1, kNone, 1, kColl, kSpan>(a, s);
  else if (a.walk_mode == 2) launch_variant<kSoft, 1, kNone, 2, kColl, kSpan>(a, s);
  else launch_variant<kSoft, 1, kNone, 0, kColl, kSpan>(a, s);
}

template <bool kSoft>
int span_blocks_per_sm() {
  return std::max(std::max(walk_blocks_per_sm<kSoft, 1, kNone, 0, false, true>(),
                           walk_blocks_per_sm<kSoft, 1, kNone, 1, false, true>()),
                  walk_blocks_per_sm<kSoft, 1, kNone, 2, false, true>());
}

template <bool kSoft>
int coll_blocks_per_sm() {
  return std::max(std::max(walk_blocks_per_sm<kSoft, 1, kNone, 0, true>(),
                           walk_blocks_per_sm<kSoft, 1, kNone, 1, true>()),
                  walk_blocks_per_sm<kSoft, 1, kNone, 2, true>());
}

}  // namespace

int walk_spill_slots(int) {
  const int b = std::max(
      std::max(std::max(walk_blocks_per_sm<true, 1>(), walk_blocks_per_sm<false, 1>()),
               std::max(walk_blocks_per_sm<true, 2>(), walk_blocks_per_sm<false, 2>())),
      std::max((std::max(walk_blocks_per_sm<true, 1, kTape>(), walk_blocks_per_sm<false, 1, kTape>()) +
                kWalkWarps - 1) / kWalkWarps,
               std::max(std::max(walk_blocks_per_sm<true, 1, kNone, 1>(),
                                 walk_blocks_per_sm<false, 1, kNone, 1>()),
                        std::max(walk_blocks_per_sm<true, 1, kNone, 2>(),
                                 walk_blocks_per_sm<false, 1, kNone, 2>()))));
  const int bc = std::max(std::max(coll_blocks_per_sm<true>(), coll_blocks_per_sm<false>()),
                          std::max(span_blocks_per_sm<true>(), span_blocks_per_sm<false>()));
  return num_sms() * std::max(b, bc) * kWalkWarps;
}

// The span walk: its span counter and chunk count zeroed, then one warp per
// span (grid-strided over the groups).
__global__ void k_span_reset(int* work, int* used, unsigned long long* counters) {
  if (threadIdx.x == 0) *work = 0;
  if (threadIdx.x == 1) *used = 0;
  if (counters && threadIdx.x >= 2 && threadIdx.x < 5) counters[threadIdx.x - 2] = 0ull;
}

void launch_span_walk(const SpanArgs& a, int n, cudaStream_t s) {
  if (n <= 0) return;
  k_span_reset<<<1, 32, 0, s>>>(a.work, a.used, a.counters);
  static int blocks = 0;
  if (blocks == 0) {
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_span_walk, kWalkWarps * 32,
                                                        0),
          "span walk occupancy");
    blocks = std::max(blocks, 1);
  }
  int grid = num_sms() * blocks;
  grid = std::min(grid, (n + kWalkWarps - 1) / kWalkWarps);
  k_span_walk<<<std::max(grid, 1), kWalkWarps * 32, 0, s>>>(a);
  check(cudaGetLastError(), "k_span_walk launch");
}

// The walk's group counter and statistics, zeroed by one launch (three
// memset nodes in a step graph cost more than this).
// Recording walks also note where their chunks begin in the tape pool.
__global__ void k_walk_reset(int* work, unsigned long long* inter, unsigned long long* counters,
                             const int* tape_used, int* tape_begin) {
  const int t = threadIdx.x;
  if (t == 5 && tape_begin) *tape_begin = *tape_used;
  if (t == 0) *work = 0;
  if (t == 1 && inter) *inter = 0ull;
  if (t >= 2 && t < 5 && counters) counters[t - 2] = 0ull;
}

void launch_walk(const WalkArgs& a, cudaStream_t s) {
  if (a.n <= 0) return;
  if (!a.counters_zeroed) {
    k_walk_reset<<<1, 32, 0, s>>>(a.work, a.inter, a.counters, a.tape_used, a.tape_begin);
    check(cudaGetLastError(), "walk reset launch");
  }
  const bool soft = a.eps > 0.f;
  if (a.tape) {  // recording: groups of <= 32 targets
    if (soft) launch_variant<true, 1, kTape>(a, s);
    else launch_variant<false, 1, kTape>(a, s);
  } else if (a.targets_per_lane == 2) {
    if (soft) launch_variant<true, 2>(a, s);
    else launch_variant<false, 2>(a, s);
  } else if (a.coll_dv[0]) {  // fused collisions
    if (soft) launch_mode<true, true>(a, s);
    else launch_mode<false, true>(a, s);
  } else if (a.span_lists) {  // shared walk
    if (soft) launch_mode<true, false, true>(a, s);
    else launch_mode<false, false, true>(a, s);
  } else if (a.walk_mode != 2 && a.list_order && a.n <= kBlockWalk2) {
    if (soft) launch_variant<true, 1, kSums, 1>(a, s);
    else launch_variant<false, 1, kSums, 1>(a, s);
  } else if (a.walk_mode != 2 && !a.list_order && a.n <= kBlockWalk4) {
    if (soft) launch_block<true, 4>(a, s);
    else launch_block<false, 4>(a, s);
  } else if (a.walk_mode != 2 && !a.list_order && a.n <= kBlockWalk2) {
    if (soft) launch_block<true, 2>(a, s);
    else launch_block<false, 2>(a, s);
  } else {
    if (soft) launch_mode<true, false>(a, s);
    else launch_mode<false, false>(a, s);
  }
  check(cudaGetLastError(), "k_walk launch");
}

}  // namespace nb
