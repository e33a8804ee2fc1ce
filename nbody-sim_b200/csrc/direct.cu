// direct.cu -- FP64 direct-sum self-gravity: the accuracy yardstick of the
// tree walk and the pair potential of the softened energy.
//
// For each target i (a list, or every body):
//   a_i   =  sum_{j != i} m_j (x_j - x_i) / (|x_j - x_i|^2 + eps^2)^{3/2}
//   phi_i = -sum_{j != i} m_j / (|x_j - x_i|^2 + eps^2)^{1/2}
// in FP64.  The softened star term of src/physics/BHTree.cu:547-553 is not
// included: callers add it in FP64.
//
// FP64 arithmetic bounds it (about 22 FP64 instructions a pair, two cycles
// each a scheduler).  A warp holds 32 targets, one a lane, and a slice of the
// sources, which it reads 32 at a time into its own shared memory; the
// kDirWarps warps of a block take slices of one target set, and so do the
// blocks of a cluster, so that few targets still fill the GPU.  The partial
// sums are added in the order of the slices (through distributed shared
// memory across the cluster): results are the same on every run.  16,384
// targets of 2^20 bodies take 26.1 ms; one thread per target over all sources
// took 101 ms (64 blocks for 148 SMs).
#include <cooperative_groups.h>

#include <algorithm>

#include "capi_util.h"
#include "common.cuh"
#include "kernels.cuh"

namespace nb {
namespace {

constexpr int kDirWarps = 8;

template <bool kPhi>
__global__ void __launch_bounds__(kDirWarps * 32)
k_direct(const double* __restrict__ x, const double* __restrict__ y,
         const double* __restrict__ z, const float* __restrict__ m, int n,
         const int* __restrict__ targets, int nt, double eps2, double* __restrict__ ax,
         double* __restrict__ ay, double* __restrict__ az, double* __restrict__ phi) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int ranks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  __shared__ double4 src[kDirWarps][32];
  __shared__ double4 part[kDirWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = ((int)blockIdx.x / ranks) * 32 + lane;
  const bool live = t < nt;
  const int i = live ? (targets ? targets[t] : t) : -1;
  const double xi = live ? x[i] : 0.0, yi = live ? y[i] : 0.0, zi = live ? z[i] : 0.0;
  double sx = 0.0, sy = 0.0, sz = 0.0, sp = 0.0;
  // the warp's slice, whole batches of 32 sources
  const int slices = ranks * kDirWarps;
  const int batches = (n + 31) / 32, per = (batches + slices - 1) / slices;
  const int b0 = min((rank * kDirWarps + warp) * per, batches), b1 = min(b0 + per, batches);
  for (int b = b0; b < b1; ++b) {
    const int base = 32 * b, j = base + lane;
    __syncwarp();
    src[warp][lane] = (j < n) ? make_double4(x[j], y[j], z[j], (double)m[j])
                              : make_double4(0.0, 0.0, 0.0, 0.0);
    __syncwarp();
    const int cnt = min(32, n - base);
#pragma unroll 4
    for (int k = 0; k < cnt; ++k) {
      const double4 s = src[warp][k];
      const double dx = s.x - xi, dy = s.y - yi, dz = s.z - zi;
      const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
      const double inv = (base + k == i) ? 0.0 : rsqrt(r2);
      const double minv = s.w * inv;
      const double f = minv * inv * inv;
      sx = fma(f, dx, sx);
      sy = fma(f, dy, sy);
      sz = fma(f, dz, sz);
      if (kPhi) sp -= minv;
    }
  }
  part[warp][lane] = make_double4(sx, sy, sz, sp);
  cl.sync();
  if (rank == 0 && warp < 4 && live) {  // warp w adds component w over the slices
    double* out = warp == 0 ? ax : warp == 1 ? ay : warp == 2 ? az : phi;
    if (out) {
      double v = 0.0;
      for (int r = 0; r < ranks; ++r) {
        const double* p = (const double*)cl.map_shared_rank(&part[0][0], r);
        for (int w = 0; w < kDirWarps; ++w) v += p[4 * (32 * w + lane) + warp];
      }
      out[t] = v;
    }
  }
  cl.sync();  // the blocks' partial sums stay until they are read
}

// Blocks per target set: a power of two up to the portable cluster size that
// gives every SM some 24 blocks, so that the last wave of blocks is a small
// part (against 2^20 bodies with 1 / 2 / 8 blocks a set: 16,384 targets 32.2 /
// 26.4 / 26.1 ms, 512 targets 15.3 / 7.7 / 2.3 ms; 131,072 targets of as many
// bodies 24.9 / 24.6 / 25.4 ms), and each warp at least two batches.
int direct_cluster(int sets, int n) {
  int c = 1;
  while (c < 8 && (long long)sets * c < 148 * 24 && n >= 2 * 32 * kDirWarps * 2 * c) c *= 2;
  return c;
}

}  // namespace
}  // namespace nb

extern "C" int nbody_direct_f64(const double* x, const double* y, const double* z,
                                const float* mass, int n, const int* targets, int n_targets,
                                double eps, double* ax, double* ay, double* az, double* phi) {
  NBODY_API_BODY({
    NBODY_REQUIRE(x && y && z && mass, "nbody_direct_f64: null array");
    NBODY_REQUIRE(n >= 0, "nbody_direct_f64: negative n");
    const int nt = targets ? n_targets : n;
    NBODY_REQUIRE(nt >= 0, "nbody_direct_f64: negative target count");
    if (nt == 0 || n == 0) return NBODY_OK;
    const int sets = nb::div_up(nt, 32), c = nb::direct_cluster(sets, n);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(sets * c));
    cfg.blockDim = dim3(nb::kDirWarps * 32);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)c, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    nb::check(cudaLaunchKernelEx(&cfg, phi ? nb::k_direct<true> : nb::k_direct<false>, x, y, z,
                                 mass, n, targets, nt, eps * eps, ax, ay, az, phi),
              "k_direct launch");
    nb::check(cudaDeviceSynchronize(), "k_direct");
  })
}

namespace {
template <typename K>
int radix_sort_api(K* keys, uint32_t* values, int n, int bits, const char* what) {
  NBODY_API_BODY({
    NBODY_REQUIRE(n >= 0, std::string(what) + ": negative n");
    NBODY_REQUIRE(bits >= 1 && bits <= 8 * (int)sizeof(K), std::string(what) + ": bad bit count");
    if (n <= 1) return NBODY_OK;
    NBODY_REQUIRE(keys && values, std::string(what) + ": null array");
    K* ka = nullptr;
    uint32_t *va = nullptr, *counts = nullptr;
    int* status = nullptr;
    auto release = [&]() {
      cudaFree(ka);
      cudaFree(va);
      cudaFree(counts);
      cudaFree(status);
    };
    try {
      nb::check(cudaMalloc(&ka, sizeof(K) * (size_t)n), "sort scratch");
      nb::check(cudaMalloc(&va, sizeof(uint32_t) * (size_t)n), "sort scratch");
      nb::check(cudaMalloc(&counts, sizeof(uint32_t) * nb::radix_sort_count_words(n)),
                "sort scratch");
      nb::check(cudaMalloc(&status, sizeof(int)), "sort status");
      nb::check(cudaMemset(status, 0, sizeof(int)), "sort status");
      nb::radix_sort_pairs<K>(keys, values, ka, va, counts, n, bits, 0, status);
      int st = 0;
      nb::check(cudaMemcpy(&st, status, sizeof(int), cudaMemcpyDeviceToHost), "sort status");
      if (st) throw nb::CudaError(std::string(what) + ": a look-back wait gave up");
    } catch (...) {
      release();
      throw;
    }
    release();
  })
}
}  // namespace

extern "C" int nbody_radix_sort_u32(uint32_t* keys, uint32_t* values, int n, int bits) {
  return radix_sort_api<uint32_t>(keys, values, n, bits, "nbody_radix_sort_u32");
}

extern "C" int nbody_radix_sort_u64(uint64_t* keys, uint32_t* values, int n, int bits) {
  return radix_sort_api<uint64_t>(keys, values, n, bits, "nbody_radix_sort_u64");
}

extern "C" int nbody_radix_tree_u32(const uint32_t* keys, int n, int key_bits, int* left,
                                    int* right, int* lo, int* hi, uint8_t* prefix) {
  NBODY_API_BODY({
    NBODY_REQUIRE(n >= 0, "nbody_radix_tree_u32: negative n");
    NBODY_REQUIRE(key_bits >= 1 && key_bits <= 32, "nbody_radix_tree_u32: bad bit count");
    if (n < 2) return NBODY_OK;
    NBODY_REQUIRE(keys && left && right && lo && hi && prefix,
                  "nbody_radix_tree_u32: null array");
    nb::radix_tree_u32(keys, n, key_bits, left, right, lo, hi, prefix);
  })
}

extern "C" int nbody_selftest_sort_wait(int* status_bits) {
  NBODY_API_BODY({
    NBODY_REQUIRE(status_bits, "nbody_selftest_sort_wait: null argument");
    *status_bits = nb::sort_wait_selftest();
  })
}
