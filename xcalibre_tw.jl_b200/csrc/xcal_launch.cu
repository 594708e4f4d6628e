// Launch of the persistent device program (xcal_kernel.cu instantiations):
// block, cluster or cooperative grid launch, and the occupancy queries the
// launch configuration uses.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "xcal_device.cuh"
#include "xcal_kernel.h"

namespace xcal {

const void *program_kernel_d1();
const void *program_kernel_d2();
const void *program_kernel_d3();
const void *program_kernel_f2();
const void *program_kernel_f3();
const void *program_kernel_d2o();
const void *program_kernel_d3o();
const void *program_kernel_f2o();
const void *program_kernel_f3o();
const void *cg_kernel_cd(int W);
const void *cg_kernel_cf(int W);
const void *cgc_kernel_cd(int W);
const void *cgc_kernel_cf(int W);
const void *serve_kernel_d2o();
const void *serve_kernel_d3o();
const void *serve_kernel_f2o();
const void *serve_kernel_f3o();
// builds for numberings with sweeps by one CTA
const void *program_kernel_d1w();
const void *program_kernel_d2w();
const void *program_kernel_d3w();
const void *program_kernel_f2w();
const void *program_kernel_f3w();
const void *serve_kernel_d2ow();
const void *serve_kernel_d3ow();
const void *serve_kernel_f2ow();
const void *serve_kernel_f3ow();

// Dynamic shared memory of the matrix tiles (cg_two_level) per CTA: what fits
// beside the static part (5 KB) and the 1 KB the system keeps per CTA with 2
// (or 4) CTAs in the 227 KB of an SM.
static constexpr size_t RING_BYTES[2] = {96 * 1024, 48 * 1024};

static size_t ring_tile_bytes(int W, int mixed) { return (size_t)W * TILE * ((mixed ? 4 : 8) + sizeof(int)); }

// Matrix tiles per CTA that its dynamic shared memory holds: all of a CTA's
// tiles where they fit (the matrix then stays there for a whole solve), else 0.
int ring_tiles(int W, int mixed, int occ, int ntiles, int nblocks) {
  if (W < 1 || W > WUNROLL) return 0;
  const int cap = (int)(RING_BYTES[occ ? 1 : 0] / ring_tile_bytes(W, mixed));
  const int want = (ntiles + nblocks - 1) / std::max(nblocks, 1);
  return want <= cap ? want : 0;
}

int sweep_bytes(size_t bytes, int occ) { return (int)std::min(bytes, RING_BYTES[occ ? 1 : 0]); }

// Serving kernel of a dimension and precision (4-CTA/SM builds).
const void *serve_kernel_ptr(int ns, int mixed, int sweeps) {
  if (sweeps && ns == 2) return mixed ? serve_kernel_f2ow() : serve_kernel_d2ow();
  if (sweeps && ns == 3) return mixed ? serve_kernel_f3ow() : serve_kernel_d3ow();
  if (ns == 2) return mixed ? serve_kernel_f2o() : serve_kernel_d2o();
  if (ns == 3) return mixed ? serve_kernel_f3o() : serve_kernel_d3o();
  return nullptr;
}

// The attributes of a build that its launches need, set once per device:
// they are process-wide state, and a serving loop launches from many threads.
static cudaError_t allow_attribute(const void *fn, cudaFuncAttribute attr, int value) {
  static std::mutex mu;
  static std::map<std::tuple<const void *, int, int>, bool> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({fn, (int)attr, dev})) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, attr, value);
  if (e == cudaSuccess) done[{fn, (int)attr, dev}] = true;
  return e;
}
static cudaError_t allow_ring(const void *fn, int occ) {
  return allow_attribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RING_BYTES[occ ? 1 : 0]);
}

// Dynamic shared memory of a CTA of the serving launch: the matrix rows of a
// full CTA (quads, hexahedra) where they fit, else none, which leaves the L1 to
// rows read from global memory; the vector of the sweeps by one CTA.
// (16 cases of up to 160 tiles, 300 iterations, mean run of a case: mixed 696 ms
// streamed beside 48 KB, 625 resident; FP64, whose 4 tiles do not fit, 730
// beside 48 KB reserved for nothing, 650 with none.)
size_t serve_shared_bytes(int ns, int mixed, int sweeps, int tiles_per_cta) {
  if (sweeps) return RING_BYTES[1];
  const size_t rows = (size_t)tiles_per_cta * ring_tile_bytes(ns == 3 ? 7 : 5, mixed);
  return rows <= RING_BYTES[1] ? rows : 0;
}

// CTAs of the serving launch: every CTA that can be resident at once (a
// cooperative launch of this size is guaranteed co-resident).
int serve_grid(int ns, int mixed, int sweeps, size_t shared_bytes, int device) {
  const void *fn = serve_kernel_ptr(ns, mixed, sweeps);
  if (!fn) return 0;
  int per_sm = 0, sms = 0;
  if (allow_ring(fn, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, TPB, shared_bytes) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return per_sm * sms;
}

const void *program_kernel_ptr(int ns, int mixed, int occ) {
  if (ns == 1) return program_kernel_d1();
  if (ns == 2) {
    if (occ) return mixed ? program_kernel_f2o() : program_kernel_d2o();
    return mixed ? program_kernel_f2() : program_kernel_d2();
  }
  if (occ) return mixed ? program_kernel_f3o() : program_kernel_d3o();
  return mixed ? program_kernel_f3() : program_kernel_d3();
}

// The program for a numbering with sweeps by one CTA: 2 CTAs per SM.
static const void *sweep_kernel_ptr(int ns, int mixed) {
  if (ns == 1) return program_kernel_d1w();
  if (ns == 2) return mixed ? program_kernel_f2w() : program_kernel_d2w();
  return mixed ? program_kernel_f3w() : program_kernel_d3w();
}

// Clusters above the portable 8 CTAs.
static cudaError_t allow_large_clusters(const void *fn) {
  return allow_attribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

size_t program_shared_bytes(int mixed, const KParams &h) {
  return std::max(h.ring * ring_tile_bytes(h.AU.W, mixed),   // one row width for both matrices
                  (size_t)std::max(h.sweep, 0));
}

cudaError_t launch_program(int ns, int mixed, int occ, int mode, int nblocks, const KParams *hparams, int prog,
                           int iters, int step, cudaStream_t stream) {
  const void *fn = hparams->sweep >= 0 ? sweep_kernel_ptr(ns, mixed) : program_kernel_ptr(ns, mixed, occ);
  void *args[4];
  args[3] = (void *)&step;
  args[0] = (void *)hparams;
  args[1] = (void *)&prog;
  args[2] = (void *)&iters;
  const size_t dyn = program_shared_bytes(mixed, *hparams);
  cudaError_t e = allow_ring(fn, occ);
  if (e != cudaSuccess) return e;
  if (mode == SYNC_BLOCK) return cudaLaunchKernel(fn, dim3(1), dim3(TPB), args, dyn, stream);
  if (mode == SYNC_CLUSTER) {
    e = allow_large_clusters(fn);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblocks);
    cfg.blockDim = dim3(TPB);
    cfg.dynamicSmemBytes = dyn;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nblocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
  }
  return cudaLaunchCooperativeKernel(fn, dim3(nblocks), dim3(TPB), args, dyn, stream);
}

static const void *cg_kernel_ptr(int mixed, int W) { return mixed ? cg_kernel_cf(W) : cg_kernel_cd(W); }

int cg_blocks(int mixed, int W, int device) {
  int per_sm = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cg_kernel_ptr(mixed, W), TPB, 0) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return per_sm * sms;
}

cudaError_t launch_cg(int mixed, int nblocks, const KParams *hparams, cudaStream_t stream) {
  void *args[1] = {(void *)hparams};
  return cudaLaunchCooperativeKernel(cg_kernel_ptr(mixed, hparams->AP.W), dim3(nblocks), dim3(TPB), args, 0, stream);
}

// Shared memory of a CTA of the cluster form: what an SM gives one CTA, less
// its static part.
static constexpr size_t CGC_BYTES = 220 * 1024;
static const void *cgc_kernel_ptr(int mixed, int W) { return mixed ? cgc_kernel_cf(W) : cgc_kernel_cd(W); }
static size_t cgc_bytes(int mixed, int W, int slots) {
  return (size_t)slots * TILE * ((size_t)(CGC_VECTORS + W) * (mixed ? 4 : 8) + W * sizeof(unsigned));
}

CgCluster cg_cluster(int mixed, int W, int n0, int ntiles) {
  CgCluster f{0, 0};
  if (n0 < 1 || W < 1 || W > WUNROLL || ntiles > CGC_TILES) return f;
  const void *fn = cgc_kernel_ptr(mixed, W);
  if (allow_large_clusters(fn) != cudaSuccess ||
      allow_attribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CGC_BYTES) != cudaSuccess) {
    (void)cudaGetLastError();
    return f;
  }
  const int N0 = (n0 - 1) / TILE + 1, N1 = ntiles - N0;
  for (int G = std::min(16, ntiles); G >= 1; G >>= 1) {
    int slots = 0;
    for (int b = 0; b < G; ++b)
      slots = std::max(slots, chunk(b + 1, N0, G) - chunk(b, N0, G) + chunk(b + 1, N1, G) - chunk(b, N1, G));
    if (slots > CGC_SLOTS || cgc_bytes(mixed, W, slots) > CGC_BYTES) return f;   // fewer CTAs hold even less
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(CGC_TPB);
    cfg.dynamicSmemBytes = cgc_bytes(mixed, W, slots);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int fits = 0;
    if (cudaOccupancyMaxActiveClusters(&fits, fn, &cfg) == cudaSuccess && fits >= 1) {
      f.ctas = G;
      f.slots = slots;
      return f;
    }
    (void)cudaGetLastError();   // this cluster size is not possible: try the next smaller
  }
  return f;
}

cudaError_t launch_cg_cluster(int mixed, const CgCluster &form, const KParams *hparams, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(form.ctas);
  cfg.blockDim = dim3(TILE * std::min(CGC_TPB / TILE, form.slots));
  cfg.dynamicSmemBytes = cgc_bytes(mixed, hparams->AP.W, form.slots);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = form.ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *args[2] = {(void *)hparams, (void *)&form.slots};
  return cudaLaunchKernelExC(&cfg, cgc_kernel_ptr(mixed, hparams->AP.W), args);
}

// Load every build of the program on the current device now.  With lazy
// module loading a build is loaded on its first query or launch, and loading
// can wait for kernels already running on the device; a serving loop, whose
// runs overlap, loads them all before its first case.
void preload_programs() {
  for (int ns = 1; ns <= 3; ++ns)
    for (int mixed = 0; mixed <= 1; ++mixed)
      for (int occ = 0; occ <= 1; ++occ) {
        if (ns == 1 && (mixed || occ)) continue;
        cudaFuncAttributes a;
        if (cudaFuncGetAttributes(&a, program_kernel_ptr(ns, mixed, occ)) != cudaSuccess) (void)cudaGetLastError();
      }
}

// Occupancy probes: a failed query counts as zero and its error is consumed
// here, so that it is not reported later by an unrelated call that reads the
// runtime's last error.
int max_coresident_blocks(int ns, int occ, int device) {
  int per_sm = 0, sms = 0, per_sm32 = 0;
  const size_t dyn = RING_BYTES[occ ? 1 : 0];
  if (allow_ring(program_kernel_ptr(ns, 0, occ), occ) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, program_kernel_ptr(ns, 0, occ), TPB, dyn) !=
          cudaSuccess) {
    (void)cudaGetLastError();
    per_sm = 0;
  }
  if (ns >= 2) {
    if (allow_ring(program_kernel_ptr(ns, 1, occ), occ) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm32, program_kernel_ptr(ns, 1, occ), TPB, dyn) !=
            cudaSuccess) {
      (void)cudaGetLastError();
      per_sm32 = 0;
    }
    per_sm = std::min(per_sm, per_sm32);
  }
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
    (void)cudaGetLastError();
    sms = 0;
  }
  return per_sm * sms;
}

static int probe_cluster_blocks(int ns, int occ);

// Largest cluster of the program that fits an empty device, cached per
// (components, build, device).
int max_cluster_blocks(int ns, int occ) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    (void)cudaGetLastError();
    dev = 0;
  }
  const std::pair<int, int> key{ns * 4 + occ, dev};
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
  }
  const int c = probe_cluster_blocks(ns, occ);
  std::lock_guard<std::mutex> lk(mu);
  cache[key] = c;
  return c;
}

static int probe_cluster_blocks(int ns, int occ) {
  const void *fn = program_kernel_ptr(ns, 0, occ);
  if (allow_large_clusters(fn) != cudaSuccess || allow_ring(fn, occ) != cudaSuccess) {
    (void)cudaGetLastError();
    return 8;
  }
  for (int c = 16; c >= 1; c >>= 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(TPB);
    cfg.dynamicSmemBytes = RING_BYTES[occ ? 1 : 0];
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();   // this cluster size is not possible: try the next smaller
      continue;
    }
    if (nclusters >= 1) return c;
  }
  return 1;
}

}  // namespace xcal
