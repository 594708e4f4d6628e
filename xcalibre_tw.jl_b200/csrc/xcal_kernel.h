// Host-visible declarations of the persistent device program.
#pragma once
#include <cuda_runtime.h>

#include "xcal_device.cuh"

namespace xcal {
// occ selects the build: 0 = two resident CTAs per SM (128 registers),
// 1 = four (64 registers); the NS = 1 standalone-solve program and the builds for
// sweeps by one CTA (taken where hparams->sweep >= 0) have only the first.
cudaError_t launch_program(int ns, int mixed, int occ, int mode, int nblocks, const KParams *hparams, int prog,
                           int iters, int step, cudaStream_t stream);
// The pressure solve between two steps of a run (two-level numbering, row
// width at most WUNROLL), on cg_blocks CTAs.
cudaError_t launch_cg(int mixed, int nblocks, const KParams *hparams, cudaStream_t stream);
int cg_blocks(int mixed, int W, int device);
// The same solve in one cluster that holds the mesh in shared memory: its CTAs
// and the tiles of the largest share; 0 CTAs when the mesh does not fit.
struct CgCluster {
  int ctas, slots;
};
CgCluster cg_cluster(int mixed, int W, int n0, int ntiles);
cudaError_t launch_cg_cluster(int mixed, const CgCluster &form, const KParams *hparams, cudaStream_t stream);
// Matrix tiles of the launch's dynamic shared memory ring (KParams::ring).
int ring_tiles(int W, int mixed, int occ, int ntiles, int nblocks);
// Dynamic shared memory of a CTA of the program's launch.
size_t program_shared_bytes(int mixed, const KParams &h);
// Dynamic shared memory for the vector of a sweep by one CTA (a vector that
// does not fit stays in global memory).
int sweep_bytes(size_t bytes, int occ);
int max_coresident_blocks(int ns, int occ, int device);
int max_cluster_blocks(int ns, int occ = 0);
const void *program_kernel_ptr(int ns, int mixed, int occ);
void preload_programs();   // load every build on the current device
// the serving kernel (xcal_serve_kernel) of a dimension and precision, and the
// dynamic shared memory and size of its launch on a device
const void *serve_kernel_ptr(int ns, int mixed, int sweeps);
size_t serve_shared_bytes(int ns, int mixed, int sweeps, int tiles_per_cta);
int serve_grid(int ns, int mixed, int sweeps, size_t shared_bytes, int device);
}  // namespace xcal
