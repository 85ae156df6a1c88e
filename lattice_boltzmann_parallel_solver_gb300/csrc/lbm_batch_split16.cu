// lbm_batch_split16.cu -- batched steps as a boundary-free step followed by the
// boundary-node pass: the 16-bit storages.
#include "lbm_batch.cuh"

namespace lbm {

int batch_launch_split16(const void* table, int n, int tiles, int bc_chunks, int storage, int npt, int threads,
                         int* gbase, int nsteps, int blocks, cudaStream_t s) {
  LBM_BATCH_DISPATCH_16(false)
  return no_batch_kernel();
}

}  // namespace lbm
