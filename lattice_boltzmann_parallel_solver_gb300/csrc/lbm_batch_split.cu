// lbm_batch_split.cu -- batched steps as a boundary-free step followed by the
// boundary-node pass: the 64- and 32-bit storages.
#include "lbm_batch.cuh"

namespace lbm {

int batch_launch_split(const void* table, int n, int tiles, int bc_chunks, int storage, int npt, int threads,
                       int* gbase, int nsteps, int blocks, cudaStream_t s) {
  LBM_BATCH_DISPATCH_WIDE(false)
  return batch_launch_split16(table, n, tiles, bc_chunks, storage, npt, threads, gbase, nsteps, blocks, s);
}

}  // namespace lbm
