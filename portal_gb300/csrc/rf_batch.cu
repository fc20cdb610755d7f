// The batched radiation-field launch: the kernel instantiated over (model,
// node) work items of many models (the batch of batch.cu; star mode runs it
// with one model).  Compiled apart from rf.cu so the two sets of
// instantiations build in parallel.
#include "rf_kernel.cuh"

namespace {

const void *batch_kernel(bool dust) {
    return dust ? (const void *)k_radiation_field<0, true, true, 0, true>
                : (const void *)k_radiation_field<0, false, true, 0, true>;
}

size_t batch_dyn_smem(const RFBatch &bw) {
    return ((bw.nch * sizeof(float2) + 15) & ~(size_t)15) + RF_BATCH_WARPS * bw.warp_bytes;
}

}  // namespace

namespace portal {

void rf_batch_shape(RFBatch *bw, const int *lines, int n_models, int nch, bool dust, int max_group, bool split) {
    int max_lines = 0;
    for (int m = 0; m < n_models; m++) max_lines = std::max(max_lines, lines[m]);
    bw->nch = nch;
    bw->max_group = max_group;
    bw->rt = rf_remainder(nch, dust, max_lines);
    bw->split = split;
    bw->warp_bytes = 0;
    for (int m = 0; m < n_models; m++)
        bw->warp_bytes = std::max(bw->warp_bytes,
                                  (size_t)rf_shape(lines[m], max_group, nch, dust, bw->rt, split).bytes);
}

// Also raises the kernel's dynamic shared-memory limit: called for every
// candidate before the pass is captured.
int rf_batch_blocks_per_sm(const RFBatch &bw, bool dust, int *blocks) {
    const void *k = batch_kernel(dust);
    const size_t dyn = batch_dyn_smem(bw);
    *blocks = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) != cudaSuccess)
        return PORTAL_ERR_CUDA;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, 32 * RF_BATCH_WARPS, dyn);
    return e == cudaSuccess ? PORTAL_OK : PORTAL_ERR_CUDA;
}

int rf_batch_launch(cudaStream_t s, int grid, bool dust, const RFBatch &bw) {
    RFArgs a0{};
    RFBatch b = bw;
    RFShape sh{};
    void *args[] = {&a0, &b, &sh};
    cudaError_t e = cudaLaunchKernel(batch_kernel(dust), dim3(grid), dim3(32 * RF_BATCH_WARPS), args,
                                     batch_dyn_smem(bw), s);
    return e == cudaSuccess ? PORTAL_OK : PORTAL_ERR_CUDA;
}

}  // namespace portal
