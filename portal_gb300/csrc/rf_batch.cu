// The batched radiation-field launch: the kernel instantiated over (model,
// node) work items of many models (the batch of batch.cu; star mode runs it
// with one model).  Compiled apart from rf.cu so the two sets of
// instantiations build in parallel.
#include "rf_kernel.cuh"

namespace {

// (instantiations in rf_batch_even.cu and rf_batch_any.cu)
const void *batch_kernel(const RFBatch &bw, bool dust) {
    const int nslot = (bw.nch - bw.rt + 31) / 32;
    if (!dust && !bw.split && nslot % 2 == 0) return rf_batch_even();
    return rf_batch_any(dust, nslot == 1, bw.split);
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

int rf_line_group(int lines, int max_group, bool dust) { return tab_shape(lines, max_group, dust).nlg; }

// Also sets the kernel's dynamic shared-memory limit: called before the pass is
// captured.
int rf_batch_blocks_per_sm(const RFBatch &bw, bool dust, int *blocks) {
    const void *k = batch_kernel(bw, dust);
    const size_t dyn = batch_dyn_smem(bw);
    *blocks = 0;
    if (allow_dyn_smem(k) != cudaSuccess) return PORTAL_ERR_CUDA;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, 32 * RF_BATCH_WARPS, dyn);
    return e == cudaSuccess ? PORTAL_OK : PORTAL_ERR_CUDA;
}

int rf_batch_launch(cudaStream_t s, int grid, bool dust, const RFBatch &bw) {
    RFArgs a0{};
    RFBatch b = bw;
    RFShape sh{};
    void *args[] = {&a0, &b, &sh};
    cudaError_t e = cudaLaunchKernel(batch_kernel(bw, dust), dim3(grid), dim3(32 * RF_BATCH_WARPS), args,
                                     batch_dyn_smem(bw), s);
    return e == cudaSuccess ? PORTAL_OK : PORTAL_ERR_CUDA;
}

}  // namespace portal
