// sssp_owner.cu -- the vertex-owner kernel and its launch helpers.
#include "sssp_owner.cuh"
#include "sssp_plain.h"

#include <algorithm>

namespace mlmq {

// LPV lanes per vertex: 2 for 32-byte tiles and row offsets, 4 for 64-byte tiles.
template <class Arcs, int LPV>
__global__ void __launch_bounds__(OWNER_THREADS, 1) sssp_owner_kernel(PlainParams p, OwnerParams o) {
    owner_solve<Arcs, LPV>(p, o);
}

namespace {
const void *owner_kernel(int tile_stride) {
    return tile_stride == 4 ? (const void *)sssp_owner_kernel<ArcsInterleaved, 4>
                            : (const void *)sssp_owner_kernel<ArcsInterleaved, 2>;
}
}  // namespace

int owner_threads() { return OWNER_THREADS; }

// Blocks of OWNER_BLOCK vertices while there are SMs for them, then larger
// ones.  Smaller blocks mean shorter lists but more messages: grid 1200x777 2.9
// ms in 22 blocks, 3.1 in 57; a million points 3.1 ms in 24 blocks, 2.9 in 64,
// 2.5 in 148; grid 512^2 1.29 ms in 7, 1.19 in 16, 1.25 in 24.
int owner_block(int n, int sms, int *ctas) {
    constexpr int OWNER_BLOCK = 16384;
    const int want = std::min(sms, (n + OWNER_BLOCK - 1) / OWNER_BLOCK);
    const int block = ((n + want - 1) / want + 31) / 32 * 32;
    *ctas = (n + block - 1) / block;
    return block <= OWNER_MAX_BLOCK ? block : 0;
}

size_t owner_tails_bytes(int ctas) { return 128 * (size_t)ctas; }

cudaError_t owner_prepare() {
    for (int stride : {2, 4}) {
        const cudaError_t e =
            cudaFuncSetAttribute(owner_kernel(stride), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)owner_smem_bytes(OWNER_MAX_BLOCK));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t owner_launch(const PlainParams &p, int block, int ctas, unsigned *tails,
                         cudaStream_t stream) {
    OwnerParams o;
    o.block = (unsigned)block;
    o.block_inv = 0xffffffffu / (unsigned)block;
    o.tails = tails;
    // The inboxes share the memory of the L2 rings, which both kernels leave
    // empty.
    const size_t slots = (size_t)(p.nb + 1) << p.l2_log;
    o.inbox_log = 0;
    while (o.inbox_log < 20 && ((size_t)ctas << (o.inbox_log + 1)) <= slots) o.inbox_log++;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(OWNER_THREADS);
    cfg.dynamicSmemBytes = owner_smem_bytes((unsigned)block);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {const_cast<PlainParams *>(&p), &o};
    return cudaLaunchKernelExC(&cfg, owner_kernel(p.tile_stride), args);
}

}  // namespace mlmq
