// The nodes of an uploaded arena with their children's first and count words
// packed into stack words (PtSceneDev::qnodes, stream.cuh).
#include "kernels.h"
#include "stream.cuh"

using namespace ptd;

namespace {

__global__ void qnodes_kernel(const uint32_t* __restrict__ nodes, uint32_t* __restrict__ qnodes, size_t words) {
    const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    if (i >= words) return;
    const uint32_t at = i & 31u;
    uint32_t w = nodes[i];
    if (at >= 28) {
        w = 0;
    } else if (at >= 24) {
        const uint32_t count = nodes[i + 4];
        if (count)
            w = PT_Q_LEAF | ((count & PT_LEAF_HAS_SPHERE) ? PT_Q_SPHERE : 0u) |
                ((count & PT_LEAF_INSTANCES) ? PT_Q_INST : 0u) | ((count & 15u) << 25) | (w & PT_Q_FIRST);
    }
    qnodes[i] = w;
}

}  // namespace

cudaError_t pt_build_qnodes(const float4* nodes, float4* qnodes, uint32_t n, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    const size_t words = 32 * size_t(n);
    qnodes_kernel<<<unsigned((words + 255) / 256), 256, 0, stream>>>(
        reinterpret_cast<const uint32_t*>(nodes), reinterpret_cast<uint32_t*>(qnodes), words);
    return cudaGetLastError();
}
