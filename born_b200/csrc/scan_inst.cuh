// Body of a translation unit that instantiates scan_kernel for one (element type, mask, history):
// included by the scan_*.cu units after they have defined
//   SCAN_INST_T      the element type (float or uint16_t)
//   SCAN_INST_MASK / SCAN_INST_HIST   whether the launches carry grammar masks / token histories
//   SCAN_INST_ATTRS / SCAN_INST_LAUNCH   the names of the two functions of scan_launch.cuh
//   SCAN_INST_LOCAL_ATTRS / SCAN_INST_LOCAL   (optional) local_kernel for the element type as well
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "../../include/born_sampler.h"
#include "scan_kernel.cuh"
#include "fallback.cuh"
#include "scan_launch.cuh"
#ifdef SCAN_INST_LOCAL
#include "local_kernel.cuh"
#endif

namespace born {
namespace {

template <bool kAligned, int R>
constexpr auto kernel_of = scan_kernel<SCAN_INST_T, SCAN_INST_MASK, SCAN_INST_HIST, kAligned, R>;

void scan_launch_config(const ScanArgs& A, int grid, cudaStream_t st, cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2]) {
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(kScanThreads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)A.L.total;
    cfg.stream = st;
    cfg.attrs = at;
    int n = 0;
    if (A.cluster) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)A.slices;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = (unsigned)(n + 1);
}

template <bool kAligned, int R>
cudaError_t attr_one() {
    return cudaFuncSetAttribute(kernel_of<kAligned, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmemMax);
}
template <bool kAligned, int R>
cudaError_t launch_one(const ScanArgs& A, int grid, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    scan_launch_config(A, grid, st, cfg, at);
    return cudaLaunchKernelEx(&cfg, kernel_of<kAligned, R>, A);
}

}  // namespace

// (rows that do not start on a 16-byte boundary reach the kernel on the candidate routes only: the
// others need their mass blocks where the row starts, and go through an aligned copy)
cudaError_t SCAN_INST_ATTRS() {
    cudaError_t e;
    if ((e = attr_one<true, 0>()) != cudaSuccess) return e;
    if ((e = attr_one<true, 1>()) != cudaSuccess) return e;
    if ((e = attr_one<true, 2>()) != cudaSuccess) return e;
    return attr_one<false, 1>();
}

#ifdef SCAN_INST_LOCAL
cudaError_t SCAN_INST_LOCAL_ATTRS() {
    return cudaFuncSetAttribute(local_kernel<SCAN_INST_T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmemTwo);
}
cudaError_t SCAN_INST_LOCAL(const ScanArgs& A, int grid, cudaStream_t st) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    scan_launch_config(A, grid, st, cfg, at);
    return cudaLaunchKernelEx(&cfg, local_kernel<SCAN_INST_T>, A);
}
#endif

#ifdef SCAN_INST_CLUSTERS
// Clusters of `size` CTAs that the current device holds at once (any instantiation: they share the
// register and shared-memory budget of two CTAs per SM).
cudaError_t SCAN_INST_CLUSTERS(int size, int* count) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    ScanArgs A;
    memset(&A, 0, sizeof A);
    A.cluster = 1;
    A.slices = size;
    A.L.total = kScanSmemTwo;
    scan_launch_config(A, size, nullptr, cfg, at);
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(count, kernel_of<true, 1>, &cfg);
}
#endif

cudaError_t SCAN_INST_LAUNCH(const ScanArgs& A, bool aligned, int route, int grid, cudaStream_t st) {
    if (!aligned) return route == 1 ? launch_one<false, 1>(A, grid, st) : cudaErrorInvalidValue;
    if (route == 1) return launch_one<true, 1>(A, grid, st);
    if (route == 2) return launch_one<true, 2>(A, grid, st);
    return launch_one<true, 0>(A, grid, st);
}

}  // namespace born
