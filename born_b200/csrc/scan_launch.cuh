// Host-side entry points of the streaming kernel's instantiations.  The kernel is instantiated
// in eight translation units that compile side by side, one per element type, with and without
// grammar masks and token histories; each holds the three route classes (RouteOf in
// scan_common.cuh) for 16-byte-aligned rows and one for the others.  capi.cu only calls these.
#pragma once
#include <cuda_runtime.h>
#include "scan_common.cuh"

namespace born {

// Dynamic shared memory: what two CTAs per SM leave each of them (an SM has 228 KB, a CTA costs 1 KB
// of it on top of its own), and what one CTA may ask for.
constexpr int kScanSmemTwo = (228 * 1024 / 2 - 1024 - (int)sizeof(ScanShared) - 16) & ~127;
constexpr int kScanSmemMax = (227 * 1024 - (int)sizeof(ScanShared) - 16) & ~127;

// SCAN_UNIT(name) declares, for one translation unit,
//   scan_attrs_<name>():  raise the dynamic shared-memory limit of its instantiations (once per device)
//   scan_launch_<name>(): launch the instantiation for (alignment, route class); returns cudaGetLastError()
#define SCAN_UNIT(name)              \
    cudaError_t scan_attrs_##name(); \
    cudaError_t scan_launch_##name(const ScanArgs& A, bool aligned, int route, int grid, cudaStream_t st);
SCAN_UNIT(f32)
SCAN_UNIT(f32_hist)
SCAN_UNIT(f32_mask)
SCAN_UNIT(f32_mask_hist)
SCAN_UNIT(bf16)
SCAN_UNIT(bf16_hist)
SCAN_UNIT(bf16_mask)
SCAN_UNIT(bf16_mask_hist)
#undef SCAN_UNIT
// local_kernel (a warp per virtual row): rows on 16-byte boundaries, no mask, no token history.
cudaError_t local_attrs_f32();
cudaError_t local_attrs_bf16();
cudaError_t local_launch_f32(const ScanArgs& A, int grid, cudaStream_t st);
cudaError_t local_launch_bf16(const ScanArgs& A, int grid, cudaStream_t st);
// Clusters of `size` CTAs of the streaming kernel that the current device holds at once.
cudaError_t scan_max_clusters(int size, int* count);

}  // namespace born
