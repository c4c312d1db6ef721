// scan_kernel for fp32 launches with grammar masks and token histories.
#include <cstdint>
#define SCAN_INST_T float
#define SCAN_INST_MASK true
#define SCAN_INST_HIST true
#define SCAN_INST_ATTRS scan_attrs_f32_mask_hist
#define SCAN_INST_LAUNCH scan_launch_f32_mask_hist
#include "scan_inst.cuh"
