// scan_kernel for fp32 launches with no mask and token histories.
#include <cstdint>
#define SCAN_INST_T float
#define SCAN_INST_MASK false
#define SCAN_INST_HIST true
#define SCAN_INST_ATTRS scan_attrs_f32_hist
#define SCAN_INST_LAUNCH scan_launch_f32_hist
#include "scan_inst.cuh"
