// scan_kernel for bf16 launches with no mask and token histories.
#include <cstdint>
#define SCAN_INST_T uint16_t
#define SCAN_INST_MASK false
#define SCAN_INST_HIST true
#define SCAN_INST_ATTRS scan_attrs_bf16_hist
#define SCAN_INST_LAUNCH scan_launch_bf16_hist
#include "scan_inst.cuh"
