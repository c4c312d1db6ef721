// scan_kernel for bf16 launches with no mask and no token history.
#include <cstdint>
#define SCAN_INST_T uint16_t
#define SCAN_INST_MASK false
#define SCAN_INST_HIST false
#define SCAN_INST_ATTRS scan_attrs_bf16
#define SCAN_INST_LAUNCH scan_launch_bf16
#define SCAN_INST_LOCAL_ATTRS local_attrs_bf16
#define SCAN_INST_LOCAL local_launch_bf16
#include "scan_inst.cuh"
