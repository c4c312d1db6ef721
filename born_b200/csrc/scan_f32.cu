// scan_kernel for fp32 launches with no mask and no token history.
#include <cstdint>
#define SCAN_INST_T float
#define SCAN_INST_MASK false
#define SCAN_INST_HIST false
#define SCAN_INST_ATTRS scan_attrs_f32
#define SCAN_INST_LAUNCH scan_launch_f32
#define SCAN_INST_CLUSTERS scan_max_clusters
#define SCAN_INST_LOCAL_ATTRS local_attrs_f32
#define SCAN_INST_LOCAL local_launch_f32
#include "scan_inst.cuh"
