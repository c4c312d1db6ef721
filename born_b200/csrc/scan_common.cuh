// Shared definitions of the streaming sampler: work decomposition, scratch records and the
// arguments of scan_kernel / merge_kernel.
//
// Work decomposition.  A row is cut into blocks of 1024 tokens, counted from its first token.  The
// part of a row inside one CTA is a *segment*; its blocks are dealt to the CTA's eight warps, each
// of which streams its own (warp_ring.cuh).  While the rows fit the GPU (rows <= two CTAs per SM)
// every row is given `slices` CTAs of its own, each with one segment; more rows take a CTA each, in
// waves.  Only long rows with a nearly empty second wave form one sequence of blocks that is cut
// into equal contiguous ranges, one per CTA, so that a CTA may end in mid-row (fill_scan in capi.cu
// has the rule).  A row that one CTA streamed from first to last block is finished by it
// at once.  The slices of a row, up to eight, form a thread-block cluster: they write their keys,
// history values and statistics straight into the first one's shared memory, which finishes the row
// after one cluster barrier.  Otherwise (more slices, or ranges) the segments leave records in scratch
// and the CTA that completes the row (atomic ticket, no spinning) finishes it.
//
// What a segment leaves behind is small and never overflows: its statistics, and one 16-bit key
// per group of 32 tokens -- the upper half of the order-preserving key of the group's maximum.  The
// finish decides from the group keys which groups can hold tokens that matter and reads those again.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/born_sampler.h"
#include "spec.cuh"
#include "warp_ring.cuh"

namespace born {

constexpr int kScanWarps = kThreads / 32;
constexpr int kScanThreads = kThreads;
constexpr int kScanStagesMax = 8;           // slots per warp ring, at most
constexpr int kMassBlock = 512;             // tokens per mass block of the whole-vocabulary routes: half a warp's block
constexpr int kSelCap = 1024;               // candidates the in-shared-memory selection handles
constexpr int kHistBuckets = 128;           // the history list of a segment is grouped by block (or run of blocks)
constexpr int kHistTables = 32768;          // ... built with tables of this size where the ring has the room
constexpr int kHistPos = 2048;              // ... and this many list positions by a hash of the token
constexpr int kClusterMax = 8;              // slices of a row that exchange through distributed shared memory
constexpr int kGrpRound = 4096;             // group keys a CTA looks at before it reads the groups it found again
constexpr int kBins = 1024;                 // bins of the finish's histograms
constexpr uint32_t kDeadKey16 = 0x7Fu;      // group key of a group with nothing above -inf (-inf itself: 0x007FFFFF)
// Shared memory of a finish: selection (rank keys, masses; before them the histograms) | group lists.
constexpr int kWorkBytes = 2 * kSelCap * 8 + kGrpRound * 2;
static_assert(kGrpRound * 2 >= kBins * 8, "the larger selection keeps its bins where the group list was");
// ... and of the exact search (fallback.cuh), which has the ring to itself
constexpr int kExactBytes = 61440;

enum : int { kScanFull = 0, kScanLocal = 1 };

struct SegHdr {        // 32 bytes, precedes the history entries of a segment record
    float m;           // maximum of the segment (NaN if a NaN was seen)
    float lse_sum;     // sum of 2^((z - m) * c2) over the segment
    uint32_t n_hist;   // entries that follow: (penalised value bits << 32) | token of the virtual row
    uint32_t pad[5];
};
static_assert(sizeof(SegHdr) == kRecordHdrBytes, "segment header size");
constexpr int64_t kSegRecordBytes = kRecordHdrBytes + 8 * (int64_t)BORN_MAX_HISTORY;

struct MassBlock {     // one per kMassBlock tokens of a row, aligned to the row start
    float m;           // maximum of the block (-inf: nothing above -inf)
    uint32_t pad;      // tokens of the block above -inf
    unsigned long long M;  // exact sum of rne(exp_det((z - m) * inv_T) * 2^40) over the block
};

// Dynamic shared memory of a launch, laid out on the host (scan_smem_layout).
struct ScanSmem {
    int stages;     // ring slots per warp
    int slot;       // bytes per slot: logits, then the mask words
    int work;       // kWorkBytes for the finish.  One segment per CTA: over the ring, idle by then
    int hash;       // the history build's tables (hist_build).  One segment per CTA: the last `held` ring
                    // stages, which are filled only after the build; else the work area
    int hash_lg;    // ... 2^hash_lg keys and counts fit
    int hash_bytes; // ... room there is
    int held;
    int gkeys;      // group keys of a row the CTA streams alone ...
    int gkeys_cap;  // ... groups there is room for
    int list;       // history list, then the kHistBuckets + 1 bucket offsets
    int list_cap;
    int per_warp;   // local_kernel: bytes of a warp's part (the offsets above are inside it)
    int total;
};

struct ScanArgs {
    const void* logits;
    int64_t row_stride;   // elements between caller rows
    const uint32_t* mask;
    int64_t mask_stride;  // words between caller rows
    const int32_t* history;
    const int32_t* history_len;
    int history_stride;
    // device-resident history (born_history_*): the finished row appends its token here
    int32_t* ring;            // [rows, ring_cap] the last ring_cap tokens of every row; NULL: off
    int32_t* ring_total;      // [rows] tokens appended since the reset
    int32_t* ring_len;        // [rows] min(total, ring_cap): what the next call reads as history_len
    int32_t* ring_finished;   // [rows] non-zero once the row has sampled a stop token
    int ring_cap, n_stop;
    int32_t stop_ids[8];
    const born_row_params* row_params;
    born_row_params params;
    const float* uniforms;
    int32_t* out_token;
    float* out_prob;
    float* out_lse;
    int32_t* out_status;
    int32_t* out_kept_ids;
    int32_t* out_kept_count;
    int kept_stride;
    int B;         // caller rows
    int G;         // contiguous vocabulary segments per caller row (1: none); a (row, segment) pair is
                   // streamed as a row of its own ("virtual row" r = b * G + g)
    int V;         // tokens per virtual row
    int nb;        // blocks per virtual row
    int slices;    // CTAs per virtual row; 0: contiguous ranges of blocks instead
    int cluster;   // the slices of a row are a thread-block cluster
    int mode;      // kScanFull: sample; kScanLocal: leave the k best of every virtual row in `packed`
    int want_lse;
    int idx_base;  // added to the token ids written in kScanLocal mode
    uint8_t* packed;            // kScanLocal: record of virtual row (b, g) at g*packed_seg_stride + b*packed_row_stride
    int64_t packed_row_stride, packed_seg_stride;
    uint8_t* records;           // segment records (kSegRecordBytes each), see seg_record
    uint16_t* gkeys;            // [rows, nb * 32] group keys of rows that do not fit one CTA's shared memory
    MassBlock* blocks;          // [rows, nblk]
    int nblk;
    uint32_t* tickets;          // [rows] zero between launches
    uint32_t* deferred;         // [rows] zero between launches: cta+1 that owes the row its exact search
    int* dev_error;                 // [0] error word, [1] rows that took the exact search, [8..16] ... by reason
    unsigned long long timeout_ns;  // limit of every on-device wait
    long long debug_skip_blk;       // test hook: the bulk copy of this block is never issued (-1: none)
    ScanSmem L;
};

// ---- thread-block clusters ------------------------------------------------------------------
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Generic address of `p` (this CTA's shared memory) in CTA `rank` of the cluster.
template <typename P>
__device__ __forceinline__ P* cluster_map(P* p, uint32_t rank) {
    unsigned long long r;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return reinterpret_cast<P*>(r);
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- geometry -----------------------------------------------------------------------------
struct RowGeom {
    int b, g;              // caller row, vocabulary segment
    const uint8_t* base;   // the row's first logit
};
template <typename T>
__device__ __forceinline__ RowGeom row_geom(const ScanArgs& A, int r) {
    RowGeom q;
    q.b = A.G == 1 ? r : r / A.G;
    q.g = r - q.b * A.G;
    q.base = reinterpret_cast<const uint8_t*>(A.logits) + ((int64_t)q.b * A.row_stride + (int64_t)q.g * A.V) * (int64_t)sizeof(T);
    return q;
}
// bytes of mask words in a slot: 32 words, one more when a segment starts in mid-word, and the
// granules on either side of them
constexpr int kMaskSlotBytes = 256;

// CTA ranges [c*N/P, (c+1)*N/P) of a sequence of N blocks over P CTAs
__host__ __device__ inline long long range_begin(long long c, long long N, long long P) { return c * N / P; }
__host__ __device__ inline int cta_of_block(long long t, long long N, long long P) {
    return (int)(((t + 1) * P + N - 1) / N - 1);
}
// first CTA with a segment of row r, and how many there are
__device__ __forceinline__ void row_ctas(const ScanArgs& A, int row, int& c_first, int& n) {
    if (A.slices > 0) { c_first = row * A.slices; n = A.slices; return; }
    const long long N = (long long)A.B * A.G * A.nb;
    c_first = cta_of_block((long long)row * A.nb, N, gridDim.x);
    n = cta_of_block((long long)(row + 1) * A.nb - 1, N, gridDim.x) - c_first + 1;
}
// Record of the segment that CTA `cta` holds of row `row` (ranges: a CTA ends in mid-row at most
// twice; the row its range begins in has the first of its two records).
__device__ __forceinline__ uint8_t* seg_record(const ScanArgs& A, int row, int cta) {
    int i = cta;
    if (A.slices == 0) i = 2 * cta + (range_begin(cta, (long long)A.B * A.G * A.nb, gridDim.x) / A.nb == row ? 0 : 1);
    return A.records + (int64_t)i * kSegRecordBytes;
}

// Room for `limit` bytes per CTA (two CTAs per SM), as many ring stages as fit.
//   one_seg: every CTA streams exactly one segment (slices > 0)
//   groups:  group keys of a row if CTAs finish whole rows from shared memory, else 0
inline ScanSmem scan_smem_layout(int elem_bytes, bool aligned, bool has_mask, int hist_cap, bool one_seg, int groups, int limit) {
    ScanSmem L;
    L.slot = ring_slot_bytes(elem_bytes, aligned) + (has_mask ? kMaskSlotBytes : 0);
    const int stage = kScanWarps * L.slot;
    L.hash_lg = 7;
    while ((1 << L.hash_lg) < 2 * hist_cap) ++L.hash_lg;
    L.list_cap = hist_cap;
    const int list = hist_cap ? hist_cap * 8 + (kHistBuckets + 4) * 2 : 0;
    int gk = (groups * 2 + 15) / 16 * 16;
    if (gk > 24576) gk = 0;  // (beyond some 390 000 tokens: global memory)
    const int fixed = gk + list + (one_seg ? 0 : kWorkBytes);
    L.stages = (limit - fixed) / stage;
    if (L.stages > kScanStagesMax) L.stages = kScanStagesMax;
    if (L.stages < 2) L.stages = 2;
    int off = L.stages * stage;
    if (one_seg) {
        L.work = 0;
        L.held = hist_cap ? (kHistTables + stage - 1) / stage : 0;
        if (L.held > L.stages - 1) L.held = L.stages - 1;
        L.hash = (L.stages - L.held) * stage;
        L.hash_bytes = L.held * stage;
    } else {
        L.work = off;
        off += kWorkBytes;
        L.hash = L.work;
        L.hash_bytes = kWorkBytes;
        L.held = 0;
    }
    if (off < kExactBytes) off = kExactBytes;
    L.gkeys = off;
    L.gkeys_cap = gk / 2;
    off += gk;
    L.list = off;
    off += list;
    L.total = (off + 127) & ~127;
    return L;
}

// local_kernel: a warp's part of the dynamic shared memory is ring | group keys | candidates | group list.
constexpr int kLocalCap = 256;     // candidates (and listed groups) a warp has room for
constexpr int kLocalMaxK = 128;    // top-k up to which the 256 maxima of a warp tell the k-th key well
// (stages: 0 when the row is too long)
inline ScanSmem local_smem_layout(int elem_bytes, int nb, int limit) {
    ScanSmem L = {};
    L.slot = ring_slot_bytes(elem_bytes, true);
    const int fixed = nb * 64 + kLocalCap * 8 + kLocalCap * 2;
    const int per = limit / kScanWarps / 128 * 128;
    L.stages = per >= fixed + 2 * L.slot ? (per - fixed) / L.slot : 0;
    if (L.stages > kScanStagesMax) L.stages = kScanStagesMax;
    L.gkeys = L.stages * L.slot;
    L.gkeys_cap = nb * 32;
    L.work = L.gkeys + nb * 64;
    L.list = L.work + kLocalCap * 8;
    L.per_warp = (L.list + kLocalCap * 2 + 127) & ~127;
    L.total = kScanWarps * L.per_warp;
    if (L.total < kExactBytes) L.total = kExactBytes;
    return L;
}

// Static shared state of a CTA of scan_kernel (and of merge_kernel, which uses the selection part).
struct ScanShared {
    unsigned long long bars[kScanStagesMax * kScanWarps];
    float wmax[kScanWarps], wsum[kScanWarps];
    float2 part[kClusterMax];       // cluster: (maximum, log-sum-exp sum) of every slice, in the first one
    uint32_t remote_hist;           // cluster: history entries the other slices have left at the list's end
    int remote_fail;                // cluster: a wait of another slice ran out
    uint32_t defer;                 // the CTA has handed a row to the exact search: its `deferred` word (0: none)
    int last;
    // finish / selection scratch
    unsigned long long red64[kScanWarps];
    unsigned long long acc[4];
    float redf[kScanWarps];
    uint32_t redu[kScanWarps];
    uint4 bcnt[kHistBuckets / 4];   // counts of the history build; after it, the finish's map of candidates
    int nl, nw;
    uint32_t ng[2], nh;             // groups listed (by parity of the round), history values added
    int found;
    unsigned long long before;
    alignas(16) SearchScratch sc;
};

__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float warp_max_nan(float v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = max_nan(v, __shfl_xor_sync(0xffffffffu, v, d));
    return v;
}

// Penalised logit of a history token (once per distinct token, `cnt` = its multiplicity):
// repetition z>0 ? z/r : z*r, then z -= (f*cnt + p) as three separately rounded operations.
__device__ __forceinline__ float penalise(const born_row_params& rp, float z, int cnt) {
    if (rp.repetition_penalty != 1.0f && rp.repetition_penalty != 0.0f)
        z = (z > 0.0f) ? __fdiv_rn(z, rp.repetition_penalty) : __fmul_rn(z, rp.repetition_penalty);
    if (rp.frequency_penalty != 0.0f || rp.presence_penalty != 0.0f) {
        float pen = __fmul_rn(rp.frequency_penalty, (float)cnt);
        pen = __fadd_rn(pen, rp.presence_penalty);
        z = __fsub_rn(z, pen);
    }
    return z;
}
// The range check that the host applies to uniform parameters (params_ok in capi.cu), for
// per-row parameter arrays that live on the device and so reach the kernel unchecked.
__device__ __forceinline__ bool row_params_ok(const born_row_params& p) {
    const bool fin = isfinite(p.temperature) && isfinite(p.top_p) && isfinite(p.repetition_penalty) &&
                     isfinite(p.frequency_penalty) && isfinite(p.presence_penalty);
    return fin && p.temperature >= 0.0f && (p.temperature == 0.0f || p.temperature >= 1e-4f) && p.top_p >= 0.0f &&
           p.min_p >= 0.0f && p.min_p <= 1.0f && p.top_k >= 0 && p.top_k <= BORN_MAX_TOP_K && p.repetition_penalty >= 0.0f;
}
__device__ __forceinline__ bool penalties_on(const born_row_params& rp) {
    return (rp.repetition_penalty != 1.0f && rp.repetition_penalty != 0.0f) || rp.frequency_penalty != 0.0f ||
           rp.presence_penalty != 0.0f;
}

// Route classes the streaming kernel is instantiated for, so that a launch whose rows all take
// the same kind of route does not carry (and pay, in registers and instruction fetches) the code
// of the others: 0 any route (per-row parameter arrays), 1 rows with candidates only (greedy, top-k,
// min-p), 2 rows whose total comes from the mass blocks (temperature only, top-p alone).
template <int kRoute>
struct RouteOf {
    static constexpr bool mass = kRoute != 1;
    static constexpr bool cand = kRoute != 2;
};

// What a row's parameters ask of the streaming pass.
struct RowPlan {
    bool greedy, minp, topp;
    bool need_mass;    // no top-k and no min-p: the row total comes from the mass blocks
    bool window;       // ... and a nucleus has to be found in it (top-p alone)
    int k;             // top-k (0: off)
    float inv_T, c2, delta;
};
__device__ __forceinline__ RowPlan row_plan(const born_row_params& rp) {
    RowPlan p;
    p.greedy = (rp.flags & BORN_FLAG_GREEDY) || rp.temperature == 0.0f;
    p.inv_T = p.greedy ? 1.0f : __fdiv_rn(1.0f, rp.temperature);
    p.c2 = p.inv_T * 1.44269504f;
    p.k = (!p.greedy && rp.top_k > 0) ? rp.top_k : 0;
    p.minp = !p.greedy && rp.min_p > 0.0f;
    p.topp = !p.greedy && rp.top_p > 0.0f && rp.top_p < 1.0f;
    p.need_mass = !p.greedy && p.k == 0 && !p.minp;
    p.window = p.need_mass && p.topp;
    // min-p: nothing this far below the maximum survives (the margin covers the logarithm's error)
    p.delta = p.minp ? (__logf(rp.min_p) - 0.05f) * rp.temperature : 0.0f;
    return p;
}

}  // namespace born
