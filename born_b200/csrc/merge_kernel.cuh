// merge_kernel: the second half of vocab-sharded sampling.  Every shard (a GPU of a
// tensor-parallel lm_head, or a vocabulary segment on one GPU) has left one packed record per
// row -- its k best tokens as rank keys with global token ids, its maximum and its share of
// the log-sum-exp.  One CTA per row folds the G records: row maximum, log-sum-exp, the union
// of the candidates, then top-p and the inverse-CDF draw on exact integer masses relative to
// the row maximum (finish.cuh), so the result does not depend on how the vocabulary was cut.
#pragma once
#include "finish.cuh"

namespace born {

struct MergeArgs {
    const uint8_t* gathered;  // record of (shard g, row b) at g*seg_stride + b*row_stride
    int64_t row_stride, seg_stride;
    int B, G;
    float temperature, top_p;
    const float* uniforms;
    int32_t* out_token;
    float* out_prob;
    float* out_lse;
    int32_t* out_status;
    int32_t* out_kept_ids;
    int32_t* out_kept_count;
    int kept_stride;
};

__global__ void __launch_bounds__(kThreads) merge_kernel(const __grid_constant__ MergeArgs A) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ ScanShared sh;
    const int tid = threadIdx.x, b = blockIdx.x;
    uint64_t* sel = reinterpret_cast<uint64_t*>(smem);
    unsigned long long* selq = reinterpret_cast<unsigned long long*>(sel + kSelCap);
    // (starts while the launch that writes the records may still be working)
    grid_launch_dependents();
    grid_dependency_wait();
    const float inv_T = __fdiv_rn(1.0f, A.temperature);
    const float c2 = inv_T * 1.44269504f;
    auto rec_of = [&](int g) { return A.gathered + (int64_t)g * A.seg_stride + (int64_t)b * A.row_stride; };
    // Every warp folds the headers for itself, a lane per record (word by word: a record of an odd number
    // of entries is only 8-byte aligned); then the warps share out the records' entries.  (A loop over the
    // records with a read and an atomic each is a chain of G round trips to L2.)
    const int lane = tid & 31, warp = tid >> 5;
    float m = -INFINITY, ls = 0.0f;
    int cnt = 0, failed = 0;
    if (tid == 0) sh.nl = 0;
    if (lane < A.G) {
        const uint32_t* h = reinterpret_cast<const uint32_t*>(rec_of(lane));
        m = __uint_as_float(__ldcg(h));
        ls = __uint_as_float(__ldcg(h + 1));
        cnt = (int)min(__ldcg(h + 2), (uint32_t)((A.row_stride - kRecordHdrBytes) / 8));  // (never beyond the record)
        failed = (int)(__ldcg(h + 3) & 2u);
    }
    cta_sync();
    const float mg = m;
    m = warp_max_nan(m);
    ls = ls > 0.0f ? ls * ex2_approx(__fmul_rn(mg - m, c2)) : 0.0f;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, d);
    failed = __any_sync(0xffffffffu, failed);
    for (int g = warp; g < A.G; g += kScanWarps) {
        const int c = __shfl_sync(0xffffffffu, cnt, g);
        const unsigned long long* ent = reinterpret_cast<const unsigned long long*>(rec_of(g) + kRecordHdrBytes);
        for (int i = 0; i < c; i += 64) {
            unsigned long long e[2];
            uint32_t ab[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) e[j] = i + 32 * j + lane < c ? __ldcg(ent + i + 32 * j + lane) : 0ull;
#pragma unroll
            for (int j = 0; j < 2; ++j) ab[j] = __ballot_sync(0xffffffffu, ck_alive(e[j]));
            int at = 0;
            if (lane == 0) at = (int)smem_atom_add(&sh.nl, (uint32_t)(__popc(ab[0]) + __popc(ab[1])));
            at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int pos = at + __popc(ab[j] & ((1u << lane) - 1u));
                if (ck_alive(e[j]) && pos < kSelCap) sel[pos] = e[j];
                at += __popc(ab[j]);
            }
        }
    }
    cta_sync();
    const int n = sh.nl;
    RowOut o;
    o.token = A.out_token; o.prob = A.out_prob; o.lse = A.out_lse; o.status = A.out_status;
    o.kept_ids = A.out_kept_ids; o.kept_count = A.out_kept_count; o.kept_stride = A.kept_stride;
    o.row = b;
    int status = BORN_ROW_OK;
    if (failed) status = 100 + BORN_ERR_DEVICE_TIMEOUT;
    else if (m != m) status = BORN_ROW_NAN;
    else if (m == INFINITY) status = BORN_ROW_POS_INF;
    else if (m == -INFINITY) status = BORN_ROW_ALL_MASKED;
    else if (n > kSelCap) status = BORN_ROW_OVERFLOW;
    if (A.out_lse && tid == 0) A.out_lse[b] = (status == BORN_ROW_OK || status == BORN_ROW_OVERFLOW) ? m * inv_T + __log2f(ls) * 0.69314718f : NAN;
    if (status != BORN_ROW_OK) {
        row_fail(o, status);
        return;
    }
    SelectIn in;
    in.n = n;
    in.k = 0;  // every shard has cut to its own k best already; the union is kept
    in.Qa = 0;
    in.top_p = A.top_p;
    in.S_ext = 0;
    in.m_row = m; in.inv_T = inv_T; in.u = A.uniforms[b];
    if (n <= kSmallMax) select_small(in, sel, selq, sh, o);
    else select_large(in, sel, selq, reinterpret_cast<uint32_t*>(selq + kSelCap), sh, o);
}

}  // namespace born
