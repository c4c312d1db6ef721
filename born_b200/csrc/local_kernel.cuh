// local_kernel: the k best of very many virtual rows, a warp per row.
//
// The first half of vocab-sharded sampling (kScanLocal) over a large batch streams thousands of
// short rows: 1024 x 8 segments of 32000 bf16 tokens are 64 KB each.  scan_kernel gives such a row to
// a CTA, which reads it in 2 us and then spends 8 us on its finish -- a dozen barriers and two
// rounds of re-reads by eight warps that mostly wait, some 12 000 warp instructions per row, twice
// those of the streaming.  Here every warp streams rows of its own through its own ring and finishes
// them alone: no barrier, no atomics, a third of the finish's instructions, and while one warp waits
// for its re-reads the other fifteen of the SM stream.  That case, with its merge: 343 -> 195 us (2.7 TB/s).
// What bounds it: latency with four warps per scheduler -- 126 registers and 13 KB of ring, keys and
// candidates per warp leave no room for more -- which issue every other cycle (12 500 warp instructions
// per row; ncu: 51 % issue active, 35 % DRAM).
//
// The records are those of scan_kernel's finish (write_packed in finish.cuh): the same candidates in the
// same order; the log-sum-exp's terms are added in another order.
#pragma once
#include "scan_kernel.cuh"

namespace born {

template <typename T>
__global__ void __launch_bounds__(kScanThreads, 2) local_kernel(const __grid_constant__ ScanArgs A) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ ScanShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = A.nb, S = A.L.stages;
    uint8_t* part = smem + warp * A.L.per_warp;
    uint16_t* keys = reinterpret_cast<uint16_t*>(part + A.L.gkeys);
    uint64_t* sel = reinterpret_cast<uint64_t*>(part + A.L.work);
    uint16_t* list = reinterpret_cast<uint16_t*>(part + A.L.list);
    const uint32_t slot_bytes = (uint32_t)A.L.slot, slot0 = smem_u32(part), bar0 = smem_u32(&sh.bars[warp]);
    if (lane == 0) {
        for (int s = 0; s < S; ++s) mbar_init(reinterpret_cast<uint64_t*>(&sh.bars[s * kScanWarps + warp]), 1);
        mbar_fence_init();
    }
    if (tid == 0) sh.defer = 0;
    cta_sync();
    grid_launch_dependents();
    grid_dependency_wait();

    // the warp's rows: every W-th, consecutive rows on different CTAs
    const int R = A.B * A.G, W = (int)gridDim.x * kScanWarps;
    const int r0 = warp * (int)gridDim.x + (int)blockIdx.x;
    const uint32_t last_bytes = ((uint32_t)(A.V - (nb - 1) * kBlkTok) * (uint32_t)sizeof(T) + 15u) & ~15u;
    int ri = r0, ji = 0;  // the copies' walk
    const uint8_t* pi = ri < R ? row_geom<T>(A, ri).base : nullptr;
    uint32_t si = 0, sc = 0, phase = 0;
    auto issue = [&]() {
        if (ri >= R) return;
        if (lane == 0) {
            const uint32_t bytes = ji == nb - 1 ? last_bytes : (uint32_t)(kBlkTok * sizeof(T));
            const uint32_t bar = bar0 + si * (kScanWarps * 8u);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            if ((long long)ri * nb + ji != A.debug_skip_blk)  // (test hook: a copy that never comes)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(slot0 + si * slot_bytes),
                             "l"(pi), "r"(bytes), "r"(bar)
                             : "memory");
        }
        pi += kBlkTok * sizeof(T);
        if (++ji == nb) {
            ji = 0;
            ri += W;
            if (ri < R) pi = row_geom<T>(A, ri).base;
        }
        if (++si == (uint32_t)S) si = 0;
    };
    for (int i = 0; i < S; ++i) issue();

    const RowPlan pl = row_plan(A.params);
    const bool want_lse = A.want_lse != 0;
    bool failed = false;
    int r = r0, j = 0;
    for (; r < R && !failed; r += W) {
        ThreadStats st;
        stats_reset(st, pl.c2);
        for (j = 0; j < nb; ++j) {
            if (!ring_wait(bar0 + sc * (kScanWarps * 8u), phase, A.timeout_ns)) {
                failed = true;
                break;
            }
            float v[2][16];
            load_half<T, true>(slot0 + sc * slot_bytes, 0, 0, v[0]);
            load_half<T, true>(slot0 + sc * slot_bytes, 0, 1, v[1]);
            __syncwarp();  // the block is in registers: its slot may be filled again
            issue();
            if (++sc == (uint32_t)S) { sc = 0; phase ^= 1u; }
            const int left = A.V - j * kBlkTok - lane * kGrpTok;
            if (j == nb - 1 && left < kGrpTok) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (group_pos<T>(h, i, true) >= left) v[h][i] = -INFINITY;
            }
            const float mt = group_max(v);
            st.mx = max_nan(st.mx, mt);
            keys[j * 32 + lane] = (uint16_t)(zkey(mt) >> 16);
            if (want_lse) lse32(st, v, mt, pl.c2);
        }
        if (failed) break;
        const float m = warp_max_nan(st.mx);
        float ls = 0.0f;
        if (want_lse) {
            const float s = st.s.x + st.s.y;
            ls = (s > 0.0f && m == m) ? s * ex2_approx(__fmul_rn(st.R - m, pl.c2)) : 0.0f;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, d);
        }
        const RowGeom q = row_geom<T>(A, r);
        int n = 0;
        if (m == m && m < INFINITY && m > -INFINITY) {
            // ---- a key that at least k of the group keys reach
            __syncwarp();
            uint32_t v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0;
            for (int i = 0; i < nb; i += 8) {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (i + e < nb) v[e] = max(v[e], (uint32_t)keys[(i + e) * 32 + lane]);
            }
            uint32_t tk = kth_of_maxima(v, pl.k);
            if (tk == 0) {  // fewer than k of the maxima are alive: over all keys
                auto reach = [&](uint32_t key) {
                    int c = 0;
                    for (int i = 0; i < nb; ++i) c += (uint32_t)keys[i * 32 + lane] >= key ? 1 : 0;
                    return __reduce_add_sync(0xffffffffu, c);
                };
                uint32_t hi = 0x10000u;
                tk = kDeadKey16 + 1u;
                if (reach(tk) >= pl.k)
                    while (hi - tk > 1u) {
                        const uint32_t mid = (tk + hi) >> 1;
                        if (reach(mid) >= pl.k) tk = mid;
                        else hi = mid;
                    }
            }
            // ---- the groups that reach it, read again: their tokens at or above it
            const float tf = fmaxf(zkey_to_float(tk << 16), -FLT_MAX);
            const uint32_t tk2 = zkey(tf) >> 16;
            const int id0 = A.idx_base + q.g * A.V;
            int nl = 0;
            auto flush = [&]() {
                __syncwarp();
                for (int i = 0; i < nl; i += 8) {
                    int tok[8];
                    float z[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) tok[e] = i + e < nl ? (int)list[i + e] * kGrpTok + lane : A.V;
#pragma unroll
                    for (int e = 0; e < 8; ++e) z[e] = tok[e] < A.V ? raw_logit<T>(q.base, tok[e]) : -INFINITY;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const uint32_t hb = __ballot_sync(0xffffffffu, z[e] >= tf);
                        const int at = n + __popc(hb & ((1u << lane) - 1u));
                        if (z[e] >= tf && at < kLocalCap) sel[at] = make_ck(z[e], id0 + tok[e]);
                        n += __popc(hb);
                    }
                }
                __syncwarp();
                nl = 0;
            };
            for (int i = 0; i < nb; ++i) {
                const bool hit = (uint32_t)keys[i * 32 + lane] >= tk2;
                const uint32_t hb = __ballot_sync(0xffffffffu, hit);
                if (hit) list[nl + __popc(hb & ((1u << lane) - 1u))] = (uint16_t)(i * 32 + lane);
                nl += __popc(hb);
                if (nl > kLocalCap - 32) flush();
            }
            if (nl) flush();
            if (n > kLocalCap) {  // (many equal values): the exact search, at the end
                if (lane == 0) {
                    write_failed(A, q.b, q.g);  // (should a wait of another warp run out)
                    A.deferred[r] = (8u << 24) | (blockIdx.x + 1u);
                    sh.defer = 1;
                }
                continue;
            }
        }
        // ---- the record, best candidate first
        uint8_t* rec = A.packed + (int64_t)q.g * A.packed_seg_stride + (int64_t)q.b * A.packed_row_stride;
        uint64_t* ent = reinterpret_cast<uint64_t*>(rec + kRecordHdrBytes);
        const int nk = min(n, pl.k);
        for (int i0 = 0; i0 < n; i0 += 96) {  // three candidates of a lane at a time
            uint64_t c[3];
            int rank[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                c[e] = i0 + 32 * e + lane < n ? sel[i0 + 32 * e + lane] : ~0ull;
                rank[e] = 0;
            }
            for (int i = 0; i < n; i += 4) {
                uint64_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) o[e] = i + e < n ? sel[i + e] : 0ull;
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int f = 0; f < 3; ++f) rank[f] += o[e] > c[f] ? 1 : 0;
            }
#pragma unroll
            for (int e = 0; e < 3; ++e)
                if (i0 + 32 * e + lane < n && rank[e] < nk) ent[rank[e]] = c[e];
        }
        if (lane == 0) {
            PackedHdr h;
            h.m = m; h.lse_s = ls; h.count = (uint32_t)nk;
            h.flags = n > pl.k ? 1u : 0u;
            h.bound = -INFINITY;
            h.pad[0] = h.pad[1] = h.pad[2] = 0;
            memcpy(rec, &h, sizeof h);
        }
        __syncwarp();
    }
    if (failed) {
        // a wait ran out: the copies still in flight (all but the one the test hook withheld) get the same bounded wait
        if (lane == 0) atomicExch(A.dev_error, BORN_ERR_DEVICE_TIMEOUT);
        for (int x = r + lane * W; x < R; x += 32 * W) {
            const RowGeom q = row_geom<T>(A, x);
            write_failed(A, q.b, q.g);
        }
        while (r < R && (r != ri || j != ji)) {
            if ((long long)r * nb + j != A.debug_skip_blk) ring_wait(bar0 + sc * (kScanWarps * 8u), phase, A.timeout_ns);
            if (++sc == (uint32_t)S) { sc = 0; phase ^= 1u; }
            if (++j == nb) { j = 0; r += W; }
        }
    }
    if (cta_sync_or(failed ? 1 : 0)) return;
    if (sh.defer == 0) return;  // (uniform)
    for (int w = 0; w < kScanWarps; ++w)
        for (int x = w * (int)gridDim.x + (int)blockIdx.x; x < R; x += W) {
            const uint32_t owner = __ldcg(&A.deferred[x]);
            if ((owner & 0xFFFFFFu) != (uint32_t)blockIdx.x + 1u) continue;
            cta_sync();
            if (tid == 0) {
                A.deferred[x] = 0;
                atomicAdd(A.dev_error + 1, 1);
                atomicAdd(A.dev_error + 8 + (owner >> 24), 1);
            }
            fallback_row<T>(A, sh, smem, x);
            cta_sync();
        }
}

}  // namespace born
