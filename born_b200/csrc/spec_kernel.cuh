// Speculative-decoding verification: accept/reject of K draft tokens per sequence and the
// resampling draw from the residual distribution max(0, p - q), in two launches.
//
// Launch 1 (spec_mass_kernel) treats every row of the call on its own -- (K+1) target rows
// and K draft rows per sequence -- and deals the 1024-token blocks of all rows to all warps of the
// grid.  A warp streams its blocks through its own ring (warp_ring.cuh) and leaves, per block, the
// block maximum and the exact fixed-point mass of the block relative to it.
//
// Launch 2 (spec_draw_kernel) gives every sequence a few CTAs.  Each of them folds the
// block results into row maxima and row totals (one rescale per block), runs the accept tests
//     u * q(x) < p(x)   <=>   (u * wq_x) * S_p < wp_x * S_q
// and so knows the first rejecting position (or that the bonus token is due).  Only that
// position is drawn: the warps of the CTAs share its blocks, leave the block sums of the
// residual masses in scratch, and the last CTA to finish (atomic ticket, no spinning) picks
// the block the target falls into, scans inside it and writes the sequence's outputs.
//
// The row arithmetic keeps the reference's shape -- maximum, exp of the shifted logits, sum
// (born: internal/autodiff/ops/softmax.go:214-238) -- with integer masses in place of the
// float32 running sum so that the result does not depend on the order of accumulation.
#pragma once
#include <string.h>
#include "../../include/born_sampler.h"
#include "spec.cuh"
#include "scan_common.cuh"

namespace born {

constexpr int kSpecThreads = 256;
constexpr int kSpecStages = 3;         // blocks in flight per warp of the first launch
constexpr int kSpecMassBlock = 1024;   // tokens per mass block, aligned to the row start
constexpr int kSpecMaxBlocks = 512;    // => vocab <= 524,288 on this path
constexpr int kSpecMaxRows = 2 * BORN_MAX_DRAFT + 1;
constexpr int kRowBadToken = 5;
static_assert(kSpecMassBlock == kBlkTok, "a mass block is what a warp streams at a time");

struct BlockMass {  // result of one 1024-token block
    float m;               // block maximum (NaN if the block holds one)
    uint32_t pad;
    unsigned long long M;  // sum of the fixed-point masses relative to m
};
static_assert(sizeof(BlockMass) == 16, "BlockMass size");

// Scratch of one call: per-sequence tickets (zero between launches), chunk sums of the draw,
// block results of every row.
struct SpecScratchLayout {
    size_t tickets, csum, blocks, total;
};
inline SpecScratchLayout spec_scratch_layout(int B, int K, int V) {
    SpecScratchLayout L;
    const size_t nblk = (size_t)(V + kSpecMassBlock - 1) / kSpecMassBlock;
    size_t off = 0;
    L.tickets = off; off += ((size_t)B * 4 + 255) / 256 * 256;
    L.csum = off; off += ((size_t)B * nblk * 8 + 255) / 256 * 256;
    L.blocks = off; off += (size_t)B * (2 * K + 1) * nblk * sizeof(BlockMass);
    L.total = off;
    return L;
}

struct SpecKernelArgs {
    const float* target;
    const float* draft;
    const int32_t* draft_tok;
    const float* u_accept;
    const float* u_resample;
    int32_t* accept_len;
    int32_t* out_tok;
    int32_t* status;
    uint32_t* tickets;
    unsigned long long* csum;
    BlockMass* blocks;
    int* dev_error;
    int B, K, V, target_rows;
    float inv_T;
    int tma;
};

// Weight of token i in the draw: residual max(0, p - q) or the plain mass of p.
struct DrawCtx {
    int residual;  // 1: max(0, p_i - q_i); 0: mass of p_i
    float mp, mq, inv_T, invSp, invSq;
};
__device__ __forceinline__ void draw_weight2(const DrawCtx& D, float2 zp, float2 zq, uint64_t& w0, uint64_t& w1) {
    if (D.residual) {
        const float2 it = make_float2(D.inv_T, D.inv_T);
        const float2 xp = __fmul2_rn(__fadd2_rn(zp, make_float2(-D.mp, -D.mp)), it), xq = __fmul2_rn(__fadd2_rn(zq, make_float2(-D.mq, -D.mq)), it);
        const float2 pi = __fmul2_rn(exp_det2(xp), make_float2(D.invSp, D.invSp)), qi = __fmul2_rn(exp_det2(xq), make_float2(D.invSq, D.invSq));
        // (exp_det2 returns 2^-115 where exp_det returns 0: far below half a unit of the result either way)
        w0 = __float2ull_rn(__fmul_rn(fmaxf(__fsub_rn(pi.x, qi.x), 0.0f), 1099511627776.0f));
        w1 = __float2ull_rn(__fmul_rn(fmaxf(__fsub_rn(pi.y, qi.y), 0.0f), 1099511627776.0f));
    } else {
        mass2_of(zp, D.mp, D.inv_T, w0, w1);
    }
}

// ------------------------------------------------------------------ launch 1: block masses
// The blocks of all rows form one sequence, dealt to all warps of the grid in contiguous, equal
// ranges; a warp streams its blocks through its own ring (warp_ring.cuh) and never meets another
// warp.  Bound by the fp32 pipe and issue slots of the deterministic exp (13 instructions per token
// in packed form, 27 in scalar), then by HBM: one pass, every logit read once.  32 sequences of five
// draft tokens over 128256-token rows (180.6 MB): 55.6 us, both launches, against 94 with tiles of 8192
// tokens behind a block-wide barrier each, which leave the pipes idle while the warps meet.
struct MassShared {
    unsigned long long bars[kSpecStages * (kSpecThreads / 32)];
};

template <bool kAligned>
__global__ void __launch_bounds__(kSpecThreads, 2) spec_mass_kernel(const __grid_constant__ SpecKernelArgs A) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ MassShared sh;
    constexpr int kSlot = ring_slot_bytes(4, kAligned), kWarps = kSpecThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int V = A.V, nblk = (V + kSpecMassBlock - 1) / kSpecMassBlock;
    const int ntarget = A.B * A.target_rows;
    const int64_t total = (int64_t)(ntarget + A.B * A.K) * nblk;
    const int64_t nw = (int64_t)gridDim.x * kWarps, w = (int64_t)blockIdx.x * kWarps + warp;
    const int64_t t0 = w * total / nw;
    const int n = (int)((w + 1) * total / nw - t0);
    const uint32_t slot0 = smem_u32(smem) + warp * kSlot, bar0 = smem_u32(&sh.bars[warp]);
    if (lane == 0)
        for (int s = 0; s < kSpecStages; ++s) mbar_init(reinterpret_cast<uint64_t*>(&sh.bars[s * kWarps + warp]), 1);
    mbar_fence_init();
    grid_launch_dependents();  // (the second launch waits for this grid's end before it reads a result)
    __syncwarp();
    auto row_ptr = [&](int row) {
        return reinterpret_cast<const uint8_t*>(row < ntarget ? A.target + (int64_t)row * V : A.draft + (int64_t)(row - ntarget) * V);
    };
    // two cursors over the warp's blocks: the copy's runs kSpecStages ahead of the reader's
    int row_i = (int)(t0 / nblk), blk_i = (int)(t0 - (int64_t)row_i * nblk), row = row_i, blk = blk_i;
    const uint8_t* ptr_i = row_ptr(row_i);
    int issued = 0;
    auto issue = [&]() {
        const int s = issued % kSpecStages;
        if (lane == 0)
            ring_issue(slot0 + (uint32_t)(s * kWarps * kSlot), bar0 + (uint32_t)(s * kWarps * 8), ptr_i, blk_i * kSpecMassBlock,
                       min(kSpecMassBlock, V - blk_i * kSpecMassBlock), 4);
        if (++blk_i == nblk) {
            blk_i = 0;
            ++row_i;
            if (issued + 1 < n) ptr_i = row_ptr(row_i);
        }
        ++issued;
    };
    for (int i = 0; i < min(kSpecStages, n); ++i) issue();
    int s = 0;
    uint32_t phase = 0;
    for (int i = 0; i < n; ++i) {
        if (!ring_wait(bar0 + (uint32_t)(s * kWarps * 8), phase, kMbarTimeoutNs)) {
            // a copy never came: say so, and do not leave while others are in flight into this CTA
            if (lane == 0) atomicExch(A.dev_error, 2);
            for (int j = i + 1; j < issued; ++j)
                ring_wait(bar0 + (uint32_t)((j % kSpecStages) * kWarps * 8), (uint32_t)(j / kSpecStages) & 1u, kMbarTimeoutNs);
            return;
        }
        const uint32_t slot = slot0 + (uint32_t)(s * kWarps * kSlot);
        uint32_t mis = 0;
        if constexpr (!kAligned) mis = (uint32_t)reinterpret_cast<uintptr_t>(row_ptr(row)) & 15u;  // (blocks are a multiple of 16 bytes)
        float v[2][16];
        load_half<float, kAligned>(slot, mis, 0, v[0]);
        load_half<float, kAligned>(slot, mis, 1, v[1]);
        __syncwarp();  // the block is in registers: its slot may be filled again
        if (issued < n) issue();
        const int left = V - blk * kSpecMassBlock - lane * kGrpTok;
        if (left < kGrpTok && blk == nblk - 1) {  // the row ends inside this group: nothing beyond it counts
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    if (group_pos<float>(h, k, kAligned) >= left) v[h][k] = -INFINITY;
        }
        float mc = -INFINITY;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 16; ++k) mc = max_nan(mc, v[h][k]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) mc = max_nan(mc, __shfl_xor_sync(0xffffffffu, mc, d));
        uint64_t M0 = 0, M1 = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
                uint64_t q0, q1;
                mass2_of(make_float2(v[h][k], v[h][k + 1]), mc, A.inv_T, q0, q1);
                M0 += q0;
                M1 += q1;
            }
        uint64_t Mc = M0 + M1;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) Mc += shfl_xor_u64(Mc, d);
        if (lane == 0) {
            BlockMass r;
            r.m = mc; r.pad = 0; r.M = Mc;
            A.blocks[(size_t)row * nblk + blk] = r;
        }
        if (++blk == nblk) { blk = 0; ++row; }
        if (++s == kSpecStages) { s = 0; phase ^= 1u; }
    }
}

// ------------------------------------------------------------------ launch 2: accept and draw
// A chain of dependent steps with little to stream (one position of every sequence): what bounds it
// is latency.  Hence no tiles and no block-wide sums -- the loads of a warp's blocks leave together,
// a block's sum stays inside its warp -- the operands of the accept tests are fetched before the
// block results are waited for, and the launch itself overlaps the first one's end (programmatic
// dependent launch: everything in front of grid_dependency_wait reads only the caller's inputs).
// Four sequences of four draft tokens, 18917-token rows: 12.7 us for both launches, 26.5 with block-wide steps.
struct DrawShared {
    unsigned long long rowS[kSpecMaxRows];   // row totals of the fixed-point masses
    unsigned long long csum[kSpecMaxBlocks];
    float rowm[kSpecMaxRows];                // row maxima (NaN if the row holds one)
    int accept[BORN_MAX_DRAFT];
    int pstat[BORN_MAX_DRAFT + 1];
    int last;
};

// Sum of the draw weights of one 1024-token block, by the warp.  All loads leave before the first use.
__device__ __forceinline__ uint64_t spec_block_sum(const DrawCtx& D, const float* rowp, const float* rowq, int tok0, int V, int vec) {
    const int lane = threadIdx.x & 31;
    float4 p[8], q[8];
    if (vec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tok0 + 4 * (lane + 32 * i);
            p[i] = e < V ? __ldg(reinterpret_cast<const float4*>(rowp + e)) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = tok0 + 4 * (lane + 32 * i);
            q[i] = (D.residual && e < V) ? __ldg(reinterpret_cast<const float4*>(rowq + e)) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float a[4], b[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int e = tok0 + lane + 32 * (4 * i + k);
                a[k] = e < V ? __ldg(rowp + e) : -INFINITY;
                b[k] = (D.residual && e < V) ? __ldg(rowq + e) : -INFINITY;
            }
            p[i] = make_float4(a[0], a[1], a[2], a[3]);
            q[i] = make_float4(b[0], b[1], b[2], b[3]);
        }
    }
    uint64_t s0 = 0, s1 = 0;  // (a token beyond the row is -inf on both sides: weight 0)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint64_t a, b;
        draw_weight2(D, make_float2(p[i].x, p[i].y), make_float2(q[i].x, q[i].y), a, b);
        s0 += a; s1 += b;
        draw_weight2(D, make_float2(p[i].z, p[i].w), make_float2(q[i].z, q[i].w), a, b);
        s0 += a; s1 += b;
    }
    uint64_t s = s0 + s1;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += shfl_xor_u64(s, d);
    return s;
}

__global__ void __launch_bounds__(kSpecThreads, 2) spec_draw_kernel(const __grid_constant__ SpecKernelArgs A) {
    __shared__ DrawShared sh;
    constexpr int kWarps = kSpecThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = blockIdx.x, nparts = gridDim.x, b = blockIdx.y;
    const int K = A.K, V = A.V, R = A.target_rows;
    const int nblk = (V + kSpecMassBlock - 1) / kSpecMassBlock;
    const int nrows = R + K;  // this sequence's rows: r < R target row r, else draft row r - R
    auto row_id = [&](int r) { return r < R ? b * R + r : A.B * R + b * K + (r - R); };

    // operands of the accept tests, one position per thread
    int x = -1;
    float zpx = 0.0f, zqx = 0.0f, ua = 0.0f;
    if (tid < K) {
        x = __ldg(A.draft_tok + (int64_t)b * K + tid);
        ua = __ldg(A.u_accept + (int64_t)b * K + tid);
        if (x >= 0 && x < V) {
            zpx = __ldg(A.target + ((int64_t)b * R + tid) * (int64_t)V + x);
            zqx = __ldg(A.draft + ((int64_t)b * K + tid) * (int64_t)V + x);
        }
    }
    grid_dependency_wait();

    // ---- row maxima and totals from the block results (every CTA of the sequence on its own):
    // one warp per row, the blocks of the row dealt out to its lanes and held in registers, so
    // that the block results are fetched once, all loads in flight together, and the warp
    // reduces by shuffles.
    for (int r = warp; r < nrows; r += kWarps) {
        constexpr int kPerLane = kSpecMaxBlocks / 32;  // 16 blocks per lane at most
        const BlockMass* rb = A.blocks + (size_t)row_id(r) * nblk;
        float bm[kPerLane];
        unsigned long long bM[kPerLane];
#pragma unroll
        for (int q = 0; q < kPerLane; ++q) {
            const int blk = lane + 32 * q;
            bm[q] = -INFINITY;
            bM[q] = 0;
            if (blk < nblk) {
                const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(rb + blk));
                bm[q] = __uint_as_float(raw.x);
                bM[q] = ((unsigned long long)raw.w << 32) | raw.z;
            }
        }
        float m = -INFINITY;
#pragma unroll
        for (int q = 0; q < kPerLane; ++q) m = max_nan(m, bm[q]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, d));
        unsigned long long S = 0;
        if (m == m && m > -INFINITY && m < INFINITY) {
#pragma unroll
            for (int q = 0; q < kPerLane; ++q) {
                if (bm[q] == -INFINITY) continue;
                const float ef = exp_det<false>(scaled_shift(bm[q], m, A.inv_T));
                S += __double2ull_rn(__dmul_rn(__ull2double_rn(bM[q]), (double)ef));
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) S += shfl_xor_u64(S, d);
        }
        if (lane == 0) {
            sh.rowm[r] = m;
            sh.rowS[r] = S;
        }
    }
    __syncthreads();
    auto row_status = [&](int r) {
        const float m = sh.rowm[r];
        if (m != m) return (int)BORN_ROW_NAN;
        if (m == INFINITY) return (int)BORN_ROW_POS_INF;
        if (m == -INFINITY) return (int)BORN_ROW_ALL_MASKED;
        return (int)BORN_ROW_OK;
    };
    const bool dev_failed = *reinterpret_cast<volatile int*>(A.dev_error) != 0;  // launch 1 gave up on a copy
    if (tid < K) {
        const int j = tid;
        int st = row_status(j);
        if (st == BORN_ROW_OK) st = row_status(R + j);
        if (dev_failed) st = 100 + BORN_ERR_DEVICE_TIMEOUT;
        int acc = 0;
        if (st == BORN_ROW_OK) {
            if (x < 0 || x >= V) st = kRowBadToken;
            else {
                const uint64_t wp = mass_of<false>(scaled_shift(zpx, sh.rowm[j], A.inv_T));
                const uint64_t wq = mass_of<false>(scaled_shift(zqx, sh.rowm[R + j], A.inv_T));
                const double lhs = __dmul_rn(__dmul_rn((double)ua, __ull2double_rn(wq)), __ull2double_rn(sh.rowS[j]));
                const double rhs = __dmul_rn(__ull2double_rn(wp), __ull2double_rn(sh.rowS[R + j]));
                acc = lhs < rhs;
            }
        }
        sh.accept[j] = acc;
        sh.pstat[j] = st;
    }
    if (tid == K) sh.pstat[K] = (R > K) ? (dev_failed ? 100 + BORN_ERR_DEVICE_TIMEOUT : row_status(K)) : BORN_ROW_OK;
    __syncthreads();

    // ---- the outcome for the sequence (same in every thread of every CTA of the sequence)
    int len = K, seq_status = BORN_ROW_OK, jstar = -1;
    DrawCtx D;
    D.residual = 0; D.inv_T = A.inv_T; D.mp = 0.0f; D.mq = 0.0f; D.invSp = 0.0f; D.invSq = 0.0f;
    for (int i = 0; i < K; ++i) {
        if (sh.pstat[i] != BORN_ROW_OK) { seq_status = sh.pstat[i]; len = i; break; }
        if (!sh.accept[i]) { len = i; jstar = i; D.residual = 1; break; }
    }
    if (len == K && seq_status == BORN_ROW_OK && R > K) {
        if (sh.pstat[K] != BORN_ROW_OK) seq_status = sh.pstat[K];
        else jstar = K;
    }
    auto write_outputs = [&](int token) {  // one thread
        int32_t* out = A.out_tok + (int64_t)b * (K + 1);
        for (int i = 0; i <= K; ++i) out[i] = i < len ? __ldg(A.draft_tok + (int64_t)b * K + i) : -1;
        if (jstar >= 0) out[jstar] = token;
        A.accept_len[b] = len;
        A.status[b] = seq_status;
    };
    if (jstar < 0) {  // nothing to draw
        if (part == 0 && tid == 0) write_outputs(-1);
        return;
    }
    const float* rowp = A.target + ((int64_t)b * R + jstar) * (int64_t)V;
    const float* rowq = D.residual ? A.draft + ((int64_t)b * K + jstar) * (int64_t)V : rowp;
    D.mp = sh.rowm[jstar];
    if (D.residual) {
        D.mq = sh.rowm[R + jstar];
        D.invSp = __double2float_rn(__ddiv_rn(1099511627776.0, __ull2double_rn(sh.rowS[jstar])));
        D.invSq = __double2float_rn(__ddiv_rn(1099511627776.0, __ull2double_rn(sh.rowS[R + jstar])));
    }

    // ---- sums of the draw weights per block: the blocks are dealt to all warps of the sequence's CTAs
    unsigned long long* csum_g = A.csum + (size_t)b * nblk;
    for (int c = part * kWarps + warp; c < nblk; c += nparts * kWarps) {
        const uint64_t s = spec_block_sum(D, rowp, rowq, c * kSpecMassBlock, V, A.tma);
        if (lane == 0) csum_g[c] = s;
    }

    // ---- ticket: the last CTA of the sequence picks the block and the token
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const uint32_t tk = atomicAdd(&A.tickets[b], 1u);
        sh.last = (tk == (uint32_t)nparts - 1);
        if (sh.last) A.tickets[b] = 0;  // ready for the next launch
        __threadfence();
    }
    __syncthreads();
    if (!sh.last) return;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (attempt == 0) {
            for (int c = tid; c < nblk; c += kSpecThreads) sh.csum[c] = __ldcg(&csum_g[c]);
        } else {  // the residual vanished in fp32: draw from the plain masses of p instead
            D.residual = 0;
            for (int c = warp; c < nblk; c += kWarps) {
                const uint64_t s = spec_block_sum(D, rowp, rowq, c * kSpecMassBlock, V, A.tma);
                if (lane == 0) sh.csum[c] = s;
            }
        }
        __syncthreads();
        // every warp works out the block the target falls into; lanes take runs of blocks
        const int per = (nblk + 31) / 32;
        uint64_t loc = 0;
        for (int i = 0; i < per; ++i) {
            const int c = lane * per + i;
            loc += c < nblk ? sh.csum[c] : 0ull;
        }
        uint64_t incl = loc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t up = shfl_up_u64(incl, d);
            if (lane >= d) incl += up;
        }
        const uint64_t W = shfl_u64(incl, 31);
        if (W == 0) {
            if (D.residual) continue;  // (uniform: the same sums in every thread)
            if (tid == 0) write_outputs(-1);
            return;
        }
        const float u = __ldg(A.u_resample + (int64_t)b * (K + 1) + jstar);
        uint64_t t = __double2ull_rz(__dmul_rn((double)u, __ull2double_rn(W)));
        if (t > W - 1) t = W - 1;
        const int hl = __ffs(__ballot_sync(0xffffffffu, incl > t)) - 1;  // (W > t: some lane's run crosses)
        uint64_t acc = incl - loc;
        int c = lane * per;
        if (lane == hl)
            for (; acc + sh.csum[c] <= t; ++c) acc += sh.csum[c];
        c = __shfl_sync(0xffffffffu, c, hl);
        t -= shfl_u64(acc, hl);
        // inside the block: warp w takes tokens 128 w .. 128 w + 127, four consecutive ones per lane
        const int e0 = c * kSpecMassBlock + 128 * warp + 4 * lane;
        float p[4], q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            p[k] = e0 + k < V ? __ldg(rowp + e0 + k) : -INFINITY;
            q[k] = e0 + k < V ? __ldg(rowq + e0 + k) : -INFINITY;
        }
        uint64_t w[4];
        draw_weight2(D, make_float2(p[0], p[1]), make_float2(q[0], q[1]), w[0], w[1]);
        draw_weight2(D, make_float2(p[2], p[3]), make_float2(q[2], q[3]), w[2], w[3]);
        const uint64_t mine = w[0] + w[1] + w[2] + w[3];
        incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t up = shfl_up_u64(incl, d);
            if (lane >= d) incl += up;
        }
        __syncthreads();  // (the sums have been read)
        if (lane == 31) sh.csum[warp] = incl;
        __syncthreads();
        for (int i = 0; i < warp; ++i) incl += sh.csum[i];
        if (incl > t && incl - mine <= t) {
            uint64_t at = incl - mine;
            int k = 0;
            for (; k < 3 && at + w[k] <= t; ++k) at += w[k];
            write_outputs(e0 + k);
        }
        return;
    }
}

inline size_t spec_mass_smem_bytes(bool aligned) { return (size_t)kSpecStages * (kSpecThreads / 32) * ring_slot_bytes(4, aligned); }

// raises the dynamic shared-memory limit of the first kernel; once per device, at handle creation
inline cudaError_t spec_attrs_all() {
    cudaError_t e = cudaFuncSetAttribute(spec_mass_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)spec_mass_smem_bytes(true));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(spec_mass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)spec_mass_smem_bytes(false));
}

// returns 0 or a cudaError_t; `num_sms` sizes the launches
inline int launch_spec(SpecKernelArgs A, int num_sms, cudaStream_t st) {
    if (A.V > kSpecMaxBlocks * kSpecMassBlock) return (int)cudaErrorInvalidValue;
    A.tma = ((uintptr_t)A.target % 16 == 0) && ((uintptr_t)A.draft % 16 == 0) && (((int64_t)A.V * 4) % 16 == 0);
    const int nblk = (A.V + kSpecMassBlock - 1) / kSpecMassBlock;
    const int64_t blocks = (int64_t)A.B * (A.target_rows + A.K) * nblk;
    constexpr int kWarps = kSpecThreads / 32;
    // one CTA per eight blocks until the GPU is full: two per SM, every warp an equal share
    const int64_t want = (blocks + kWarps - 1) / kWarps;
    const unsigned grid = (unsigned)(want < 2 * num_sms ? want : 2 * num_sms);
    if (A.tma) spec_mass_kernel<true><<<grid, kSpecThreads, spec_mass_smem_bytes(true), st>>>(A);
    else spec_mass_kernel<false><<<grid, kSpecThreads, spec_mass_smem_bytes(false), st>>>(A);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    // CTAs per sequence: as many as fill the GPU twice over, each with at least a block per warp
    int parts = 2 * num_sms / A.B;
    if (parts > (nblk + kWarps - 1) / kWarps) parts = (nblk + kWarps - 1) / kWarps;
    if (parts < 1) parts = 1;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3((unsigned)parts, (unsigned)A.B, 1);
    cfg.blockDim = dim3(kSpecThreads, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, spec_draw_kernel, A);
}

}  // namespace born
