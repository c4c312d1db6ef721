// scan_kernel: the streaming pass of the sampler.
//
// One launch does penalties -> grammar mask -> row max / log-sum-exp -> group keys (or whole-row
// mass blocks) and -- in the CTA that completes a row -- the selection and the inverse-CDF draw
// (finish.cuh).  Every logit crosses HBM once; the finish reads the few groups of 32 tokens that
// can matter a second time.
//
// The loop over the blocks knows no thresholds and keeps no candidates: per block of 1024 tokens a
// warp waits for its copy, reads 32 values per lane, folds them into a running maximum and an
// online log-sum-exp, and stores one 16-bit key per lane.  The k-th largest group maximum is
// reached by at least k tokens, so the groups that reach it hold the k best tokens; a group below
// running maximum + delta holds no min-p survivor; and so on for every route -- decided once, in the
// finish, when everything is known.  (Thresholds that tighten while the row streams, with hits pushed
// into buffers, send nine iterations in ten down the hit path for top-k.)
//
// 8 warps per CTA, two CTAs per SM, no producer warp: warp_ring.cuh.  What bounds it on long
// rows is HBM; on one-block-per-warp rows the chain launch -> history list -> copy -> reduction ->
// finish.
//
// Token histories.  At the start of a segment the CTA builds, in shared memory, the list of the
// row's distinct history tokens that fall into the segment, grouped by block (hist_build).  A warp
// applies the entries of a block to its slot before it reads it (hist_apply), and leaves the
// penalised values in the list for the finish.
//
// The greedy branch keeps the reference's tie rule -- the first maximum wins
// (born: internal/nn/cross_entropy.go:241-251); the row arithmetic keeps its structure
// (maximum, exp of the shifted logits, sum: internal/autodiff/ops/softmax.go:214-238).
#pragma once
#include <float.h>
#include "scan_common.cuh"
#include "finish.cuh"

namespace born {

struct ThreadStats {
    float mx;   // running maximum (NaN-propagating)
    float R;    // reference of the online log-sum-exp (z domain)
    float nRc;  // -R * c2
    float2 s;   // two partial sums of 2^((z - R) * c2)
};
__device__ __forceinline__ void stats_reset(ThreadStats& st, float c2) {
    st.mx = -INFINITY;
    st.R = -1e30f;
    st.nRc = 1e30f * c2;
    st.s = make_float2(0.0f, 0.0f);
}
__device__ __forceinline__ void lse_reference(ThreadStats& st, float mt, float c2) {
    if (mt > st.R && mt < INFINITY) {
        const float f = ex2_approx(__fmul_rn(st.R - mt, c2));
        st.s = __fmul2_rn(st.s, make_float2(f, f));
        st.R = mt;
        st.nRc = -mt * c2;
    }
}
// Online log-sum-exp of 32 values: the reference moves at most once (to their maximum mt), then
// the terms are formed two at a time with packed fp32x2 operations in four chains.
__device__ __forceinline__ void lse32(ThreadStats& st, const float (&v)[2][16], float mt, float c2) {
    lse_reference(st, mt, c2);
    const float2 cc = make_float2(c2, c2), rr = make_float2(st.nRc, st.nRc);
    float2 s[4];
    s[0] = st.s;
    s[1] = s[2] = s[3] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const float2 t = __ffma2_rn(make_float2(v[h][i], v[h][i + 1]), cc, rr);
            s[(i >> 1) & 3] = __fadd2_rn(s[(i >> 1) & 3], make_float2(ex2_approx(t.x), ex2_approx(t.y)));
        }
    st.s = __fadd2_rn(__fadd2_rn(s[0], s[1]), __fadd2_rn(s[2], s[3]));
}

// Maximum of a lane's group (NaN-propagating).
__device__ __forceinline__ float group_max(const float (&v)[2][16]) {
    float m8[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        m8[i] = max_nan(max3_nan(v[i >> 2][4 * (i & 3)], v[i >> 2][4 * (i & 3) + 1], v[i >> 2][4 * (i & 3) + 2]), v[i >> 2][4 * (i & 3) + 3]);
    return max3_nan(max3_nan(m8[0], m8[1], m8[2]), max3_nan(m8[3], m8[4], m8[5]), max_nan(m8[6], m8[7]));
}

// ---- token history -----------------------------------------------------------------------------
// Penalties touch at most BORN_MAX_HISTORY tokens of a row.  The global read of the ids is the only
// memory round trip of the build; for a CTA's first row it leaves before the CTA's first copies
// (behind them it would wait in the memory system's queues).
constexpr int kHistPer = BORN_MAX_HISTORY / kThreads;  // history ids per thread

__device__ __forceinline__ void hist_ids(const ScanArgs& A, int b, int (&ids)[kHistPer]) {
    // the ids do not wait for the length: both reads leave together, the length cuts afterwards.  (Not
    // through the read-only path: the launch before this one, which may still have been running when this
    // one began, appends to the ring that the generate loop passes here.)
    const int cap = min(A.history_stride, (int)BORN_MAX_HISTORY);
    const int32_t* gh = A.history + (int64_t)b * A.history_stride;
#pragma unroll
    for (int r = 0; r < kHistPer; ++r) {
        const int p = (int)threadIdx.x + r * kThreads;
        ids[r] = p < cap ? __ldcg(gh + p) : -1;
    }
    const int len = A.history_len ? __ldcg(A.history_len + b) : cap;
#pragma unroll
    for (int r = 0; r < kHistPer; ++r)
        if ((int)threadIdx.x + r * kThreads >= len) ids[r] = -1;
}

// Shift that maps the blocks of a segment to the list's buckets.
__device__ __forceinline__ int hist_shift(int span) {
    int s = 0;
    while (((span - 1) >> s) >= kHistBuckets) ++s;
    return s;
}

// The list of the distinct history tokens of blocks [j0, j1) of the row, with their multiplicities,
// grouped by bucket.  What tells a token's first occurrence from its repeats: a bit per token of the
// segment, where the bits fit and are not crowded (one atomic per id; a repeat finds its token afterwards, by a table of list
// positions, and counts itself there), else a compare-and-swap into a hash table.  Chains of swaps
// bound the latter, 3.6 us for 512 ids with two CTAs on an SM.  256 rows, 512 ids, hash table -> bits:
// 32000 tokens fp32 18.9 -> 14.7 us, 128256 33.5 -> 30.4, 151936 39.5 -> 34.9; bf16 200000 45.9 -> 41.6.
// For a first occurrence the atomic on the bucket's counter counts the token and returns its place.  After one
// barrier every warp works out the bucket starts for itself (all of them write the same offsets) and
// stores its tokens.
__device__ __forceinline__ int hist_build(const ScanArgs& A, ScanShared& sh, uint8_t* smem, const int (&ids)[kHistPer], int g, int j0, int j1) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int lg = A.L.hash_lg, slots = 1 << lg, hs = hist_shift(j1 - j0);
    // (many ids on few words of bits queue up behind one another: 256 rows of 8192 tokens, 512 ids, take 15.1 us
    // with the hash table and 12.5 with bits, 4096 tokens with 1024 ids 16.4 and 23.4, 1000 with 512 12.4 and 18.7)
    const bool bits = (j1 - j0) * (kBlkTok / 8) + kHistPos * 2 <= A.L.hash_bytes && A.L.list_cap <= 64 * (j1 - j0);
    uint32_t* keys = reinterpret_cast<uint32_t*>(smem + A.L.hash);  // hash table: keys, multiplicities; or the bits
    uint32_t* mult = keys + slots;
    uint16_t* where = reinterpret_cast<uint16_t*>(keys + (j1 - j0) * (kBlkTok / 32));
    unsigned long long* list = reinterpret_cast<unsigned long long*>(smem + A.L.list);
    uint16_t* offs = reinterpret_cast<uint16_t*>(list + A.L.list_cap);
    if (bits) {
        for (int i = tid; i < (j1 - j0) * (kBlkTok / 128); i += kThreads) reinterpret_cast<uint4*>(keys)[i] = make_uint4(0u, 0u, 0u, 0u);
    } else {
        for (int i = tid; i < slots / 4; i += kThreads) {
            reinterpret_cast<uint4*>(keys)[i] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
            reinterpret_cast<uint4*>(mult)[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    if (tid < kHistBuckets / 4) sh.bcnt[tid] = make_uint4(0u, 0u, 0u, 0u);
    cta_sync();
    uint32_t* bcnt = reinterpret_cast<uint32_t*>(sh.bcnt);
    uint32_t tok[kHistPer];
    int at[kHistPer];   // first occurrence: the token's slot (hash table) or 0 (bits); -1: none; -2: a repeat
    uint32_t rank[kHistPer];
    int repeats = 0;
#pragma unroll
    for (int r = 0; r < kHistPer; ++r) {
        at[r] = -1;
        rank[r] = 0;
        tok[r] = 0;
        const int id = ids[r];
        if (id < 0) continue;
        tok[r] = (uint32_t)id;
        if (A.G > 1) {
            const int g2 = id / A.V;
            if (g2 != g) continue;  // another vocabulary segment's token
            tok[r] = (uint32_t)(id - g2 * A.V);
        }
        const int j = (int)(tok[r] / (uint32_t)kBlkTok);
        if (tok[r] >= (uint32_t)A.V || j < j0 || j >= j1) continue;  // (ids beyond the vocabulary are ignored)
        if (bits) {
            const uint32_t t = tok[r] - (uint32_t)j0 * (uint32_t)kBlkTok;
            at[r] = (smem_atom_or(&keys[t >> 5], 1u << (t & 31u)) >> (t & 31u)) & 1u ? -2 : 0;
            if (at[r] == -2) repeats = 1;
        } else {
            uint32_t slot = (tok[r] * 2654435761u) >> (32 - lg);
            for (int probe = 0; probe < slots; ++probe) {
                const uint32_t old = atomicCAS(&keys[slot], 0xFFFFFFFFu, tok[r]);
                if (old == 0xFFFFFFFFu) { at[r] = (int)slot; break; }
                if (old == tok[r]) { smem_red_add(&mult[slot], 1u); break; }  // a repeat
                slot = (slot + 1) & (uint32_t)(slots - 1);
            }
        }
        if (at[r] >= 0) rank[r] = smem_atom_add(&bcnt[(j - j0) >> hs], 1u);
    }
    cta_sync();
    const uint4 c = sh.bcnt[lane];
    const uint32_t tot = c.x + c.y + c.z + c.w;
    uint32_t incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += u;
    }
    const uint32_t n = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t e = incl - tot;
    offs[4 * lane] = (uint16_t)e;
    offs[4 * lane + 1] = (uint16_t)(e + c.x);
    offs[4 * lane + 2] = (uint16_t)(e + c.x + c.y);
    offs[4 * lane + 3] = (uint16_t)(e + c.x + c.y + c.z);
    if (lane == 0) offs[kHistBuckets] = (uint16_t)n;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kHistPer; ++r) {
        if (at[r] < 0) continue;
        const int i = offs[((int)(tok[r] / (uint32_t)kBlkTok) - j0) >> hs] + (int)rank[r];
        list[i] = ((unsigned long long)(bits ? 1u : mult[at[r]] + 1u) << 32) | tok[r];
        if (bits) where[(tok[r] * 2654435761u) >> 21] = (uint16_t)i;
    }
    if (cta_sync_or(repeats)) {
#pragma unroll
        for (int r = 0; r < kHistPer; ++r) {
            if (at[r] != -2) continue;
            int i = where[(tok[r] * 2654435761u) >> 21];
            if ((uint32_t)list[i] != tok[r]) {  // (another token with the same hash was stored later)
                i = offs[((int)(tok[r] / (uint32_t)kBlkTok) - j0) >> hs];
                while ((uint32_t)list[i] != tok[r]) ++i;
            }
            smem_red_add(reinterpret_cast<uint32_t*>(&list[i]) + 1, 1u);
        }
        cta_sync();
    }
    if (tid < kHistBuckets / 4) sh.bcnt[tid] = make_uint4(0u, 0u, 0u, 0u);  // (now the finish's map of candidates)
    return (int)n;
}
static_assert(kHistPos == 2048, "eleven bits of the hash");

// Mask bit of token `off` of the block in the slot (the mask words begin `mword` words into the mask
// area, the block's first bit `mbit` bits into them).
__device__ __forceinline__ bool slot_mask_bit(uint32_t marea, uint32_t mword, uint32_t mbit, int off) {
    const uint32_t bit = mbit + (uint32_t)off;
    uint32_t w;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(marea + 4u * (mword + (bit >> 5))) : "memory");
    return (w >> (bit & 31u)) & 1u;
}

// The history tokens of block j, by the warp that is about to read it.  fp32: the penalised value
// goes over the logit.  bf16 (a bf16 slot cannot hold it): the token is taken out of the block and
// its value joins the lane's statistics.  Either way the list entry becomes (penalised value,
// token): the finish adds the list to its candidates and skips the raw values.
template <typename T, bool kMask>
__device__ __forceinline__ void hist_apply(const ScanArgs& A, uint8_t* smem, const born_row_params& rp, int j, int bucket, uint32_t slot,
                                           uint32_t mis, uint32_t marea, uint32_t mword, uint32_t mbit, bool want_lse, float c2,
                                           ThreadStats& st) {
    unsigned long long* list = reinterpret_cast<unsigned long long*>(smem + A.L.list);
    const uint16_t* offs = reinterpret_cast<const uint16_t*>(list + A.L.list_cap);
    const int lane = threadIdx.x & 31;
    const int lo = offs[bucket], hi = offs[bucket + 1];
    if (lo == hi) return;
    bool wrote = false;
    for (int i = lo + lane; i < hi; i += 32) {
        const unsigned long long e = list[i];
        const int off = (int)(uint32_t)e - j * kBlkTok;
        if (off < 0 || off >= kBlkTok) continue;  // (a bucket may hold several blocks)
        const uint32_t a = slot + mis + (uint32_t)off * (uint32_t)sizeof(T);
        float z;
        if constexpr (sizeof(T) == 4) z = lds32f(a);
        else z = bf16_bits_to_f32(lds16u(a));
        float zp = penalise(rp, z, (int)(e >> 32));
        if constexpr (sizeof(T) == 4) asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(zp) : "memory");
        else asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)0xFF80u) : "memory");
        if constexpr (kMask)
            if (!slot_mask_bit(marea, mword, mbit, off)) zp = -INFINITY;
        if constexpr (sizeof(T) == 2) {
            st.mx = max_nan(st.mx, zp);
            if (want_lse) {
                lse_reference(st, zp, c2);
                st.s.x += ex2_approx(fmaf(zp, c2, st.nRc));
            }
        }
        list[i] = ((unsigned long long)__float_as_uint(zp) << 32) | (uint32_t)e;
        wrote = true;
    }
    if (wrote) fence_proxy_async();  // the slot is next written by a bulk copy
    __syncwarp();
}

// Device-resident history: the CTA that finished caller row b appends the sampled token to the
// row's ring (the next call reads the ring as its history), marks the row finished when the
// token is a stop token, and blanks the outputs of a row that had finished before.  One thread,
// after a barrier that follows the row's output writes.
__device__ __forceinline__ void ring_append(const ScanArgs& A, int b) {
    if (A.ring_finished[b]) {
        A.out_token[b] = -1;
        A.out_status[b] = BORN_ROW_FINISHED;
        if (A.out_prob) A.out_prob[b] = 0.0f;
        if (A.out_kept_count) A.out_kept_count[b] = 0;
        return;
    }
    const int tok = A.out_token[b];
    if (A.out_status[b] != BORN_ROW_OK || tok < 0) return;
    const int total = A.ring_total[b];
    A.ring[(int64_t)b * A.ring_cap + total % A.ring_cap] = tok;
    A.ring_total[b] = total + 1;
    A.ring_len[b] = min(total + 1, A.ring_cap);
    for (int i = 0; i < A.n_stop; ++i)
        if (A.stop_ids[i] == tok) A.ring_finished[b] = 1;
}

// ---- copies -------------------------------------------------------------------------------------
// First mask word of block j of virtual row (b, g) that is loaded, and the bits in front of the
// block's first one: the copy begins at the 16-byte granule of its word.
__device__ __forceinline__ void mask_pos(const ScanArgs& A, int b, int g, int j, const uint32_t*& p, uint32_t& mword, uint32_t& mbit) {
    const int64_t bit = (int64_t)g * A.V + (int64_t)j * kBlkTok;
    const uint32_t* w = A.mask + (int64_t)b * A.mask_stride + (bit >> 5);
    mword = (uint32_t)(reinterpret_cast<uintptr_t>(w) & 15u) >> 2;
    mbit = (uint32_t)bit & 31u;
    p = w - mword;
}

// A warp's walk over its blocks: every eighth block of the CTA's range.
template <typename T>
struct BlockCursor {
    int row, j;
    RowGeom q;
    __device__ __forceinline__ void start(const ScanArgs& A, long long t) {
        if (t <= 0x7FFFFFFFll) row = (int)((uint32_t)t / (uint32_t)A.nb);  // (a 64-bit division is a long subroutine)
        else row = (int)(t / A.nb);
        j = (int)(t - (long long)row * A.nb);
        q = row_geom<T>(A, row);
    }
    __device__ __forceinline__ void next(const ScanArgs& A, bool more) {
        j += kScanWarps;
        if (j < A.nb) return;
        while (j >= A.nb) { j -= A.nb; ++row; }
        if (more) q = row_geom<T>(A, row);
    }
};

// Lane 0: the copies of one block (logits, and the mask words beside them) into a slot.
template <typename T, bool kMask, bool kAligned>
__device__ __forceinline__ void issue_block(const ScanArgs& A, const RowGeom& q, int j, long long t, uint32_t slot, uint32_t bar) {
    const int n = min(kBlkTok, A.V - j * kBlkTok);
    const uint8_t* p = q.base + (int64_t)j * (kBlkTok * (int)sizeof(T));
    const uint32_t mis = kAligned ? 0u : (uint32_t)reinterpret_cast<uintptr_t>(p) & 15u;
    const uint32_t bytes = (mis + (uint32_t)n * (uint32_t)sizeof(T) + 15u) & ~15u;
    uint32_t mbytes = 0;
    const uint32_t* mp = nullptr;
    if constexpr (kMask) {
        uint32_t mword, mbit;
        mask_pos(A, q.b, q.g, j, mp, mword, mbit);
        // (whole granules that hold words of the block's bits: every one of them holds a word of the row)
        mbytes = ((mword + ((mbit + (uint32_t)n + 31u) >> 5)) * 4u + 15u) & ~15u;
    }
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes + mbytes) : "memory");
    if (t == A.debug_skip_blk) return;  // test hook: the barrier expects bytes that never come
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(slot), "l"(p - mis),
                 "r"(bytes), "r"(bar)
                 : "memory");
    if constexpr (kMask)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         slot + (uint32_t)ring_slot_bytes((int)sizeof(T), kAligned)),
                     "l"(mp), "r"(mbytes), "r"(bar)
                     : "memory");
}

// ---- the kernel -------------------------------------------------------------------------------
// kHist: the launch has token histories.  kAligned: every virtual row starts on a 16-byte boundary.
// kRoute: RouteOf.
template <typename T, bool kMask, bool kHist, bool kAligned, int kRoute>
__global__ void __launch_bounds__(kScanThreads, 2) scan_kernel(const __grid_constant__ ScanArgs A) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ ScanShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = A.nb, S = A.L.stages;
    const uint32_t slot_bytes = (uint32_t)A.L.slot;
    // the CTA's blocks
    long long t0, t1;
    if (A.slices > 0) {
        const int row = (int)blockIdx.x / A.slices, s = (int)blockIdx.x - row * A.slices;
        t0 = (long long)row * nb + (int)((int64_t)s * nb / A.slices);
        t1 = (long long)row * nb + (int)((int64_t)(s + 1) * nb / A.slices);
    } else {
        const long long N = (long long)A.B * A.G * nb;
        t0 = range_begin(blockIdx.x, N, gridDim.x);
        t1 = range_begin(blockIdx.x + 1, N, gridDim.x);
    }
    // ring barriers: the warp's own
    const uint32_t slot0 = smem_u32(smem) + (uint32_t)warp * slot_bytes, bar0 = smem_u32(&sh.bars[warp]);
    if (lane == 0) {
        for (int s = 0; s < S; ++s) mbar_init(reinterpret_cast<uint64_t*>(&sh.bars[s * kScanWarps + warp]), 1);
        mbar_fence_init();
    }
    if (tid == 0) { sh.defer = 0; sh.remote_hist = 0; sh.remote_fail = 0; }
    __syncwarp();
    // Everything above runs while the launch before this one may still be working (programmatic
    // dependent launch); nothing below starts before its results are there.
    grid_launch_dependents();
    grid_dependency_wait();
    if (A.cluster) cluster_arrive();  // (waited for before the first access to another CTA's shared memory)
    int ids[kHistPer];
    BlockCursor<T> ci;  // the copies' walk
    long long ti = t0 + warp;
    ci.start(A, ti < t1 ? ti : t0);
    // The first row's parameters, history ids and uniform go ahead of the bulk copies: behind them
    // they would wait in the memory system's queues.
    BlockCursor<T> c0;
    c0.start(A, t0);
    born_row_params rp = A.row_params ? A.row_params[c0.q.b] : A.params;
    float u_row = (A.uniforms != nullptr && A.mode == kScanFull) ? __ldg(A.uniforms + c0.q.b) : 0.0f;
    if constexpr (kHist) hist_ids(A, c0.q.b, ids);
    uint32_t si = 0;    // slot of the next copy
    auto issue = [&]() {
        if (lane == 0) issue_block<T, kMask, kAligned>(A, ci.q, ci.j, ti, slot0 + si * (kScanWarps * slot_bytes), bar0 + si * (kScanWarps * 8u));
        ti += kScanWarps;
        ci.next(A, ti < t1);
        if (++si == (uint32_t)S) si = 0;
    };
    // one segment per CTA with a history: the last stages hold the history build's tables until the list is there
    const int held = kHist ? A.L.held : 0;
    for (int i = 0; i < S - held && ti < t1; ++i) issue();

    bool failed = false;
    int bad = 0;
    uint32_t sc = 0, phase = 0;   // slot the next block arrives in, and the parity of its use
    long long t = t0;             // segment start
    long long tc = t0 + warp;     // the warp's next block
    bool first_seg = true;
    while (t < t1) {
        // ---- segment set-up (block-synchronous)
        if (!first_seg) {
            c0.start(A, t);
            rp = A.row_params ? A.row_params[c0.q.b] : A.params;
            u_row = (A.uniforms != nullptr && A.mode == kScanFull) ? __ldg(A.uniforms + c0.q.b) : 0.0f;
        }
        const int row = c0.row, j0 = c0.j;
        const RowGeom q = c0.q;
        const long long row_t0 = (long long)row * nb;
        const long long te = min(t1, row_t0 + nb);
        const bool whole = j0 == 0 && te == row_t0 + nb;
        const RowPlan pl = row_plan(rp);
        const bool mass = RouteOf<kRoute>::mass && (!RouteOf<kRoute>::cand || pl.need_mass);
        const bool want_lse = !mass && (A.out_lse != nullptr || A.want_lse);
        // group keys: shared memory of the CTA that finishes the row, if there is room
        const bool keys_smem = (whole || A.cluster) && nb * 32 <= A.L.gkeys_cap;
        uint16_t* gk = keys_smem ? reinterpret_cast<uint16_t*>(smem + A.L.gkeys) : A.gkeys + (int64_t)row * (nb * 32);
        const uint32_t rank = A.cluster ? (uint32_t)((int)blockIdx.x - row * A.slices) : 0u;
        if (keys_smem && rank > 0) gk = cluster_map(gk, 0u);
        MassBlock* row_blocks = A.blocks + (int64_t)row * A.nblk;
        cta_sync();  // (the finish of the segment before is done with what the set-up writes)
        if (tid == 0) { sh.nl = 0; sh.ng[0] = sh.ng[1] = sh.nh = 0; }
        int hn = 0, hs = 0;
        if constexpr (kHist) {
            if (!first_seg) hist_ids(A, q.b, ids);  // (those of the first row were fetched before the first copies)
            if (penalties_on(rp)) {
                hn = hist_build(A, sh, smem, ids, q.g, j0, j0 + (int)(te - t));
                hs = hist_shift((int)(te - t));
            }
            if (held > 0) {
                fence_proxy_async();
                cta_sync();  // every warp is done with the tables, and its writes are ordered before the copies
                for (int i = 0; i < held && ti < t1; ++i) issue();
            }
        }
        first_seg = false;
        if (A.cluster) cluster_wait();  // every CTA of the cluster has started
        ThreadStats st;
        stats_reset(st, pl.c2);
        // ---- the warp's blocks of the segment
        for (; tc < te; tc += kScanWarps) {
            const int j = (int)(tc - row_t0);
            const uint32_t bar = bar0 + sc * (kScanWarps * 8u), slot = slot0 + sc * (kScanWarps * slot_bytes);
            if (!ring_wait(bar, phase, A.timeout_ns)) {
                failed = true;
                break;
            }
            uint32_t mis = 0;
            if constexpr (!kAligned) mis = (uint32_t)reinterpret_cast<uintptr_t>(q.base) & 15u;  // (a block is a multiple of 16 bytes)
            const uint32_t marea = slot + (uint32_t)ring_slot_bytes((int)sizeof(T), kAligned);
            uint32_t mword = 0, mbit = 0;
            if constexpr (kMask) {
                const uint32_t* mp;
                mask_pos(A, q.b, q.g, j, mp, mword, mbit);
            }
            if constexpr (kHist)
                if (hn > 0) hist_apply<T, kMask>(A, smem, rp, j, (j - j0) >> hs, slot, mis, marea, mword, mbit, want_lse, pl.c2, st);
            float v[2][16];
            load_half<T, kAligned>(slot, mis, 0, v[0]);
            load_half<T, kAligned>(slot, mis, 1, v[1]);
            if constexpr (kMask) {
                const uint32_t wa = marea + 4u * (mword + (uint32_t)lane);
                uint32_t w0, w1 = 0;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w0) : "r"(wa) : "memory");
                if (mbit) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w1) : "r"(wa + 4u) : "memory");
                const uint32_t bits = __funnelshift_r(w0, w1, mbit);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if constexpr (kAligned) {
                            constexpr int VEC = 16 / (int)sizeof(T);
                            const uint32_t vb = bits >> (group_pos<T>(h, i, true) & ~(VEC - 1));  // (one shift per vector)
                            v[h][i] = (vb & (1u << (i & (VEC - 1)))) ? v[h][i] : -INFINITY;
                        } else {
                            v[h][i] = ((bits >> group_pos<T>(h, i, false)) & 1u) ? v[h][i] : -INFINITY;
                        }
                    }
            }
            __syncwarp();  // the block is in registers: its slot may be filled again
            if (ti < t1) issue();
            const int left = A.V - j * kBlkTok - lane * kGrpTok;
            if (j == nb - 1 && left < kGrpTok) {  // the row ends inside this group: nothing beyond it counts
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (group_pos<T>(h, i, kAligned) >= left) v[h][i] = -INFINITY;
            }
            const float mt = group_max(v);
            st.mx = max_nan(st.mx, mt);
            if (!mass || pl.window) gk[j * 32 + lane] = (uint16_t)(zkey(mt) >> 16);
            if (want_lse) lse32(st, v, mt, pl.c2);
            if (RouteOf<kRoute>::mass && mass) {
                // two mass blocks, half a warp each: maximum, exact mass relative to it
                float mb = mt;
#pragma unroll
                for (int d = 8; d > 0; d >>= 1) mb = max_nan(mb, __shfl_xor_sync(0xffffffffu, mb, d));
                uint64_t Q0 = 0, Q1 = 0;
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        uint64_t q0, q1;
                        mass2_of(make_float2(v[h][i], v[h][i + 1]), mb, pl.inv_T, q0, q1);
                        Q0 += q0;
                        Q1 += q1;
                    }
                uint64_t Q = Q0 + Q1;
#pragma unroll
                for (int d = 8; d > 0; d >>= 1) Q += shfl_xor_u64(Q, d);
                int fin = 0;
                if (A.out_kept_count != nullptr && !pl.topp) {  // (temperature only: the kept set is every token above -inf)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < 16; ++i) fin += (v[h][i] > -INFINITY) ? 1 : 0;
#pragma unroll
                    for (int d = 8; d > 0; d >>= 1) fin += __shfl_xor_sync(0xffffffffu, fin, d);
                }
                const int blk = 2 * j + (lane >> 4);
                if ((lane & 15) == 0 && blk < A.nblk) {
                    MassBlock o;
                    o.m = mb; o.pad = (uint32_t)fin; o.M = Q;
                    row_blocks[blk] = o;
                }
            }
            if (++sc == (uint32_t)S) { sc = 0; phase ^= 1u; }
        }

        // ---- segment statistics (block-synchronous)
        const float wm = warp_max_nan(st.mx);
        float ws = 0.0f;
        if (want_lse) {
            const float ssum = st.s.x + st.s.y;
            ws = (ssum > 0.0f && wm == wm) ? ssum * ex2_approx(__fmul_rn(st.R - wm, pl.c2)) : 0.0f;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) ws += __shfl_xor_sync(0xffffffffu, ws, d);
        }
        if (lane == 0) { sh.wmax[warp] = wm; sh.wsum[warp] = ws; }
        if (cta_sync_or(failed ? 1 : 0)) {
            bad = 1;
            if (A.cluster) {  // (the first slice must not wait for this one for good)
                if (tid == 0) *cluster_map(&sh.remote_fail, 0u) = 1;
                cluster_arrive();
                cluster_wait();
            }
            break;
        }
        float m_seg = sh.wmax[0];
#pragma unroll
        for (int w = 1; w < kScanWarps; ++w) m_seg = max_nan(m_seg, sh.wmax[w]);
        float s_seg = 0.0f;
        if (want_lse) {
#pragma unroll
            for (int w = 0; w < kScanWarps; ++w) {
                const float x = sh.wsum[w];
                if (x > 0.0f) s_seg += x * ex2_approx(__fmul_rn(sh.wmax[w] - m_seg, pl.c2));
            }
        }
        RowSrc src;
        src.row = row; src.b = q.b; src.g = q.g; src.u = u_row; src.rp = rp; src.plan = pl;
        src.direct = whole;
        src.m = m_seg; src.ls = s_seg;
        src.gkeys = gk;
        src.hist_n = hn;
        src.remote_hist = 0;
        src.c_first = (int)blockIdx.x; src.nseg = 1;
        bool finish_here = true;
        if (A.cluster) {
            if (tid == 0) *cluster_map(&sh.part[rank], 0u) = make_float2(m_seg, s_seg);
            if constexpr (kHist) {
                if (rank > 0 && hn > 0) {  // history values: from the end of the first slice's list downwards
                    const unsigned long long* list = reinterpret_cast<const unsigned long long*>(smem + A.L.list);
                    if (tid == 0) sh.found = (int)atomicAdd(cluster_map(&sh.remote_hist, 0u), (uint32_t)hn);
                    cta_sync();
                    unsigned long long* dst = cluster_map(reinterpret_cast<unsigned long long*>(smem + A.L.list), 0u) + (A.L.list_cap - 1 - sh.found);
                    for (int i = tid; i < hn; i += kThreads) dst[-i] = list[i];
                }
            }
            cluster_arrive();
            cluster_wait();
            finish_here = rank == 0;
            if (finish_here) {
                if (sh.remote_fail) { bad = 1; break; }
                src.direct = true;
                src.remote_hist = (int)sh.remote_hist;
                src.m = -INFINITY;
                src.ls = 0.0f;
                for (int s = 0; s < A.slices; ++s) src.m = max_nan(src.m, sh.part[s].x);
                if (want_lse)
                    for (int s = 0; s < A.slices; ++s)
                        if (sh.part[s].y > 0.0f) src.ls += sh.part[s].y * ex2_approx(__fmul_rn(sh.part[s].x - src.m, pl.c2));
            }
        } else if (!whole) {
            uint8_t* rec = seg_record(A, row, (int)blockIdx.x);
            if constexpr (kHist) {
                const unsigned long long* list = reinterpret_cast<const unsigned long long*>(smem + A.L.list);
                unsigned long long* ent = reinterpret_cast<unsigned long long*>(rec + kRecordHdrBytes);
                for (int i = tid; i < hn; i += kThreads) ent[i] = list[i];
            }
            if (tid == 0) *reinterpret_cast<float4*>(rec) = make_float4(m_seg, s_seg, __uint_as_float((uint32_t)hn), 0.0f);  // (SegHdr)
            cta_sync();  // orders every thread's keys, mass blocks and entries before the fence below
            if (tid == 0) {
                int c_first, n;
                row_ctas(A, row, c_first, n);
                __threadfence();
                const uint32_t tk = atomicAdd(&A.tickets[row], 1u);
                sh.last = (tk == (uint32_t)n - 1u);
                if (sh.last) A.tickets[row] = 0;  // ready for the next launch
                __threadfence();
            }
            cta_sync();
            finish_here = sh.last != 0;
            if (finish_here) row_ctas(A, row, src.c_first, src.nseg);
        }
        if (finish_here) {
            finish_row<T, kHist, kRoute>(A, sh, smem, src);
            if (A.ring != nullptr && A.mode == kScanFull) {
                cta_sync();  // the row's outputs are written (or the row is handed to the exact search)
                if (tid == 0 && (A.slices > 0 ? sh.defer : A.deferred[row]) == 0) ring_append(A, q.b);
            }
        }
        t = te;
    }

    if (bad) {
        // A wait ran out.  Every row this CTA had a part in reports the failure.  A CTA must not exit
        // with bulk copies in flight into its shared memory: every warp gives those it issued and
        // did not consume (all but the one the test hook withheld) the same bounded wait.
        if (tid == 0) atomicExch(A.dev_error, BORN_ERR_DEVICE_TIMEOUT);
        for (long long tt = tc; tt < ti; tt += kScanWarps) {
            if (tt != A.debug_skip_blk) ring_wait(bar0 + sc * (kScanWarps * 8u), phase, A.timeout_ns);
            if (++sc == (uint32_t)S) { sc = 0; phase ^= 1u; }
        }
        const int r0 = (int)(t0 / nb), r1 = (int)((t1 - 1) / nb), rf = (int)(t / nb);
        for (int r = r0 + tid; r <= r1; r += kThreads) {
            if (A.mode == kScanFull) {
                A.out_status[r / A.G] = 100 + BORN_ERR_DEVICE_TIMEOUT;
                A.out_token[r / A.G] = -1;
            } else if (r >= rf) {  // (an earlier row's record is written, or another CTA's to write)
                write_failed(A, r / A.G, r % A.G);
            }
        }
        return;
    }

    // ---- rows whose kept set the selection could not hold: exact search, now that the ring is idle
    cta_sync();
    if (sh.defer == 0) return;  // (uniform)
    const int r0 = (int)(t0 / nb), r1 = (int)((t1 - 1) / nb);
    for (int r = r0; r <= r1; ++r) {
        const uint32_t owner = A.slices > 0 ? sh.defer : __ldcg(&A.deferred[r]);
        if ((owner & 0xFFFFFFu) != (uint32_t)blockIdx.x + 1u) continue;
        cta_sync();
        if (tid == 0) {
            if (A.slices == 0) A.deferred[r] = 0;
            atomicAdd(A.dev_error + 1, 1);
            atomicAdd(A.dev_error + 8 + (owner >> 24), 1);
        }
        fallback_row<T>(A, sh, smem, r);
        cta_sync();
        if (A.ring != nullptr && A.mode == kScanFull && tid == 0) ring_append(A, r / A.G);
    }
}

}  // namespace born
