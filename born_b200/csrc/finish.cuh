// Finishing a row: fold the segments' statistics, work out from the group keys which groups of 32
// tokens can hold tokens that matter, read those again, select (top-k -> min-p -> top-p on exact
// integer masses) and draw by inverse CDF in ascending token index.  Runs in the CTA that
// completes the row (scan_kernel) or, from the selection on, in merge_kernel over all-gathered
// shard records.
//
// Every decision sum is an exact integer sum of fixed-point masses
// q = rne(exp_det((z - m) * inv_T) * 2^40), so thread order cannot matter.  Rank order is
// (value descending, token index ascending): the first maximum wins, as in the reference's
// argmax (born: internal/nn/cross_entropy.go:241-251).
#pragma once
#include <float.h>
#include <string.h>
#include "scan_common.cuh"

namespace born {

struct PackedHdr {  // 32 bytes: header of a packed shard / segment record (the all-gather payload)
    float m;        // maximum of the shard's row (NaN if a NaN was seen)
    float lse_s;    // sum of 2^((z - m) * c2)
    uint32_t count; // entries that follow: rank keys, best first
    uint32_t flags; // bit 0: the shard held more than `count` candidates; bit 1: the pass over the shard failed (no entries)
    float bound;
    uint32_t pad[3];
};
static_assert(sizeof(PackedHdr) == kRecordHdrBytes, "packed header size");

struct RowOut {   // where a finished row reports
    int32_t* token; float* prob; float* lse; int32_t* status; int32_t* kept_ids; int32_t* kept_count;
    int kept_stride;
    int row;
};
__device__ __forceinline__ void row_fail(const RowOut& o, int status) {
    if (threadIdx.x == 0) {
        o.token[o.row] = -1;
        o.status[o.row] = status;
        if (o.prob) o.prob[o.row] = 0.0f;
        if (o.kept_count) o.kept_count[o.row] = 0;
    }
}

struct SelectIn {
    int n;          // entries in sel[]: rank keys, all alive
    int k;          // keep the k best first (0: keep all)
    unsigned long long Qa;     // min-p threshold on the masses (0: off)
    float top_p;    // (0,1): on
    unsigned long long S_ext;  // top-p total when the candidates are only the heavy part of the row (0: their own sum)
    float m_row, inv_T, u;
};

// Threads that share the loops over one of n candidates: log2.  The loops are chains of
// shared-memory reads, so the CTA's 256 threads are dealt over (candidate, part of the loop).
__device__ __forceinline__ int split_lg(int n) { return n <= 32 ? 3 : n <= 64 ? 2 : n <= 128 ? 1 : 0; }
// Candidates up to which every one is compared with every other (select_small).  The comparisons are quadratic: a
// merge launch over 200 candidates takes 13.4 us with them, one that sorts 400 takes 9.9.
constexpr int kSmallMax = 128;

// Selection and draw over n <= kSmallMax candidates in shared memory (sel: rank keys; selq: scratch for
// their masses and, from kThreads on, for the masses of the kept ones).  Nothing is sorted: one loop over
// the candidates gives each its rank (the number of larger keys: keys are unique, the token index is
// part of them) and the mass ahead of it, and since a mass never grows along the rank order the kept
// set of every filter is a prefix of it; a second loop over the kept ones gives the mass at smaller
// token indices.  Returns false when the nucleus of S_ext is not inside the candidates (nothing is
// written then); all threads get the same answer.
__device__ __forceinline__ bool select_small(const SelectIn& in, uint64_t* sel, unsigned long long* selq, ScanShared& sh,
                                             const RowOut& o) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = in.n, lg = split_lg(n), step = 1 << lg;
    const int ci = tid >> lg, sub = tid & (step - 1);
    const int k_eff = in.k > 0 ? in.k : 0x7fffffff;
    const bool topp = in.top_p > 0.0f && in.top_p < 1.0f;
    unsigned long long* kq = selq + kThreads;
    if (tid < n) {
        const uint64_t c = sel[tid];
        uint64_t q = 0;
        if (ck_alive(c)) {
            const float x = scaled_shift(ck_z(c), in.m_row, in.inv_T);
            q = (x < -30.0f) ? 0ull : mass_of(x);
            if (in.Qa && q < in.Qa) { q = 0; sel[tid] = c & (uint64_t)kIdxMask; }  // min-p: a dead entry keeps its index only
        }
        selq[tid] = q;
    }
    if (tid == 0) { sh.acc[0] = 0; sh.nw = 0; }
    cta_sync();
    const uint64_t ck = ci < n ? sel[ci] : 0ull;
    const uint64_t q = ci < n ? (uint64_t)selq[ci] : 0ull;
    int rank = 0;
    uint64_t before = 0;
    for (int j = sub; j < n; j += 8 * step) {  // (eight broadcast reads in flight: the loop is bound by latency otherwise)
        uint64_t cj[8], qj[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = j + i * step;
            cj[i] = at < n ? sel[at] : 0ull;
            qj[i] = at < n ? (uint64_t)selq[at] : 0ull;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            rank += cj[i] > ck ? 1 : 0;
            before += cj[i] > ck ? qj[i] : 0ull;
        }
    }
    for (int d = 1; d < step; d <<= 1) {
        rank += __shfl_xor_sync(0xffffffffu, rank, d);
        before += shfl_xor_u64(before, d);
    }
    const bool first = sub == 0 && ci < n;
    const bool in_k = ck_alive(ck) && rank < k_eff;
    bool kept = in_k;
    uint64_t w = (first && in_k) ? q : 0ull;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) w += shfl_xor_u64(w, d);
    if (lane == 0) sh.red64[warp] = w;
    if (!topp) {
        if (first) kq[ci] = in_k ? q : 0ull;
        const uint32_t kb = __ballot_sync(0xffffffffu, first && in_k);
        if (lane == 0 && kb) smem_red_add(&sh.nw, (uint32_t)__popc(kb));
    }
    cta_sync();
    uint64_t S = 0;
#pragma unroll
    for (int i = 0; i < kScanWarps; ++i) S += sh.red64[i];
    if (topp) {
        // kept: the mass ahead still short of the nucleus; the one that completes it reports the sum
        uint64_t Tp = __double2ull_rz(__dmul_rn((double)in.top_p, __ull2double_rn(in.S_ext ? in.S_ext : S)));
        if (Tp < 1) Tp = 1;
        kept = in_k && before < Tp;
        if (first) kq[ci] = kept ? q : 0ull;
        if (first && kept && before + q >= Tp) sh.acc[0] = before + q;
        const uint32_t kb = __ballot_sync(0xffffffffu, first && kept);
        if (lane == 0 && kb) smem_red_add(&sh.nw, (uint32_t)__popc(kb));
        cta_sync();
        S = sh.acc[0];
        if (in.S_ext && S < Tp) return false;  // (uniform)
    }
    if (S == 0) {  // cannot happen while the row maximum is finite; never divide by it
        row_fail(o, BORN_ROW_ALL_MASKED);
        return true;
    }
    uint64_t t = __double2ull_rz(__dmul_rn((double)in.u, __ull2double_rn(S)));
    if (t > S - 1) t = S - 1;
    const uint32_t my_low = (uint32_t)(ck & kIdxMask);  // larger low bits = smaller token index
    uint64_t pre = 0;
    for (int j = sub; j < n; j += 8 * step) {
        uint32_t lj[8];
        uint64_t qj[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = j + i * step;
            lj[i] = at < n ? (uint32_t)sel[at] & kIdxMask : 0u;
            qj[i] = at < n ? (uint64_t)kq[at] : 0ull;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) pre += lj[i] > my_low ? qj[i] : 0ull;
    }
    for (int d = 1; d < step; d <<= 1) pre += shfl_xor_u64(pre, d);
    if (first && kept) {
        if (pre <= t && t < pre + q) {
            o.token[o.row] = ck_idx(ck);
            o.status[o.row] = BORN_ROW_OK;
            if (o.prob) o.prob[o.row] = __double2float_rn(__ddiv_rn(__ull2double_rn(q), __ull2double_rn(S)));
        }
        if (o.kept_ids && rank < o.kept_stride) o.kept_ids[(int64_t)o.row * o.kept_stride + rank] = ck_idx(ck);
    }
    if (o.kept_count && tid == 0) o.kept_count[o.row] = sh.nw;
    return true;
}

// First bin at which the running total of `total_of(bin)` exceeds `target`, the total ahead of it in
// `before`; -1 when the whole total does not.  All threads get the same answer.  (The caller's last
// barrier covers the bins.)
template <typename F>
__device__ __forceinline__ int find_bin(F total_of, unsigned long long target, unsigned long long& before, ScanShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = kBins / kThreads;
    uint64_t w[PER], loc = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) { w[j] = total_of(PER * tid + j); loc += w[j]; }
    uint64_t incl = loc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t up = shfl_up_u64(incl, d);
        if (lane >= d) incl += up;
    }
    if (lane == 31) sh.red64[warp] = incl;
    if (tid == 0) sh.found = -1;
    cta_sync();
    for (int i = 0; i < warp; ++i) incl += sh.red64[i];
    if (incl > target && incl - loc <= target) {
        uint64_t acc = incl - loc;
        int j = 0;
        for (; j < PER - 1 && acc + w[j] <= target; ++j) acc += w[j];
        sh.found = PER * tid + j;
        sh.before = acc;
    }
    cta_sync();
    before = sh.before;
    return sh.found;
}

// Selection and draw over kSmallMax < n <= kSelCap candidates, the same rules, four candidates per thread.
// A counting sort puts them in rank order: bins of equal width in value from the best candidate down,
// places inside a bin by comparison.  Then the masses are scanned in rank order, and the draw finds its
// token through bins of the token index.  (Three radix descents, over keys, masses and indices, take
// 18 us for 300 candidates.)  `bins`: kBins 64-bit words.
static __device__ __noinline__ bool select_large(const SelectIn in, uint64_t* sel, unsigned long long* selq, uint32_t* bins,
                                                 ScanShared& sh, const RowOut o) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = in.n;
    const int k_eff = in.k > 0 ? in.k : 0x7fffffff;
    const bool topp = in.top_p > 0.0f && in.top_p < 1.0f;
    constexpr int PER = kSelCap / kThreads;
    static_assert(PER == 4 && kBins == 4 * kThreads, "four candidates and four bins per thread");
    cta_sync();
    // ---- ranges of the values and of the indices
    uint64_t c[PER];
    uint32_t zlo = 0xFFFFFFFFu, zhi = 0u, ilo = 0xFFFFFFFFu, ihi = 0u;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int i = tid + j * kThreads;
        c[j] = i < n ? sel[i] : 0ull;
        if (!ck_alive(c[j])) continue;
        const uint32_t z = (uint32_t)(c[j] >> 24), low = (uint32_t)c[j] & kIdxMask;
        zlo = min(zlo, z); zhi = max(zhi, z);
        ilo = min(ilo, low); ihi = max(ihi, low);
    }
    zlo = __reduce_min_sync(0xffffffffu, zlo); zhi = __reduce_max_sync(0xffffffffu, zhi);
    ilo = __reduce_min_sync(0xffffffffu, ilo); ihi = __reduce_max_sync(0xffffffffu, ihi);
    if (lane == 0) { sh.sc.c[4 * warp] = zlo; sh.sc.c[4 * warp + 1] = zhi; sh.sc.c[4 * warp + 2] = ilo; sh.sc.c[4 * warp + 3] = ihi; }
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) { sh.acc[0] = 0; sh.nw = 0; sh.nl = 0; }
    cta_sync();
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) {
        zlo = min(zlo, sh.sc.c[4 * w]); zhi = max(zhi, sh.sc.c[4 * w + 1]);
        ilo = min(ilo, sh.sc.c[4 * w + 2]); ihi = max(ihi, sh.sc.c[4 * w + 3]);
    }
    // ---- counting sort (the bin never falls as the value falls; dead entries go last: their keys are the smallest)
    const float top = zkey_to_float(zhi), span = top - zkey_to_float(zlo);
    const float scale = span > 0.0f ? (float)(kBins - 1) / span : 0.0f;
    int bin[PER];
    uint32_t pos[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        bin[j] = ck_alive(c[j]) ? (int)fminf(__fmul_rn(top - ck_z(c[j]), scale), (float)(kBins - 1)) : kBins - 1;
        pos[j] = tid + j * kThreads < n ? smem_atom_add(&bins[bin[j]], 1u) : 0u;
    }
    cta_sync();
    const uint4 cnt = reinterpret_cast<const uint4*>(bins)[tid];
    uint32_t incl = cnt.x + cnt.y + cnt.z + cnt.w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
    }
    if (lane == 31) sh.redu[warp] = incl;
    cta_sync();
    for (int w = 0; w < warp; ++w) incl += sh.redu[w];
    const uint32_t o3 = incl - cnt.w, o2 = o3 - cnt.z, o1 = o2 - cnt.y;
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(o1 - cnt.x, o1, o2, o3);
    cta_sync();
#pragma unroll
    for (int j = 0; j < PER; ++j)
        if (tid + j * kThreads < n) selq[bins[bin[j]] + pos[j]] = c[j];
    cta_sync();
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (tid + j * kThreads >= n) continue;
        const int b0 = (int)bins[bin[j]], b1 = bin[j] + 1 < kBins ? (int)bins[bin[j] + 1] : n;
        int r = b0;
        for (int i = b0; i < b1; ++i) r += selq[i] > c[j] ? 1 : 0;
        sel[r] = c[j];
    }
    cta_sync();
    // ---- masses in rank order (four consecutive ranks per thread), kept prefix
    uint64_t q[PER], loc = 0;
    bool kept[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int r = PER * tid + j;
        c[j] = r < n ? sel[r] : 0ull;
        q[j] = 0;
        kept[j] = ck_alive(c[j]) && r < k_eff;
        if (kept[j]) {
            const float x = scaled_shift(ck_z(c[j]), in.m_row, in.inv_T);
            q[j] = (x < -30.0f) ? 0ull : mass_of(x);
            if (in.Qa && q[j] < in.Qa) { q[j] = 0; kept[j] = false; }
        }
        loc += q[j];
    }
    uint64_t run = loc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t up = shfl_up_u64(run, d);
        if (lane >= d) run += up;
    }
    if (lane == 31) sh.red64[warp] = run;
    unsigned long long* ibins = reinterpret_cast<unsigned long long*>(bins);
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4*>(bins)[tid + kThreads] = make_uint4(0u, 0u, 0u, 0u);
    cta_sync();
    uint64_t S = 0;
    run -= loc;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) {
        if (w < warp) run += sh.red64[w];
        S += sh.red64[w];
    }
    uint64_t Tp = ~0ull;
    if (topp) {
        Tp = __double2ull_rz(__dmul_rn((double)in.top_p, __ull2double_rn(in.S_ext ? in.S_ext : S)));
        if (Tp < 1) Tp = 1;
    }
    const int sft = max(0, 22 - __clz((int)(ihi - ilo)));  // (the index range is below 2^24: at most kBins bins)
    int nkept = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        kept[j] = kept[j] && run < Tp;
        nkept += kept[j] ? 1 : 0;
        if (topp && kept[j] && run + q[j] >= Tp) sh.acc[0] = run + q[j];
        run += q[j];
        if (!kept[j]) q[j] = 0;
        bin[j] = (int)((ihi - ((uint32_t)c[j] & kIdxMask)) >> sft);  // larger low bits = smaller token index
        if (q[j]) atomicAdd(&ibins[bin[j]], (unsigned long long)q[j]);
    }
    nkept = __reduce_add_sync(0xffffffffu, nkept);
    if (lane == 0 && nkept) smem_red_add(&sh.nw, (uint32_t)nkept);
    cta_sync();
    if (topp) {
        S = sh.acc[0];
        if (in.S_ext && S < Tp) return false;  // (uniform)
    }
    const int R = sh.nw;
    if (S == 0) {
        row_fail(o, BORN_ROW_ALL_MASKED);
        return true;
    }
    // ---- the draw: the bin of the index that holds t, then its members by comparison
    uint64_t t = __double2ull_rz(__dmul_rn((double)in.u, __ull2double_rn(S)));
    if (t > S - 1) t = S - 1;
    unsigned long long before;
    const int hit = find_bin([&](int i) { return (uint64_t)ibins[i]; }, t, before, sh);
    const uint32_t rel_mask = (1u << sft) - 1u;  // sft <= 14, and a mass has 41 bits
    uint32_t rel[PER];
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        rel[j] = (ihi - ((uint32_t)c[j] & kIdxMask)) & rel_mask;
        if (q[j] && bin[j] == hit) ibins[smem_atom_add(&sh.nl, 1u)] = (q[j] << 14) | rel[j];
    }
    cta_sync();
    const int nb = sh.nl;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (q[j] && bin[j] == hit) {
            uint64_t pre = before;
            for (int i = 0; i < nb; ++i) pre += ((uint32_t)ibins[i] & 0x3FFFu) < rel[j] ? (uint64_t)(ibins[i] >> 14) : 0ull;
            if (pre <= t && t < pre + q[j]) {
                o.token[o.row] = ck_idx(c[j]);
                o.status[o.row] = BORN_ROW_OK;
                if (o.prob) o.prob[o.row] = __double2float_rn(__ddiv_rn(__ull2double_rn(q[j]), __ull2double_rn(S)));
            }
        }
        const int r = PER * tid + j;
        if (o.kept_ids && kept[j] && r < o.kept_stride) o.kept_ids[(int64_t)o.row * o.kept_stride + r] = ck_idx(c[j]);
    }
    if (o.kept_count && tid == 0) o.kept_count[o.row] = R;
    return true;
}

// Block-wide reductions (results to every thread).
__device__ __forceinline__ float block_max(float v, float* buf) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    cta_sync();
    if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
    cta_sync();
    float r = buf[0];
#pragma unroll
    for (int w = 1; w < kScanWarps; ++w) r = fmaxf(r, buf[w]);
    return r;
}

__device__ __forceinline__ MassBlock load_block(const MassBlock* p) {
    const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
    MassBlock b;
    b.m = __uint_as_float((uint32_t)v.x);
    b.pad = (uint32_t)(v.x >> 32);
    b.M = v.y;
    return b;
}

// One mass block's contribution to the row total: rne_u64((double)M_c * (double)exp_det((m_c - m) * inv_T)).
__device__ __forceinline__ unsigned long long block_share(const MassBlock& bk, float m, float inv_T) {
    if (!(bk.m > -INFINITY) || bk.M == 0) return 0ull;
    const float ef = exp_det(scaled_shift(bk.m, m, inv_T));
    return __double2ull_rn(__dmul_rn(__ull2double_rn(bk.M), (double)ef));
}

// Logit of token `tok` of virtual row (b, g) as the sampler sees it: upcast, history
// penalties, grammar mask.  O(history) per call; used by the paths that look at few tokens.
template <typename T>
__device__ __forceinline__ float token_logit(const ScanArgs& A, const born_row_params& rp, int b, int g, int tok) {
    const T* row = reinterpret_cast<const T*>(A.logits) + (int64_t)b * A.row_stride + (int64_t)g * A.V;
    float z;
    if constexpr (sizeof(T) == 4) z = __ldg(reinterpret_cast<const float*>(row) + tok);
    else z = bf16_bits_to_f32(__ldg(reinterpret_cast<const uint16_t*>(row) + tok));
    if (A.history && penalties_on(rp)) {
        int len = A.history_len ? A.history_len[b] : A.history_stride;
        len = max(0, min(min(len, A.history_stride), BORN_MAX_HISTORY));
        const int32_t* gh = A.history + (int64_t)b * A.history_stride;
        const int id = g * A.V + tok;
        int cnt = 0;
        for (int p = 0; p < len; ++p) cnt += (gh[p] == id) ? 1 : 0;  // (plain reads, cached in L1: hist_ids has why not read-only ones)
        if (cnt > 0) z = penalise(rp, z, cnt);
    }
    if (A.mask) {
        const int64_t bi = (int64_t)g * A.V + tok;
        if (!((__ldg(A.mask + (int64_t)b * A.mask_stride + (bi >> 5)) >> (bi & 31)) & 1u)) z = -INFINITY;
    }
    return z;
}

// Temperature-only rows: the draw descends the mass blocks.  t = min(floor(u * S), S - 1)
// picks the block (ascending order, shares S_c), then the token inside it by the block's own
// masses: t'' = min(floor((t - before) * M_c / S_c), M_c - 1) in float64.
template <typename T>
__device__ __forceinline__ void draw_whole_row(const ScanArgs& A, ScanShared& sh, const RowOut& o, const born_row_params& rp,
                                               int b, int g, int row, float m, float inv_T,
                                               unsigned long long S, float u) {
    const int tid = threadIdx.x;
    const MassBlock* blocks = A.blocks + (int64_t)row * A.nblk;
    unsigned long long t = __double2ull_rz(__dmul_rn((double)u, __ull2double_rn(S)));
    if (t > S - 1) t = S - 1;
    unsigned long long run = 0;
    if (tid == 0) sh.found = -1;
    cta_sync();
    for (int base = 0; base < A.nblk; base += kThreads) {
        const int c = base + tid;
        MassBlock bk;
        bk.m = -INFINITY; bk.M = 0; bk.pad = 0;
        if (c < A.nblk) bk = load_block(blocks + c);
        const unsigned long long v = block_share(bk, m, inv_T);
        unsigned long long incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long up = shfl_up_u64(incl, d);
            if ((tid & 31) >= d) incl += up;
        }
        cta_sync();
        if ((tid & 31) == 31) sh.red64[tid >> 5] = incl;
        cta_sync();
        unsigned long long off = 0, total = 0;
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) {
            const unsigned long long x = sh.red64[w];
            if (w < (tid >> 5)) off += x;
            total += x;
        }
        incl += off;
        if (run + total > t) {  // the block is in this chunk (uniform)
            if (run + incl > t && run + incl - v <= t) {
                sh.found = c;
                sh.before = run + incl - v;
            }
            cta_sync();
            break;
        }
        run += total;
    }
    cta_sync();
    const int c = sh.found;
    if (c < 0) {  // cannot happen: S is the sum of the shares
        row_fail(o, BORN_ROW_ALL_MASKED);
        return;
    }
    const MassBlock bk = load_block(blocks + c);
    const unsigned long long Sc = block_share(bk, m, inv_T);
    const unsigned long long tb = t - sh.before;
    unsigned long long tt = __double2ull_rz(__ddiv_rn(__dmul_rn(__ull2double_rn(tb), __ull2double_rn(bk.M)), __ull2double_rn(Sc)));
    if (tt > bk.M - 1) tt = bk.M - 1;
    // the block's tokens again, two consecutive ones per thread
    unsigned long long q[2];
    const int tok0 = c * kMassBlock + 2 * tid;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        q[i] = 0;
        if (tok0 + i < A.V) {
            const float z = token_logit<T>(A, rp, b, g, tok0 + i);
            q[i] = mass_of(scaled_shift(z, bk.m, inv_T));
        }
    }
    const unsigned long long v = q[0] + q[1];
    unsigned long long incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long up = shfl_up_u64(incl, d);
        if ((tid & 31) >= d) incl += up;
    }
    cta_sync();
    if ((tid & 31) == 31) sh.red64[tid >> 5] = incl;
    cta_sync();
    unsigned long long off = 0;
    for (int w = 0; w < (tid >> 5); ++w) off += sh.red64[w];
    incl += off;
    if (incl > tt && incl - v <= tt) {
        const int i = (incl - v + q[0] > tt) ? 0 : 1;
        o.token[o.row] = g * A.V + tok0 + i;
        o.status[o.row] = BORN_ROW_OK;
        if (o.prob) {
            const double p = __dmul_rn(__ddiv_rn(__ull2double_rn(q[i]), __ull2double_rn(bk.M)),
                                       __ddiv_rn(__ull2double_rn(Sc), __ull2double_rn(S)));
            o.prob[o.row] = __double2float_rn(p);
        }
    }
}

// Mass bins: a token z (scaled distance below the maximum x = (m - z) * inv_T) falls into bin
// floor(32 x); masses are summed per bin as three 14-bit limbs in 32-bit words (32-bit shared-memory
// atomics run at two cycles per warp here, 64-bit ones are compare-and-swap loops), which holds the
// exact sum of up to 2^18 tokens.
constexpr float kBinScale = 32.0f;
__device__ __forceinline__ int nucleus_bin(float z, float m, float inv_T) {
    return (int)fminf(__fmul_rn(__fmul_rn(__fsub_rn(m, z), inv_T), kBinScale), (float)(kBins - 1));
}
template <bool kTakeOut = false>
__device__ __forceinline__ void bin_mass(uint32_t* limb, int bin, uint64_t q) {
    if (q == 0) return;
    auto add = [&](uint32_t* p, uint32_t part) { smem_red_add(p, kTakeOut ? 0u - part : part); };
    add(&limb[bin], (uint32_t)q & 0x3FFFu);
    add(&limb[kBins + bin], (uint32_t)(q >> 14) & 0x3FFFu);
    if (q >> 28) add(&limb[2 * kBins + bin], (uint32_t)(q >> 28));
}
__device__ __forceinline__ uint64_t bin_total(const uint32_t* limb, int bin) {
    return (uint64_t)limb[bin] + ((uint64_t)limb[kBins + bin] << 14) + ((uint64_t)limb[2 * kBins + bin] << 28);
}
// A completed row: where its statistics, group keys and history values are.
struct RowSrc {
    int row, b, g;               // virtual row; caller row and vocabulary segment
    bool direct;                 // one CTA streamed the whole row: statistics and history list in its shared memory
    float m, ls;                 // direct: the row's maximum and log-sum-exp sum
    const uint16_t* gkeys;       // group keys of the row
    int hist_n;                  // direct: entries of the history list ...
    int remote_hist;             // ... and those that other CTAs of the cluster left at its end
    int c_first, nseg;           // records: CTAs that hold a segment of the row
    float u;                     // the caller row's uniform, fetched while the row was streamed
    born_row_params rp;
    RowPlan plan;
};

// Hands row `row` to the exact search that its CTA runs once the ring is idle.  The reason goes in
// the upper byte.
__device__ __forceinline__ void defer_row(const ScanArgs& A, ScanShared& sh, int row, uint32_t why) {
    const uint32_t word = (why << 24) | (blockIdx.x + 1u);
    sh.defer = word;
    if (A.slices == 0) A.deferred[row] = word;
}

// A key that at least k of the 256 keys a warp holds (eight per lane) reach, and not many more: by
// bisection.  0 when fewer than k are alive.
__device__ __forceinline__ uint32_t kth_of_maxima(const uint32_t (&v)[8], int k) {
    auto reach = [&](uint32_t key) {
        int c = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) c += v[i] >= key ? 1 : 0;
        return __reduce_add_sync(0xffffffffu, c);
    };
    uint32_t lo = kDeadKey16 + 1u;
    if (reach(lo) < k) return 0u;
    uint32_t hi = v[0], mn = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) { hi = max(hi, v[i]); mn = min(mn, v[i]); }
    hi = __reduce_max_sync(0xffffffffu, hi) + 1u;
    lo = max(lo, __reduce_min_sync(0xffffffffu, mn));
    while (hi - lo > 1u) {  // k of the keys reach lo, fewer reach hi
        const uint32_t mid = (lo + hi) >> 1;
        const int c = reach(mid);
        if (c >= k) lo = mid;
        else hi = mid;
        if (c >= k && c <= k + k / 16) break;
    }
    return lo;
}

// A key that at least k of the n 16-bit keys (key_of(i), zero: none) reach, and not many more.  Up to
// half as many as there are threads: the k-th largest of the threads' own maxima -- k keys reach it, and
// few more, since the k best seldom share a thread (50 of 4008 keys: 54 reach it).  Every warp holds all
// 256 maxima and finds it by bisection, so one barrier is enough (bins over all keys, the way of larger k,
// take four and 2.3 us).
// Larger k, or too few threads with a live key: bins -- equal steps of the value below the maximum m --
// down to the smallest of the threads' maxima (at least as many keys as threads reach that).  All
// threads get the same answer; kDeadKey16 + 1 when fewer than k are alive.  `bins`: 2 x kBins words.
template <typename F>
__device__ __forceinline__ uint32_t kth_key(F key_of, int n, int k, float m, uint32_t* bins, ScanShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kReg = 16;  // keys a thread keeps in registers: 4096 in all
    uint32_t kk[kReg];
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < kReg; ++i) {
        const int g = tid + i * kThreads;
        kk[i] = g < n ? key_of(g) : 0u;
    }
#pragma unroll
    for (int i = 0; i < kReg; ++i) mx = max(mx, kk[i]);
    for (int g = tid + kReg * kThreads; g < n; g += kThreads) mx = max(mx, key_of(g));
    if (k <= kThreads / 2) {
        uint16_t* maxima = reinterpret_cast<uint16_t*>(sh.sc.c);
        maxima[tid] = (uint16_t)mx;
        cta_sync();
        const uint4 w = reinterpret_cast<const uint4*>(maxima)[lane];
        uint32_t v[8] = {w.x & 0xFFFFu, w.x >> 16, w.y & 0xFFFFu, w.y >> 16, w.z & 0xFFFFu, w.z >> 16, w.w & 0xFFFFu, w.w >> 16};
        const uint32_t t = kth_of_maxima(v, k);
        if (t) return t;
    }
    uint32_t mn = 0xFFFFu;
    auto see = [&](uint32_t key) { mn = min(mn, key > kDeadKey16 ? key : 0xFFFFu); };
#pragma unroll
    for (int i = 0; i < kReg; ++i) see(kk[i]);
    for (int g = tid + kReg * kThreads; g < n; g += kThreads) see(key_of(g));
    const uint32_t lo_w = __reduce_min_sync(0xffffffffu, mx), mn_w = __reduce_min_sync(0xffffffffu, mn);
    if (lane == 0) sh.redu[warp] = (lo_w << 16) | mn_w;
    uint32_t* least = bins + kBins;
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4*>(least)[tid] = make_uint4(~0u, ~0u, ~0u, ~0u);
    cta_sync();
    uint32_t lo = 0xFFFFu;
    mn = 0xFFFFu;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) {
        const uint32_t x = sh.redu[w];
        lo = min(lo, x >> 16);
        mn = min(mn, x & 0xFFFFu);
    }
    lo = max(k > kThreads ? 0u : lo, mn);
    const float span = m - zkey_to_float(lo << 16);
    const float scale = span > 0.0f ? (float)(kBins - 1) / span : 0.0f;
    auto bin_of = [&](uint32_t key) { return (int)fminf(__fmul_rn(m - zkey_to_float(key << 16), scale), (float)(kBins - 1)); };
    auto count = [&](uint32_t key) {
        if (key < lo) return;
        const int bin = bin_of(key);
        smem_red_add(&bins[bin], 1u);
        smem_red_min(&least[bin], key);
    };
#pragma unroll
    for (int i = 0; i < kReg; ++i) count(kk[i]);
    for (int g = tid + kReg * kThreads; g < n; g += kThreads) count(key_of(g));
    cta_sync();
    const uint4 c = reinterpret_cast<const uint4*>(bins)[tid];
    uint32_t incl = c.x + c.y + c.z + c.w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
    }
    if (lane == 31) sh.redu[warp] = incl;
    if (tid == 0) sh.found = -1;
    cta_sync();
    uint32_t off = 0;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) off += w < warp ? sh.redu[w] : 0u;
    const uint32_t before = off + incl - (c.x + c.y + c.z + c.w);
    if (before < (uint32_t)k && off + incl >= (uint32_t)k) {
        int j = 3;
        if (before + c.x >= (uint32_t)k) j = 0;
        else if (before + c.x + c.y >= (uint32_t)k) j = 1;
        else if (before + c.x + c.y + c.z >= (uint32_t)k) j = 2;
        sh.found = 4 * tid + j;
    }
    cta_sync();
    const int b = sh.found;
    if (b < 0) return kDeadKey16 + 1u;
    // The smallest key counted into the crossing bin: the bins follow the order of the keys, so k keys reach
    // it by that count.  (An edge worked back from the bin's number would carry the rounding of m - z, half a
    // unit in the last place of m, which is many steps of a key that is small beside m.)
    return least[b];
}

// Raw logit of token `tok` of the row at `base` (no mask, no penalties).
template <typename T>
__device__ __forceinline__ float raw_logit(const uint8_t* base, int tok) {
    if constexpr (sizeof(T) == 4) return __ldg(reinterpret_cast<const float*>(base) + tok);
    else return bf16_bits_to_f32(__ldg(reinterpret_cast<const uint16_t*>(base) + tok));
}

// Every group of the row whose key reaches `tk`, read again: f(tok, z) with eight groups at a time, a
// lane per token (z = -inf where there is none, or the mask hides it; no penalties).  The CTA lists
// the groups it finds, 4096 keys a round, and deals them over its warps eight at a time: each warp has
// one round of reads in flight as long as there are no more than 64 groups.  (Lists per warp left some
// warps with two rounds, a microsecond apart.)  sh.ng is zero on entry; the caller's next barrier
// frees the list.
template <typename T, typename F>
__device__ __forceinline__ void for_groups(const ScanArgs& A, ScanShared& sh, const uint16_t* keys, int b, int g, uint32_t tk, uint16_t* list,
                                           F f) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ngrp = (A.V + kGrpTok - 1) / kGrpTok;
    const uint8_t* base = reinterpret_cast<const uint8_t*>(A.logits) + ((int64_t)b * A.row_stride + (int64_t)g * A.V) * (int64_t)sizeof(T);
    const uint32_t* mrow = A.mask ? A.mask + (int64_t)b * A.mask_stride : nullptr;
    constexpr int kPer = kGrpRound / kThreads;
    int round = 0;
    for (int g0 = 0; g0 < ngrp; g0 += kGrpRound, round ^= 1) {
        uint32_t hits = 0;
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
            const int gi = g0 + e * kThreads + tid;
            const uint32_t key = gi < ngrp ? (uint32_t)keys[gi] : 0u;
            hits |= key >= tk ? 1u << e : 0u;
        }
        if (__any_sync(0xffffffffu, hits != 0)) {
            uint32_t incl = (uint32_t)__popc(hits);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += up;
            }
            uint32_t at = 0;
            if (lane == 31) at = smem_atom_add(&sh.ng[round], incl);
            at = __shfl_sync(0xffffffffu, at, 31) + incl - (uint32_t)__popc(hits);
            for (; hits; hits &= hits - 1u) list[at++] = (uint16_t)((__ffs(hits) - 1) * kThreads + tid);
        }
        cta_sync();
        const int n = (int)sh.ng[round];
        if (tid == 0) sh.ng[round ^ 1] = 0;
        for (int i = warp * 8; i < n; i += kScanWarps * 8) {
            int tok[8];
            float z[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) tok[e] = i + e < n ? (g0 + (int)list[i + e]) * kGrpTok + lane : A.V;
#pragma unroll
            for (int e = 0; e < 8; ++e) z[e] = tok[e] < A.V ? raw_logit<T>(base, tok[e]) : -INFINITY;
            if (mrow) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int64_t bi = (int64_t)g * A.V + tok[e];
                    if (tok[e] < A.V && !((__ldg(mrow + (bi >> 5)) >> (bi & 31)) & 1u)) z[e] = -INFINITY;
                }
            }
            f(tok, z);
        }
        if (g0 + kGrpRound < ngrp) cta_sync();
    }
}

// The row's history values: f(token of the virtual row, penalised value) for every entry, dealt over
// the threads.
template <typename F>
__device__ __forceinline__ void for_history(const ScanArgs& A, const uint8_t* smem, const RowSrc& src, F f) {
    auto one = [&](unsigned long long e) { f((int)(uint32_t)e, __uint_as_float((uint32_t)(e >> 32))); };
    if (src.direct) {
        const unsigned long long* list = reinterpret_cast<const unsigned long long*>(smem + A.L.list);
        for (int i = threadIdx.x; i < src.hist_n; i += kThreads) one(list[i]);
        for (int i = threadIdx.x; i < src.remote_hist; i += kThreads) one(list[A.L.list_cap - 1 - i]);
        return;
    }
    const int lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < src.nseg; s0 += 32) {
        uint32_t cnt = 0;
        if (s0 + lane < src.nseg) cnt = __ldcg(reinterpret_cast<const uint32_t*>(seg_record(A, src.row, src.c_first + s0 + lane)) + 2);
        for (int s = s0; s < min(src.nseg, s0 + 32); ++s) {
            const int n = (int)__shfl_sync(0xffffffffu, cnt, s - s0);
            const unsigned long long* ent = reinterpret_cast<const unsigned long long*>(seg_record(A, src.row, src.c_first + s) + kRecordHdrBytes);
            for (int i = threadIdx.x; i < n; i += kThreads) one(__ldcg(ent + i));
        }
    }
}
// ... and an upper bound of how many there are.
__device__ __forceinline__ int history_bound(const ScanArgs& A, const RowSrc& src) {
    if (!penalties_on(src.rp)) return 0;
    return src.direct ? src.hist_n + src.remote_hist : A.history_stride;
}

// The key that the k best tokens of the row reach.  From the group keys where there are enough groups
// for their maxima to tell tokens apart; on shorter rows (some 40 k tokens) from the tokens
// themselves, of which `extra` may not count (history tokens: their raw values).
template <typename T>
__device__ __forceinline__ uint32_t kth_token_key(const ScanArgs& A, const RowSrc& src, int k, int extra, float m, uint32_t* bins, ScanShared& sh) {
    const int ngrp = (A.V + kGrpTok - 1) / kGrpTok;
    if (4 * ngrp >= 5 * k) return kth_key([&](int i) { return (uint32_t)src.gkeys[i]; }, ngrp, k, m, bins, sh);
    const uint8_t* base = reinterpret_cast<const uint8_t*>(A.logits) + ((int64_t)src.b * A.row_stride + (int64_t)src.g * A.V) * (int64_t)sizeof(T);
    const uint32_t* mrow = A.mask ? A.mask + (int64_t)src.b * A.mask_stride : nullptr;
    return kth_key([&](int i) {
        const int64_t bi = (int64_t)src.g * A.V + i;
        const float z = raw_logit<T>(base, i);
        const bool hidden = (mrow && !((__ldg(mrow + (bi >> 5)) >> (bi & 31)) & 1u)) || z != z;
        return hidden ? 0u : min(zkey(z), zkey(m)) >> 16;  // (a raw history value may lie above the maximum)
    }, A.V, k + extra, m, bins, sh);
}

// Every token of the row at or above tau into sel (rank keys); returns their number, which may exceed
// kSelCap (what does not fit is dropped: the caller looks at the number).  sh.nl is zero on entry.
// A history token's raw value is struck out (its key keeps the index only, so that keys stay
// unique) and its penalised value added.  The candidates leave a bit each in a 4096-bit map of
// (token mod 4096), so that only the few history tokens that may be candidates look for themselves
// among them (every one of 512 comparing itself with 50 candidates took 1.5 us).
template <typename T, bool kHist>
__device__ __forceinline__ int gather_row(const ScanArgs& A, ScanShared& sh, const uint8_t* smem, const RowSrc& src, float tau, uint64_t* sel,
                                          uint16_t* wl) {
    const int lane = threadIdx.x & 31;
    const float tf = fmaxf(tau, -FLT_MAX);
    const int id0 = A.idx_base + src.g * A.V;
    uint32_t* seen = reinterpret_cast<uint32_t*>(sh.bcnt);
    const bool strike = kHist && penalties_on(src.rp);
    for_groups<T>(A, sh, src.gkeys, src.b, src.g, zkey(tf) >> 16, wl, [&](const int (&tok)[8], const float (&z)[8]) {
        uint32_t hb[8], sum = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            hb[e] = __ballot_sync(0xffffffffu, z[e] >= tf);
            sum += __popc(hb[e]);
        }
        if (sum == 0) return;
        uint32_t pos = 0;
        if (lane == 0) pos = smem_atom_add(&sh.nl, sum);
        pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t at = pos + __popc(hb[e] & ((1u << lane) - 1u));
            if (z[e] >= tf && at < (uint32_t)kSelCap) {
                sel[at] = make_ck(z[e], id0 + tok[e]);
                if (strike) smem_red_or(&seen[((uint32_t)tok[e] >> 5) & 127u], 1u << (tok[e] & 31));
            }
            pos += __popc(hb[e]);
        }
    });
    cta_sync();
    int n = sh.nl;
    if constexpr (kHist) {
        if (strike && n <= kSelCap) {
            for_history(A, smem, src, [&](int tok, float zp) {
                if ((seen[((uint32_t)tok >> 5) & 127u] >> (tok & 31)) & 1u) {
                    const uint32_t low = kIdxMask - (uint32_t)(id0 + tok);
                    for (int i = 0; i < n; ++i)
                        if ((uint32_t)(sel[i] & kIdxMask) == low) sel[i] = low;
                }
                if (!(zp >= tf)) return;
                const uint32_t pos = (uint32_t)n + smem_atom_add(&sh.nh, 1u);
                if (pos < (uint32_t)kSelCap) sel[pos] = make_ck(zp, id0 + tok);
            });
            cta_sync();
            n += (int)sh.nh;
        }
    }
    return n;
}

// sel[0..n) cut to its k best (n > k), compacted through tmp; returns k.
__device__ __forceinline__ int cut_to_k(uint64_t* sel, uint64_t* tmp, int n, int k, ScanShared& sh) {
    const int tid = threadIdx.x;
    const uint64_t Tk = block_radix_search<true, 56, true>(
        n, (unsigned long long)(k - 1), [&](int i) { return sel[i]; }, [&](int) { return 1ull; }, sh.sc);
    if (tid == 0) sh.nl = 0;
    cta_sync();
    for (int i = tid; i < n; i += kThreads)
        if (sel[i] >= Tk) tmp[smem_atom_add(&sh.nl, 1u)] = sel[i];
    cta_sync();
    for (int i = tid; i < k; i += kThreads) sel[i] = tmp[i];
    cta_sync();
    return k;
}

// Exactly the k best of a virtual row (k <= kThreads), in rank order, into its packed record.
__device__ __forceinline__ void write_packed(const ScanArgs& A, ScanShared& sh, uint64_t* sel, uint64_t* tmp, int n, int k, int b, int g,
                                             float m, float lse_s) {
    const int tid = threadIdx.x;
    uint8_t* rec = A.packed + (int64_t)g * A.packed_seg_stride + (int64_t)b * A.packed_row_stride;
    uint64_t* ent = reinterpret_cast<uint64_t*>(rec + kRecordHdrBytes);
    if (n > kThreads) n = cut_to_k(sel, tmp, n, k, sh);
    const int lg = split_lg(n), step = 1 << lg, ci = tid >> lg, sub = tid & (step - 1);
    const uint64_t ck = ci < n ? sel[ci] : 0ull;
    const int alive = cta_sync_count(sub == 0 && ck_alive(ck));
    int rank = 0;
    for (int j = sub; j < n; j += 8 * step) {
        uint64_t v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = j + i * step < n ? sel[j + i * step] : 0ull;
#pragma unroll
        for (int i = 0; i < 8; ++i) rank += (v[i] > ck) ? 1 : 0;
    }
    for (int d = 1; d < step; d <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, d);
    const int nk = min(alive, k);
    if (sub == 0 && ci < n && rank < nk) ent[rank] = ck;
    if (tid == 0) {
        PackedHdr h;
        h.m = m; h.lse_s = lse_s; h.count = (uint32_t)nk;
        h.flags = alive > k ? 1u : 0u;
        h.bound = -INFINITY;
        h.pad[0] = h.pad[1] = h.pad[2] = 0;
        memcpy(rec, &h, sizeof h);
    }
}

// The record of a virtual row that could not be streamed: the merge reports the failure instead of
// sampling whatever the record's place held before.  One thread.
__device__ __forceinline__ void write_failed(const ScanArgs& A, int b, int g) {
    PackedHdr h;
    h.m = -INFINITY; h.lse_s = 0.0f; h.count = 0; h.flags = 2u; h.bound = -INFINITY;
    h.pad[0] = h.pad[1] = h.pad[2] = 0;
    memcpy(A.packed + (int64_t)g * A.packed_seg_stride + (int64_t)b * A.packed_row_stride, &h, sizeof h);
}

template <typename T>
__device__ __noinline__ void fallback_row(const ScanArgs& A, ScanShared& sh, uint8_t* smem, int row);

// A row is complete: fold its statistics, select, draw.
template <typename T, bool kHist, int kRoute>
__device__ __forceinline__ void finish_row(const ScanArgs& A, ScanShared& sh, uint8_t* smem, const RowSrc& src) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int row = src.row, b = src.b, g = src.g;
    const born_row_params& rp = src.rp;
    const RowPlan& pl = src.plan;
    const bool mass = RouteOf<kRoute>::mass && (!RouteOf<kRoute>::cand || pl.need_mass);
    uint64_t* sel = reinterpret_cast<uint64_t*>(smem + A.L.work);
    unsigned long long* selq = reinterpret_cast<unsigned long long*>(sel + kSelCap);
    uint16_t* wl = reinterpret_cast<uint16_t*>(selq + kSelCap);  // group list; bins of the larger selection
    const int ngrp = (A.V + kGrpTok - 1) / kGrpTok;

    float m = src.m, ls = src.ls;
    if (!src.direct) {  // every warp folds the segments' headers for itself
        m = -INFINITY;
        for (int s = lane; s < src.nseg; s += 32) m = max_nan(m, __ldcg(reinterpret_cast<const float*>(seg_record(A, row, src.c_first + s))));
        m = warp_max_nan(m);
        ls = 0.0f;
        if (!mass) {
            for (int s = lane; s < src.nseg; s += 32) {
                const float2 h = __ldcg(reinterpret_cast<const float2*>(seg_record(A, row, src.c_first + s)));
                if (h.y > 0.0f) ls += h.y * ex2_approx(__fmul_rn(h.x - m, pl.c2));
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, d);
        }
    }
    int status = BORN_ROW_OK;
    if (m != m) status = BORN_ROW_NAN;
    else if (m == INFINITY) status = BORN_ROW_POS_INF;
    else if (m == -INFINITY) status = BORN_ROW_ALL_MASKED;

    if (A.mode == kScanLocal) {
        // ---- the k best of the virtual row, in rank order
        int n = 0;
        if (status == BORN_ROW_OK) {
            const uint32_t tk = kth_token_key<T>(A, src, pl.k, kHist ? history_bound(A, src) : 0, m, reinterpret_cast<uint32_t*>(selq), sh);
            n = gather_row<T, kHist>(A, sh, smem, src, zkey_to_float(tk << 16), sel, wl);
            if (n > kSelCap) {
                if (tid == 0) defer_row(A, sh, row, 8u);
                return;
            }
        }
        write_packed(A, sh, sel, reinterpret_cast<uint64_t*>(selq), n, pl.k, b, g, m, ls);
        return;
    }

    RowOut o;
    o.token = A.out_token; o.prob = A.out_prob; o.lse = A.out_lse; o.status = A.out_status;
    o.kept_ids = A.out_kept_ids; o.kept_count = A.out_kept_count; o.kept_stride = A.kept_stride;
    o.row = b;
    if (A.row_params != nullptr && !row_params_ok(rp)) status = BORN_ROW_BAD_PARAMS;  // (device arrays are not checked on the host)
    if (status != BORN_ROW_OK) {
        if (tid == 0 && A.out_lse) A.out_lse[b] = NAN;
        row_fail(o, status);
        return;
    }
    if (!mass && A.out_lse && tid == 0) A.out_lse[b] = m * pl.inv_T + __log2f(ls) * 0.69314718f;

    unsigned long long S_tot = 0;
    float tau = -INFINITY;
    if (RouteOf<kRoute>::mass && mass) {
        // row total from the mass blocks; log-sum-exp from it
        const MassBlock* blocks = A.blocks + (int64_t)row * A.nblk;
        unsigned long long part = 0;
        int fin = 0;
        for (int c = tid; c < A.nblk; c += kThreads) {
            const MassBlock bkc = load_block(blocks + c);
            part += block_share(bkc, m, pl.inv_T);
            fin += (int)bkc.pad;
        }
        S_tot = block_sum_u64(part, sh.red64);
        if (S_tot == 0) {
            row_fail(o, BORN_ROW_ALL_MASKED);
            return;
        }
        if (A.out_lse && tid == 0)
            A.out_lse[b] = (float)((double)m * (double)pl.inv_T + log(__ull2double_rn(S_tot) * (1.0 / 1099511627776.0)));
        if (!pl.window) {
            if (A.out_kept_count) {
                const int nfin = (int)block_sum_u64((uint64_t)fin, sh.red64);
                if (tid == 0) A.out_kept_count[b] = nfin;
            }
            if (A.out_kept_ids) {  // the kept set is the whole row: no list of a useful size exists
                if (tid == 0) defer_row(A, sh, row, 2u);
                return;
            }
            draw_whole_row<T>(A, sh, o, rp, b, g, row, m, pl.inv_T, S_tot, src.u);
            return;
        }
        const bool pen = kHist && penalties_on(rp);
        if (pen && sizeof(T) == 2) {  // (group keys without the history tokens; such rows come here as an fp32 copy)
            if (tid == 0) defer_row(A, sh, row, 7u);
            return;
        }
        // Nucleus of the whole row: a value that the tokens of the nucleus all reach.  First from the
        // group keys alone -- if the groups' best tokens, their values rounded down, already hold the
        // nucleus' share above some value, so do all tokens above it.  Exact masses go into bins of
        // 1/32 of a scaled logit; the bin in which the share is reached is the last that matters.
        // Flat rows, where a group has more than one token that counts, take the tokens themselves:
        // tokens lighter than (1 - P) * S / V weigh less than (1 - P) * S together, so none of those is
        // in the nucleus, and the groups that reach beyond them are read again.
        const float s_all = (float)S_tot * (1.0f / 1099511627776.0f);
        const float cut = fmaxf(m + (__logf((1.0f - rp.top_p) * s_all / (float)A.V) - 0.05f) * rp.temperature, -FLT_MAX);
        unsigned long long Tp = __double2ull_rz(__dmul_rn((double)rp.top_p, __ull2double_rn(S_tot)));
        if (Tp < 1) Tp = 1;
        uint32_t* limb = reinterpret_cast<uint32_t*>(sel);  // [3][kBins]
        unsigned long long before;
        int bin = -1;
        for (int level = 0; level < 2 && bin < 0; ++level) {
            for (int i = tid; i < 3 * kBins / 4; i += kThreads) reinterpret_cast<uint4*>(limb)[i] = make_uint4(0u, 0u, 0u, 0u);
            cta_sync();
            if (level == 0) {
                const uint32_t ck16 = zkey(cut) >> 16;
                for (int i = tid; i < ngrp; i += 2 * kThreads) {
                    const uint32_t k0 = src.gkeys[i], k1 = i + kThreads < ngrp ? (uint32_t)src.gkeys[i + kThreads] : 0u;
                    const float z0 = zkey_to_float(k0 << 16), z1 = zkey_to_float(max(k1, 0x80u) << 16);
                    uint64_t q0, q1;
                    mass2_of(make_float2(z0, z1), m, pl.inv_T, q0, q1);
                    if (k0 >= ck16) bin_mass(limb, nucleus_bin(z0, m, pl.inv_T), q0);
                    if (k1 >= ck16) bin_mass(limb, nucleus_bin(z1, m, pl.inv_T), q1);
                }
            } else {
                for_groups<T>(A, sh, src.gkeys, b, g, zkey(cut) >> 16, wl, [&](const int (&)[8], const float (&z)[8]) {
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        uint64_t q[2];
                        mass2_of(make_float2(z[e], z[e + 1]), m, pl.inv_T, q[0], q[1]);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (z[e + h] >= cut && (!pen || z[e + h] <= m)) bin_mass(limb, nucleus_bin(z[e + h], m, pl.inv_T), q[h]);
                    }
                });
                if (pen) {
                    const uint8_t* base = reinterpret_cast<const uint8_t*>(A.logits) + ((int64_t)b * A.row_stride + (int64_t)g * A.V) * (int64_t)sizeof(T);
                    for_history(A, smem, src, [&](int tok, float zp) {
                        const float z = raw_logit<T>(base, tok);
                        uint64_t q, qp;
                        mass2_of(make_float2(z, zp), m, pl.inv_T, q, qp);
                        if (z >= cut && z <= m && zp > -INFINITY && (uint32_t)src.gkeys[tok / kGrpTok] >= zkey(cut) >> 16)
                            bin_mass<true>(limb, nucleus_bin(z, m, pl.inv_T), q);
                        if (zp >= cut) bin_mass(limb, nucleus_bin(zp, m, pl.inv_T), qp);
                    });
                }
            }
            cta_sync();
            if (tid == 0) sh.ng[0] = sh.ng[1] = 0;  // (for the candidates' own round)
            bin = find_bin([&](int i) { return bin_total(limb, i); }, Tp - 1, before, sh);
            cta_sync();
        }
        if (bin < 0) {  // (the share of what was left out is an estimate)
            if (tid == 0) defer_row(A, sh, row, 7u);
            return;
        }
        // (a shade below the bin's lower edge: more candidates than needed do no harm)
        tau = fmaxf(cut, m - ((float)(bin + 1) * (1.0f / kBinScale) + 0.002f) * rp.temperature - fabsf(m) * 1e-6f);
    } else {
        if (pl.greedy) tau = m;
        if (pl.minp) tau = m + pl.delta;
        if (pl.k > 0) {
            const uint32_t tk = kth_token_key<T>(A, src, pl.k, kHist ? history_bound(A, src) : 0, m, reinterpret_cast<uint32_t*>(selq), sh);
            tau = fmaxf(tau, zkey_to_float(tk << 16));
        }
    }
    const int n = gather_row<T, kHist>(A, sh, smem, src, tau, sel, wl);
    if (n > kSelCap) {
        if (tid == 0) defer_row(A, sh, row, mass ? 7u : pl.k > 0 ? 5u : pl.greedy ? 1u : 6u);
        return;
    }
    if (RouteOf<kRoute>::cand && pl.greedy) {
        uint64_t best = 0;
        for (int i = tid; i < n; i += kThreads) best = max(best, (uint64_t)sel[i]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) best = max(best, shfl_xor_u64(best, d));
        if (lane == 0) sh.red64[tid >> 5] = best;
        cta_sync();
        if (tid == 0) {
            for (int w = 1; w < kScanWarps; ++w) best = max(best, (uint64_t)sh.red64[w]);
            const int tok = ck_idx(best);
            A.out_token[b] = tok;
            A.out_status[b] = BORN_ROW_OK;
            if (A.out_prob) A.out_prob[b] = 1.0f;
            if (A.out_kept_count) A.out_kept_count[b] = 1;
            if (A.out_kept_ids && A.kept_stride > 0) A.out_kept_ids[(int64_t)b * A.kept_stride] = tok;
        }
        return;
    }
    SelectIn in;
    in.n = n;
    in.k = pl.k;
    in.Qa = pl.minp ? __double2ull_ru((double)rp.min_p * 1099511627776.0) : 0ull;
    in.top_p = rp.top_p;
    in.S_ext = mass ? S_tot : 0ull;
    in.m_row = m; in.inv_T = pl.inv_T; in.u = src.u;
    const bool inside = n <= kSmallMax ? select_small(in, sel, selq, sh, o) : select_large(in, sel, selq, reinterpret_cast<uint32_t*>(wl), sh, o);
    if (!inside && tid == 0) defer_row(A, sh, row, 7u);
}

}  // namespace born
