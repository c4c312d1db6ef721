// Exact search for rows whose kept set does not fit the 1024 candidates of the in-shared-memory
// selection: a min-p survivor set or a nucleus of thousands of tokens, rows of equal values, a
// kept-id list of a whole-vocabulary row, a nucleus over penalised values.
//
// The kept set is a prefix of the rank order, {rank key >= lowkey}.  The key is found by a threshold
// search without sorting: one pass over the row sums counts or exact masses in 1024 bins of scaled
// distance below the maximum, a second one collects the entries of the bin in which the target
// is crossed, and a radix search over those (at most 1024) gives the exact key; only a bin with more
// entries than that -- ties -- goes through the digits of the 56-bit rank key one by one.  Another
// pass sums the kept mass per chunk of the row, and the draw scans the one chunk it falls into.
// Never approximate.  It runs in the CTA that finished the row, when its ring is idle; the row comes
// from L2.  A pass takes a warp through the row's blocks: the group keys of a block (where the row
// still has them) say which of its 32 groups are read at all.
//
// What bounds it is the one CTA's issue rate: 0.6 us per pass and 10 000 tokens.
#pragma once
#include "scan_common.cuh"
#include "finish.cuh"

namespace born {

constexpr int kFbChunks = 1024;      // chunk sums of the draw
constexpr int kFbHash = 2048;        // slots of the history table

struct FbCtx {
    const ScanArgs* A;
    ScanShared* sh;
    const uint8_t* base;             // the row's first logit
    const uint32_t* mrow;            // the caller row's mask words
    const uint16_t* gkeys;           // group keys (nullptr: every group counts)
    uint32_t* limb;                  // [3][kBins]
    uint32_t* hkeys;                 // history table: keys, then multiplicities
    uint64_t* sel;                   // kSelCap rank keys
    unsigned long long* selq;        // kSelCap masses
    unsigned long long* chunk;       // kFbChunks
    bool hist;
    int b, g, V, id0, nb;
    born_row_params rp;
    float m, inv_T;
};

// The row's distinct history tokens with their multiplicities, in a hash table.
__device__ __forceinline__ void fb_history(FbCtx& c) {
    const ScanArgs& A = *c.A;
    const int tid = threadIdx.x;
    c.hist = A.history != nullptr && penalties_on(c.rp);
    if (!c.hist) return;
    for (int i = tid; i < kFbHash; i += kThreads) { c.hkeys[i] = 0xFFFFFFFFu; c.hkeys[kFbHash + i] = 0u; }
    cta_sync();
    int len = A.history_len ? A.history_len[c.b] : A.history_stride;
    len = max(0, min(min(len, A.history_stride), BORN_MAX_HISTORY));
    const int32_t* gh = A.history + (int64_t)c.b * A.history_stride;
    for (int p = tid; p < len; p += kThreads) {
        const long long tok = (long long)__ldcg(gh + p) - (long long)c.g * c.V;  // (hist_ids: not read-only)
        if (tok < 0 || tok >= c.V) continue;
        uint32_t slot = ((uint32_t)tok * 2654435761u) >> 21;
        for (int probe = 0; probe < kFbHash; ++probe) {
            const uint32_t old = atomicCAS(&c.hkeys[slot], 0xFFFFFFFFu, (uint32_t)tok);
            if (old == 0xFFFFFFFFu || old == (uint32_t)tok) { smem_red_add(&c.hkeys[kFbHash + slot], 1u); break; }
            slot = (slot + 1) & (kFbHash - 1);
        }
    }
    cta_sync();
}

// Logit of token `tok` as the sampler sees it.
template <typename T>
__device__ __forceinline__ float fb_token(const FbCtx& c, int tok) {
    float z = raw_logit<T>(c.base, tok);
    if (c.hist) {
        uint32_t slot = ((uint32_t)tok * 2654435761u) >> 21;
        for (;;) {
            const uint32_t key = c.hkeys[slot];
            if (key == 0xFFFFFFFFu) break;
            if (key == (uint32_t)tok) { z = penalise(c.rp, z, (int)c.hkeys[kFbHash + slot]); break; }
            slot = (slot + 1) & (kFbHash - 1);
        }
    }
    if (c.mrow) {
        const int64_t bi = (int64_t)c.g * c.V + tok;
        if (!((__ldg(c.mrow + (bi >> 5)) >> (bi & 31)) & 1u)) z = -INFINITY;
    }
    return z;
}

// One block of 1024 tokens by the warp: f(tok, z) with eight groups at a time, a lane per token
// (z = -inf where there is none).  Groups whose key is below `low16` are not read.
template <typename T, typename F>
__device__ __forceinline__ void fb_block(const FbCtx& c, int j, uint32_t low16, F f) {
    const int lane = threadIdx.x & 31;
    const int ngrp = (c.V + kGrpTok - 1) / kGrpTok;
    const int gi = j * 32 + lane;
    const uint32_t key = gi < ngrp ? (c.gkeys ? (uint32_t)c.gkeys[gi] : 0xFFFFu) : 0u;
    uint32_t hb = __ballot_sync(0xffffffffu, key >= low16 && gi < ngrp);
    while (hb) {
        int tok[8];
        float z[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            tok[e] = hb ? (j * 32 + __ffs(hb) - 1) * kGrpTok + lane : c.V;
            hb &= hb - 1;
        }
        if (!c.hist && !c.mrow) {  // (the loads leave together)
#pragma unroll
            for (int e = 0; e < 8; ++e) z[e] = tok[e] < c.V ? raw_logit<T>(c.base, tok[e]) : -INFINITY;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) z[e] = tok[e] < c.V ? fb_token<T>(c, tok[e]) : -INFINITY;
        }
        f(tok, z);
    }
}
// One pass over the row; ends on a barrier.
template <typename T, typename F>
__device__ __forceinline__ void fb_pass(const FbCtx& c, uint32_t low16, F f) {
    for (int j = threadIdx.x >> 5; j < c.nb; j += kScanWarps) fb_block<T>(c, j, low16, f);
    cta_sync();
}

__device__ __forceinline__ unsigned long long fb_mass(const FbCtx& c, float z) { return mass_of(scaled_shift(z, c.m, c.inv_T)); }
__device__ __forceinline__ uint32_t fb_low16(unsigned long long lowkey) { return (uint32_t)(lowkey >> 40); }

// Walking the tokens with rank key >= lowkey in rank order (key descending), the key at which the
// running weight (1 per token, or its mass) first exceeds `target`.  Returns 0 when the total
// weight does not exceed target (the caller keeps everything).
template <typename T, bool kWeighted>
__device__ __noinline__ unsigned long long fb_search(FbCtx& c, unsigned long long lowkey, unsigned long long target) {
    const int tid = threadIdx.x;
    ScanShared& sh = *c.sh;
    uint32_t* limb = c.limb;
    const uint32_t low16 = fb_low16(lowkey);
    auto clear = [&]() {
        for (int i = tid; i < 3 * kBins / 4; i += kThreads) reinterpret_cast<uint4*>(limb)[i] = make_uint4(0u, 0u, 0u, 0u);
        cta_sync();
    };
    auto total_of = [&](int i) { return kWeighted ? bin_total(limb, i) : (uint64_t)limb[i]; };
    unsigned long long before = 0;
    int bin = -1;
    // (three 14-bit limbs hold the masses of 2^18 tokens; longer rows go digit by digit, in 64-bit words)
    const bool wide = kWeighted && c.V > (1 << 18);
    if (!wide) {
        clear();
        fb_pass<T>(c, low16, [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                uint64_t q[2] = {1, 1};
                if (kWeighted) mass2_of(make_float2(z[e], z[e + 1]), c.m, c.inv_T, q[0], q[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!(z[e + h] > -INFINITY) || make_ck(z[e + h], c.id0 + tok[e + h]) < lowkey) continue;
                    const int bn = nucleus_bin(z[e + h], c.m, c.inv_T);
                    if (kWeighted) bin_mass(limb, bn, q[h]);
                    else smem_red_add(&limb[bn], 1u);
                }
            }
        });
        bin = find_bin(total_of, target, before, sh);
        if (bin < 0) return 0ull;
        target -= before;
        // the entries of the crossing bin
        if (tid == 0) sh.nl = 0;
        cta_sync();
        fb_pass<T>(c, low16, [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned long long ck = make_ck(z[e], c.id0 + tok[e]);
                if (!(z[e] > -INFINITY) || ck < lowkey || nucleus_bin(z[e], c.m, c.inv_T) != bin) continue;
                const uint32_t pos = smem_atom_add(&sh.nl, 1u);
                if (pos < (uint32_t)kSelCap) { c.sel[pos] = ck; c.selq[pos] = kWeighted ? fb_mass(c, z[e]) : 1ull; }
            }
        });
        const int n = sh.nl;
        if (n <= kSelCap)
            return block_radix_search<true, 56, !kWeighted>(
                n, target, [&](int i) { return c.sel[i]; }, [&](int i) { return c.selq[i]; }, sh.sc);
    }
    // more entries than that in one bin: ten bits of the rank key per pass
    unsigned long long prefix = 0, pmask = 0;
    unsigned long long* wide_bins = c.selq;  // kBins 64-bit words, when limbs could overflow
    for (int shift = 46;; shift = shift > 10 ? shift - 10 : 0) {
        clear();
        if (wide) {
            for (int i = tid; i < kBins; i += kThreads) wide_bins[i] = 0;
            cta_sync();
        }
        fb_pass<T>(c, low16, [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned long long ck = make_ck(z[e], c.id0 + tok[e]);
                if (!(z[e] > -INFINITY) || ck < lowkey || (ck & pmask) != prefix) continue;
                if (!wide && nucleus_bin(z[e], c.m, c.inv_T) != bin) continue;
                const int d = (int)((ck >> shift) & (unsigned long long)(kBins - 1));
                if (!kWeighted) smem_red_add(&limb[d], 1u);
                else if (wide) atomicAdd(&wide_bins[d], fb_mass(c, z[e]));
                else bin_mass(limb, d, fb_mass(c, z[e]));
            }
        });
        // (walk order is descending digit)
        const int o = find_bin([&](int i) { return wide ? (uint64_t)wide_bins[kBins - 1 - i] : total_of(kBins - 1 - i); }, target, before, sh);
        if (o < 0) return 0ull;
        target -= before;
        prefix |= (unsigned long long)(kBins - 1 - o) << shift;
        pmask |= (unsigned long long)(kBins - 1) << shift;
        prefix &= pmask;
        cta_sync();
        if (shift == 0) return prefix;
    }
}

// The (at most kSelCap) tokens with rank key >= lowkey, in sel.
template <typename T>
__device__ __forceinline__ int fb_gather(FbCtx& c, unsigned long long lowkey) {
    cta_sync();
    if (threadIdx.x == 0) c.sh->nl = 0;
    cta_sync();
    fb_pass<T>(c, fb_low16(lowkey), [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const unsigned long long ck = make_ck(z[e], c.id0 + tok[e]);
            if (!(z[e] > -INFINITY) || ck < lowkey) continue;
            const uint32_t pos = smem_atom_add(&c.sh->nl, 1u);
            if (pos < (uint32_t)kSelCap) c.sel[pos] = ck;
        }
    });
    return min(c.sh->nl, kSelCap);
}

// The `count` first tokens in rank order of {rank key >= lowkey}, into the caller's kept-id list.
template <typename T>
__device__ __forceinline__ void fb_kept_ids(FbCtx& c, unsigned long long lowkey, int count) {
    const ScanArgs& A = *c.A;
    unsigned long long Cr = fb_search<T, false>(c, lowkey, (unsigned long long)(count - 1));
    if (Cr < lowkey) Cr = lowkey;
    const int n = fb_gather<T>(c, Cr);
    for (int i = threadIdx.x; i < n; i += kThreads) {
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += (c.sel[j] > c.sel[i]) ? 1 : 0;
        if (rank < A.kept_stride) A.out_kept_ids[(int64_t)c.b * A.kept_stride + rank] = ck_idx(c.sel[i]);
    }
    cta_sync();
}

template <typename T>
__device__ __noinline__ void fallback_row(const ScanArgs& A, ScanShared& sh, uint8_t* smem, int row) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    FbCtx c;
    c.A = &A;
    c.sh = &sh;
    // (kExactBytes of the CTA's dynamic shared memory)
    c.limb = reinterpret_cast<uint32_t*>(smem);
    c.hkeys = c.limb + 3 * kBins;
    c.sel = reinterpret_cast<uint64_t*>(c.hkeys + 2 * kFbHash);
    c.selq = reinterpret_cast<unsigned long long*>(c.sel + kSelCap);
    c.chunk = c.selq + kSelCap;
    static_assert(3 * kBins * 4 + 2 * kFbHash * 4 + 2 * kSelCap * 8 + kFbChunks * 8 <= kExactBytes, "the exact search's shared memory");
    c.b = row / A.G;
    c.g = row - c.b * A.G;
    c.V = A.V;
    c.nb = A.nb;
    c.id0 = A.idx_base + c.g * A.V;
    c.rp = A.row_params ? A.row_params[c.b] : A.params;
    c.base = row_geom<T>(A, row).base;
    c.mrow = A.mask ? A.mask + (int64_t)c.b * A.mask_stride : nullptr;
    const RowPlan pl = row_plan(c.rp);
    c.inv_T = pl.inv_T;
    fb_history(c);
    // Group keys: still there when the row has a CTA or more to itself (a CTA that streams many rows
    // re-uses their place).  bf16 rows with penalties have history tokens that are not in them.
    c.gkeys = nullptr;
    if (A.slices > 0 && (!pl.need_mass || pl.window) && !(sizeof(T) == 2 && c.hist))
        c.gkeys = (A.slices == 1 || A.cluster) && c.nb * 32 <= A.L.gkeys_cap ? reinterpret_cast<const uint16_t*>(smem + A.L.gkeys) : A.gkeys + (int64_t)row * (c.nb * 32);

    // row maximum (the row is known to be valid: only rows with a finite maximum get here)
    {
        uint32_t top16 = 0;
        if (c.gkeys) {  // only the groups that share the best key
            for (int i = tid; i < c.nb * 32; i += kThreads) top16 = max(top16, (uint32_t)c.gkeys[i]);
            top16 = __reduce_max_sync(0xffffffffu, top16);
            if (lane == 0) sh.redu[warp] = top16;
            cta_sync();
#pragma unroll
            for (int w = 0; w < kScanWarps; ++w) top16 = max(top16, sh.redu[w]);
        }
        float mx = -INFINITY;
        fb_pass<T>(c, top16, [&](const int (&)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) mx = fmaxf(mx, z[e]);
        });
        c.m = block_max(mx, sh.redf);
    }

    RowOut o;
    o.token = A.out_token; o.prob = A.out_prob; o.lse = A.out_lse; o.status = A.out_status;
    o.kept_ids = A.out_kept_ids; o.kept_count = A.out_kept_count; o.kept_stride = A.kept_stride;
    o.row = c.b;
    const unsigned long long alive = 1ull << 24;  // smallest rank key of a token above -inf

    if (A.mode == kScanLocal) {
        // the k best of the virtual row, in rank order; the record's sum of 2^((z - m) * c2) with them
        unsigned long long Ck = fb_search<T, false>(c, alive, (unsigned long long)(pl.k - 1));
        if (Ck == 0) Ck = alive;
        float ls = 0.0f;
        fb_pass<T>(c, 0u, [&](const int (&)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) ls += ex2_approx(__fmul_rn(z[e] - c.m, pl.c2));
        });
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, d);
        if (lane == 0) sh.redf[warp] = ls;
        const int n = fb_gather<T>(c, Ck);
        ls = 0.0f;
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) ls += sh.redf[w];
        write_packed(A, sh, c.sel, reinterpret_cast<uint64_t*>(c.selq), n, pl.k, c.b, c.g, c.m, ls);
        return;
    }

    if (pl.greedy) {
        uint64_t best = 0;
        fb_pass<T>(c, zkey(c.m) >> 16, [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (z[e] >= c.m) best = max(best, make_ck(z[e], c.id0 + tok[e]));
        });
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) best = max(best, shfl_xor_u64(best, d));
        if (lane == 0) sh.red64[warp] = best;
        cta_sync();
        if (tid == 0) {
            for (int w = 1; w < kScanWarps; ++w) best = max(best, (uint64_t)sh.red64[w]);
            const int tok = ck_idx(best);
            A.out_token[c.b] = tok;
            A.out_status[c.b] = BORN_ROW_OK;
            if (A.out_prob) A.out_prob[c.b] = 1.0f;
            if (A.out_kept_count) A.out_kept_count[c.b] = 1;
            if (A.out_kept_ids && A.kept_stride > 0) A.out_kept_ids[(int64_t)c.b * A.kept_stride] = tok;
        }
        return;
    }

    const float u = A.uniforms[c.b];
    unsigned long long lowkey = alive;
    if (pl.k > 0) {
        const unsigned long long Ck = fb_search<T, false>(c, lowkey, (unsigned long long)(pl.k - 1));
        if (Ck > lowkey) lowkey = Ck;
    }
    if (pl.minp) {
        // the survivors are a prefix of the rank order (masses fall with the value): lowest surviving value
        const unsigned long long Qa = __double2ull_ru((double)c.rp.min_p * 1099511627776.0);
        const unsigned long long near_cut = (unsigned long long)zkey(c.m + pl.delta) << 24;
        uint32_t zmin = 0xFFFFFFFFu;
        fb_pass<T>(c, fb_low16(max(lowkey, near_cut)), [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                uint64_t q[2];
                mass2_of(make_float2(z[e], z[e + 1]), c.m, c.inv_T, q[0], q[1]);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (z[e + h] > -INFINITY && q[h] >= Qa && make_ck(z[e + h], c.id0 + tok[e + h]) >= lowkey) zmin = min(zmin, zkey(z[e + h]));
            }
        });
        zmin = __reduce_min_sync(0xffffffffu, zmin);
        if (lane == 0) sh.redu[warp] = zmin;
        cta_sync();
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) zmin = min(zmin, sh.redu[w]);
        const unsigned long long Cm = (unsigned long long)zmin << 24;
        if (Cm > lowkey) lowkey = Cm;
        cta_sync();
    }
    unsigned long long S_tot = 0;
    if (pl.need_mass) {
        const MassBlock* blocks = A.blocks + (int64_t)row * A.nblk;
        unsigned long long part = 0;
        for (int ci = tid; ci < A.nblk; ci += kThreads) part += block_share(load_block(blocks + ci), c.m, pl.inv_T);
        S_tot = block_sum_u64(part, sh.red64);
    }
    if (pl.need_mass && !pl.window) {
        // whole-row draw; only the kept-id list brought the row here
        if (A.out_kept_ids) fb_kept_ids<T>(c, alive, min(A.kept_stride, kSelCap));
        draw_whole_row<T>(A, sh, o, c.rp, c.b, c.g, row, c.m, pl.inv_T, S_tot, u);
        return;
    }
    if (pl.topp) {
        unsigned long long S = S_tot;
        if (!pl.need_mass) {
            unsigned long long part = 0;
            fb_pass<T>(c, fb_low16(lowkey), [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    uint64_t q[2];
                    mass2_of(make_float2(z[e], z[e + 1]), c.m, c.inv_T, q[0], q[1]);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (make_ck(z[e + h], c.id0 + tok[e + h]) >= lowkey) part += q[h];
                }
            });
            S = block_sum_u64(part, sh.red64);
        }
        unsigned long long Tp = __double2ull_rz(__dmul_rn((double)c.rp.top_p, __ull2double_rn(S)));
        if (Tp < 1) Tp = 1;
        const unsigned long long Cp = fb_search<T, true>(c, lowkey, Tp - 1);
        if (Cp > lowkey) lowkey = Cp;
    }
    // the kept set is {rank key >= lowkey}: its mass per chunk of the row, and its size
    int cl = 0;  // blocks per chunk, as a shift
    while (((c.nb - 1) >> cl) >= kFbChunks) ++cl;
    const int nchunk = ((c.nb - 1) >> cl) + 1;
    int cnt = 0;
    cta_sync();
    for (int ch = warp; ch < nchunk; ch += kScanWarps) {
        unsigned long long part = 0;
        for (int j = ch << cl; j < min(c.nb, (ch + 1) << cl); ++j)
            fb_block<T>(c, j, fb_low16(lowkey), [&](const int (&tok)[8], const float (&z)[8]) {
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    uint64_t q[2];
                    mass2_of(make_float2(z[e], z[e + 1]), c.m, c.inv_T, q[0], q[1]);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (z[e + h] > -INFINITY && make_ck(z[e + h], c.id0 + tok[e + h]) >= lowkey) { part += q[h]; ++cnt; }
                }
            });
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) part += shfl_xor_u64(part, d);
        if (lane == 0) c.chunk[ch] = part;
    }
    const int n_kept = (int)block_sum_u64((uint64_t)cnt, sh.red64);  // (its barriers cover the chunk sums)
    unsigned long long part = 0;
    for (int ch = tid; ch < nchunk; ch += kThreads) part += c.chunk[ch];
    const unsigned long long S = block_sum_u64(part, sh.red64);
    if (S == 0) {
        row_fail(o, BORN_ROW_ALL_MASKED);
        return;
    }
    unsigned long long t = __double2ull_rz(__dmul_rn((double)u, __ull2double_rn(S)));
    if (t > S - 1) t = S - 1;
    unsigned long long before;
    cta_sync();
    const int ch = find_bin([&](int i) { return i < nchunk ? (uint64_t)c.chunk[i] : 0ull; }, t, before, sh);
    t -= before;
    // inside the chunk: four consecutive tokens per thread, block by block
    for (int j = ch << cl; j < min(c.nb, (ch + 1) << cl); ++j) {
        const int tok0 = j * kBlkTok + 4 * tid;
        uint64_t q[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (tok0 + i >= c.V) continue;
            const float z = fb_token<T>(c, tok0 + i);
            if (z > -INFINITY && make_ck(z, c.id0 + tok0 + i) >= lowkey) q[i] = fb_mass(c, z);
        }
        const uint64_t loc = q[0] + q[1] + q[2] + q[3];
        uint64_t incl = loc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t up = shfl_up_u64(incl, d);
            if (lane >= d) incl += up;
        }
        cta_sync();
        if (lane == 31) sh.red64[warp] = incl;
        cta_sync();
        uint64_t total = 0;
#pragma unroll
        for (int w = 0; w < kScanWarps; ++w) {
            const uint64_t x = sh.red64[w];
            if (w < warp) incl += x;
            total += x;
        }
        if (total > t) {  // (uniform)
            if (incl > t && incl - loc <= t) {
                uint64_t acc = incl - loc;
                int i = 0;
                for (; i < 3 && acc + q[i] <= t; ++i) acc += q[i];
                A.out_token[c.b] = c.id0 + tok0 + i;
                A.out_status[c.b] = BORN_ROW_OK;
                if (A.out_prob) A.out_prob[c.b] = __double2float_rn(__ddiv_rn(__ull2double_rn(q[i]), __ull2double_rn(S)));
            }
            break;
        }
        t -= total;
    }
    if (A.out_kept_count && tid == 0) A.out_kept_count[c.b] = n_kept;
    if (A.out_kept_ids) fb_kept_ids<T>(c, lowkey, min(min(A.kept_stride, kSelCap), n_kept));
}

}  // namespace born
