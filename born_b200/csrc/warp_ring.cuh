// Warp-private streaming of logits.
//
// Every warp owns a few shared-memory slots of one 1024-token block each and fills them with its
// own 1-D bulk copies (TMA, no multicast), one mbarrier per slot: lane 0 issues a copy, the warp
// waits, reads the block into registers and issues the next copy into the same slot.  No warp
// ever waits for another one, and no producer warp hands tiles round -- with a barrier or a
// hand-over per tile the loops of this library were bound by latency, not by the bytes in flight.
//
// A lane reads 32 consecutive tokens of the block (a *group*: one 128-byte line of fp32, half a
// line of bf16).  Its 16-byte vectors are read in an order rotated by the lane number (XOR), so
// that eight lanes of a 128-bit access touch eight different bank groups.  Consequences: the grammar
// mask word of a group is one word of the mask; a 512-token mass block is half a warp, a
// 1024-token one a whole warp; a group whose maximum matters is re-read as one piece.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include "spec.cuh"

namespace born {

constexpr int kBlkTok = 1024;                 // tokens per block: 32 per lane
constexpr int kGrpTok = 32;                   // tokens per group
// bytes between the slots of a ring: a block, plus one 16-byte granule when rows do not start on
// 16-byte boundaries (rounded up so that slots stay 128-byte aligned: the XOR order needs that)
__host__ __device__ constexpr int ring_slot_bytes(int elem_bytes, bool aligned) {
    return kBlkTok * elem_bytes + (aligned ? 0 : 128);
}

// Lane 0: starts the copy of tokens [tok0, tok0 + n) of the row at `row` (bytes); the copy begins at
// the 16-byte boundary at or below the first of them and ends at the one at or above the last
// (inside the granules that hold the row's own tokens: never beyond an allocation).
__device__ __forceinline__ void ring_issue(uint32_t slot, uint32_t bar, const uint8_t* row, int tok0, int n, int elem_bytes) {
    const uint8_t* p = row + (int64_t)tok0 * elem_bytes;
    const uint32_t mis = (uint32_t)reinterpret_cast<uintptr_t>(p) & 15u;
    const uint32_t bytes = (mis + (uint32_t)n * (uint32_t)elem_bytes + 15u) & ~15u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(slot), "l"(p - mis),
                 "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ bool ring_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of the whole warp (every lane gets the same answer); false when the limit ran out.
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity, unsigned long long limit_ns) {
    if (__all_sync(0xffffffffu, ring_try(bar, parity))) return true;
    unsigned long long t0 = 0;
    for (uint32_t it = 0; it < kMbarSpinLimit; ++it) {
        if (__all_sync(0xffffffffu, ring_try(bar, parity))) return true;
        if ((it & 15u) == 15u) {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0) t0 = now;
            else if (__any_sync(0xffffffffu, now - t0 > limit_ns)) return false;
        }
    }
    return false;
}

__device__ __forceinline__ float4 lds128f(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 lds128u(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float lds32f(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t lds16u(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}

// Position, within the lane's group, of the value that load_half left in v[i] of half h.
template <typename T>
__device__ __forceinline__ int group_pos(int h, int i, bool aligned) {
    const int lane = (int)threadIdx.x & 31;
    if (!aligned) return (16 * h + i) ^ lane;
    if constexpr (sizeof(T) == 4) return 4 * ((4 * h + (i >> 2)) ^ (lane & 7)) + (i & 3);
    else return 8 * ((2 * h + (i >> 3)) ^ ((lane >> 1) & 3)) + (i & 7);
}

// Half h (16 values) of the lane's group of the block in `slot`.  kAligned: the row starts on a
// 16-byte boundary; otherwise the block begins `mis` bytes into the slot and is read element by
// element (XOR with the lane number: 32 different banks, or 16 words of two halves).
template <typename T, bool kAligned>
__device__ __forceinline__ void load_half(uint32_t slot, uint32_t mis, int h, float (&v)[16]) {
    const uint32_t lane = threadIdx.x & 31u;
    if constexpr (kAligned && sizeof(T) == 4) {
        const uint32_t a = slot + lane * 128u + ((lane & 7u) << 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 q = lds128f(a ^ (uint32_t)((4 * h + j) << 4));
            v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
        }
    } else if constexpr (kAligned) {
        const uint32_t a = slot + lane * 64u + (((lane >> 1) & 3u) << 4);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint4 q = lds128u(a ^ (uint32_t)((2 * h + j) << 4));
            v[8 * j] = __uint_as_float(q.x << 16); v[8 * j + 1] = __uint_as_float(q.x & 0xFFFF0000u);
            v[8 * j + 2] = __uint_as_float(q.y << 16); v[8 * j + 3] = __uint_as_float(q.y & 0xFFFF0000u);
            v[8 * j + 4] = __uint_as_float(q.z << 16); v[8 * j + 5] = __uint_as_float(q.z & 0xFFFF0000u);
            v[8 * j + 6] = __uint_as_float(q.w << 16); v[8 * j + 7] = __uint_as_float(q.w & 0xFFFF0000u);
        }
    } else {
        const uint32_t a = slot + mis + lane * (uint32_t)(kGrpTok * sizeof(T));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t e = (uint32_t)(16 * h + i) ^ lane;
            if constexpr (sizeof(T) == 4) v[i] = lds32f(a + 4u * e);
            else v[i] = __uint_as_float(lds16u(a + 2u * e) << 16);
        }
    }
}

}  // namespace born
