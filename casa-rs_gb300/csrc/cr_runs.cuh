// cr_runs.cuh -- sums of the 7 x 7 taps of a run of records with one start cell.
//
// A warp's four groups of eight lanes take a record each: lane ix of a group
// holds row ix of the footprint (row 7 is padding), its columns as four pairs
// per component, so a record costs the group one x tap, two 16-byte loads of
// y taps and twelve paired FMAs (eight without the PSF).
#pragma once

#include <cstdint>

namespace cr {

// COMPS: (PSF,) re, im -- 3 or 2
template <int COMPS>
struct RunSums {
    float2 acc[4 * COMPS];

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < 4 * COMPS; ++q) acc[q] = make_float2(0.0f, 0.0f);
    }

    // a record of weight w and value v; x: this lane's x tap, y: the y taps in
    // pairs; nothing unless `mine`
    __device__ __forceinline__ void add(bool mine, float x, const float2 (&y)[4], float w,
                                        float2 v) {
        float p[COMPS];
        if (COMPS == 3) p[0] = mine ? __fmul_rn(x, w) : 0.0f;
        p[COMPS - 2] = mine ? __fmul_rn(x, v.x) : 0.0f;
        p[COMPS - 1] = mine ? __fmul_rn(x, v.y) : 0.0f;
#pragma unroll
        for (int c = 0; c < COMPS; ++c)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                acc[4 * c + q] = __ffma2_rn(make_float2(p[c], p[c]), y[q], acc[4 * c + q]);
    }

    // the sums over the groups: group g of lanes gets columns 2 g and 2 g + 1
    // of its lanes' rows
    __device__ __forceinline__ void exchange(int lane, float (&n)[COMPS][2]) const {
        const bool hi = lane & 16, hi2 = lane & 8;
#pragma unroll
        for (int c = 0; c < COMPS; ++c) {
            float m[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const float2 p0 = acc[4 * c + (t >> 1)], p1 = acc[4 * c + 2 + (t >> 1)];
                const float f0 = (t & 1) ? p0.y : p0.x, f1 = (t & 1) ? p1.y : p1.x;
                m[t] = (hi ? f1 : f0) + __shfl_xor_sync(0xffffffffu, hi ? f0 : f1, 16);
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
                n[c][t] = (hi2 ? m[t + 2] : m[t]) +
                          __shfl_xor_sync(0xffffffffu, hi2 ? m[t] : m[t + 2], 8);
        }
    }
};

// a row of the tap table ([rows][8], 16-byte aligned) in pairs
__device__ __forceinline__ void tap_pairs(const float* row, float2 (&y)[4]) {
    const float4* r = reinterpret_cast<const float4*>(row);
    const float4 a = r[0], b = r[1];
    y[0] = make_float2(a.x, a.y);
    y[1] = make_float2(a.z, a.w);
    y[2] = make_float2(b.x, b.y);
    y[3] = make_float2(b.z, b.w);
}

// (re, im) += (x, y) in shared memory, one 64-bit compare-and-swap per try (a
// float32 add is such a loop as well, which the hardware serialises by lane)
__device__ __forceinline__ void shared_add2(float2* p, float x, float y) {
    unsigned long long* q = reinterpret_cast<unsigned long long*>(p);
    unsigned long long old = *q, seen;
    do {
        seen = old;
        const float re = __uint_as_float((uint32_t)seen) + x;
        const float im = __uint_as_float((uint32_t)(seen >> 32)) + y;
        old = atomicCAS(q, seen,
                        (unsigned long long)__float_as_uint(im) << 32 | __float_as_uint(re));
    } while (old != seen);
}

}  // namespace cr
