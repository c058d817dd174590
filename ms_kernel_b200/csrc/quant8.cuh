// The gs = 2 block quantiser on eight consecutive values per thread, four neighbouring lanes to a 32-block: the body of
// the weight packer (weight_pack.cu) and of the cache writers (kv_quant_row.cuh).
//
// Codes equal those of ms_lib/pack.py:47-60 of the reference (float64) bit for bit, in fp32:
//   * scaling by a power of two is exact, so rint(x / 2^(e+u)) is the same number;
//   * the residual x - q * 2^(e+u) is a multiple of x's last place and no larger than x (or than the grid step when q is
//     clipped), hence representable: one fused multiply-add gives it exactly;
//   * the sum of a pair's residuals is rounded, but rounding is monotonic and the half-way points of the shared
//     code are representable: only a sum that comes out ON a half-way point and was rounded to it can end on the other
//     side, and such a pair -- and any block with an infinity in it -- is evaluated in float64.
#pragma once

#include "msaq_common.cuh"

namespace msaq {

struct Codes8 {
    uint64_t up;      // eight upper codes of 8 - u bits, dense, first one lowest
    uint32_t sh;      // four shared codes of u bits
    int e;            // the block's exponent
};

template <int U>
__device__ __forceinline__ int quant8_pair_f64(float x0, float x1, int e, int* q0, int* q1) {
    const double lim = (1 << (7 - U)) - 1, slo = -(1 << (U - 1)), shi = (1 << (U - 1)) - 1;
    const double inv = __hiloint2double((1023 - (e + U)) << 20, 0), coarse = __hiloint2double((1023 + e + U) << 20, 0);
    const double a = (double)x0, b = (double)x1;
    const double qa = fmin(fmax(rint(a * inv), -lim), lim), qb = fmin(fmax(rint(b * inv), -lim), lim);
    const double sum = (a - qa * coarse) + (b - qb * coarse);
    *q0 = (int)qa;
    *q1 = (int)qb;
    return (int)fmin(fmax(rint(sum * __hiloint2double((1022 - e) << 20, 0)), slo), shi);
}

// All 32 lanes take part; lanes 4i..4i+3 hold one block, lane 4i + p the elements 8p..8p+7.
template <int U>
__device__ __forceinline__ Codes8 quant8(const float (&v)[8]) {
    constexpr int WB = 8 - U;
    constexpr float LIM = (1 << (7 - U)) - 1, SLO = -(1 << (U - 1)), SHI = (1 << (U - 1)) - 1;
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));              // fmaxf passes over a NaN
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    Codes8 c;
    c.e = block_exponent(amax);
    c.up = 0;
    c.sh = 0;
    const bool inf = c.e > 121;                                              // no finite value has this exponent
    const int e = inf ? 0 : c.e;
    const float inv = __int_as_float((127 - (e + U)) << 23), coarse = __int_as_float((127 + e + U) << 23);
    const float half_fine = __int_as_float((126 - e) << 23);                 // 2^-(e+1)
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const float a = v[2 * g], b = v[2 * g + 1];
        const float qa = fminf(fmaxf(rintf(a * inv), -LIM), LIM), qb = fminf(fmaxf(rintf(b * inv), -LIM), LIM);
        const float ra = fmaf(-qa, coarse, a), rb = fmaf(-qb, coarse, b);
        const float sum = ra + rb, t = sum * half_fine, n = rintf(t);
        int ia = (int)qa, ib = (int)qb, is = (int)fminf(fmaxf(n, SLO), SHI);
        bool exact = !inf;
        if (fabsf(t - n) == 0.5f) {                                          // on a half-way point: was the sum rounded to it?
            const float bb = sum - ra;
            exact = exact && (ra - (sum - bb)) + (rb - bb) == 0.0f;
        }
        if (!exact) is = quant8_pair_f64<U>(a, b, c.e, &ia, &ib);
        const uint32_t pair = ((uint32_t)ia & ((1u << WB) - 1u)) | (((uint32_t)ib & ((1u << WB) - 1u)) << WB);
        c.up |= (uint64_t)pair << (2 * g * WB);
        c.sh |= ((uint32_t)is & ((1u << U) - 1u)) << (g * U);
    }
    return c;
}

// Stores the codes of a block: `up` and `sh` point at the block's UB and SB bytes (4- and 2-byte aligned; u = 2: any
// alignment for sh).  All 32 lanes take part, those with live == false store nothing.
template <int U>
__device__ __forceinline__ void quant8_store(const Codes8& c, int lane, bool live, uint8_t* up, uint8_t* sh) {
    constexpr int WB = 8 - U;
    const int p = lane & 3;
    if constexpr (U == 4) {
        if (live) {
            reinterpret_cast<uint32_t*>(up)[p] = (uint32_t)c.up;
            reinterpret_cast<uint16_t*>(sh)[p] = (uint16_t)c.sh;
        }
    } else {
        // a lane stores the words (and, u = 3, the half-words of shared codes) that begin in its run of bits; their ends
        // may come from the next lane's
        const uint64_t nxt = __shfl_down_sync(0xffffffffu, c.up, 1);
        const uint32_t nsh = __shfl_down_sync(0xffffffffu, c.sh, 1);
        if (live) {
            const int w0 = (p * WB + 3) >> 2;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int w = w0 + k, off = 32 * w - p * 8 * WB;
                if (off < 8 * WB) reinterpret_cast<uint32_t*>(up)[w] = (uint32_t)((c.up >> off) | (nxt << (8 * WB - off)));
            }
            if constexpr (U == 3) {
                if (p < 3) reinterpret_cast<uint16_t*>(sh)[p] = (uint16_t)((c.sh >> (4 * p)) | (nsh << (12 - 4 * p)));
            } else {
                sh[p] = (uint8_t)c.sh;
            }
        }
    }
}

}  // namespace msaq
