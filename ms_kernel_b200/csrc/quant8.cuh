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

// sum of 2^(width * i + width - 1), i < n: the sign bits of n packed codes
__host__ __device__ constexpr uint32_t q8_signs(int width, int n) {
    uint32_t p = 0;
    for (int i = 0; i < n; ++i) p |= 1u << (width * i + width - 1);
    return p;
}

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
// Rounding to an integer is one fused multiply-add onto 1.5 * 2^23, and codes are packed as floats: with the sign bit flipped
// they are not negative, so sum((code + 2^(w-1)) * 2^(w*i)) on top of 2^23 leaves the packed field in the mantissa.  (With rintf
// and conversions to int, which share a quarter-rate unit, and a branch per pair the weight packer
// took 338 instructions per 256 weights and 86 us for 14336 x 4096, now 270 and 72 us.)
template <int U>
__device__ __forceinline__ Codes8 quant8(const float (&v)[8]) {
    constexpr int WB = 8 - U, PER = U == 2 ? 2 : 4;                          // upper codes per float: at most 23 bits
    constexpr float LIM = (1 << (7 - U)) - 1, SLO = -(1 << (U - 1)), SHI = (1 << (U - 1)) - 1;
    constexpr float MAGIC = 12582912.0f, TWO23 = 8388608.0f;
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));              // fmaxf passes over a NaN
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    // block_exponent(): floats at or above 1e-30 are the same whether compared in 32 or in 64 bits
    const bool inf = __float_as_uint(amax) == 0x7F800000u;
    const int e = amax >= 1e-30f ? (int)(__float_as_uint(amax) >> 23) - 127 - E_MAX : -100 - E_MAX;
    Codes8 c;
    c.e = inf ? 127 : e;
    const float inv = __int_as_float((127 - (e + U)) << 23), ncoarse = -__int_as_float((127 + e + U) << 23);
    const float half_fine = __int_as_float((126 - e) << 23);                 // 2^-(e+1)
    float q[8], f[4];
    uint32_t slow = inf ? 0xFu : 0u;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        float r[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float x = v[2 * g + i];
            q[2 * g + i] = fminf(fmaxf(fmaf(x, inv, MAGIC), MAGIC - LIM), MAGIC + LIM) - MAGIC;
            r[i] = fmaf(q[2 * g + i], ncoarse, x);
        }
        const float sum = r[0] + r[1], n = fmaf(sum, half_fine, MAGIC) - MAGIC;
        // on a half-way point: was the sum rounded to it?  (It was not if both operands can be had back from it.)
        const float back = sum - r[0];
        if (fabsf(fmaf(sum, half_fine, -n)) == 0.5f && !(back == r[1] && sum - back == r[0])) slow |= 1u << g;
        f[g] = fminf(fmaxf(n, SLO), SHI);
    }
    if (slow) {                                                              // rare: an infinity in the block, a rounded sum
#pragma unroll
        for (int g = 0; g < 4; ++g)
            if (slow >> g & 1u) {
                int ia, ib;
                f[g] = (float)quant8_pair_f64<U>(v[2 * g], v[2 * g + 1], c.e, &ia, &ib);
                q[2 * g] = (float)ia;
                q[2 * g + 1] = (float)ib;
            }
    }
    c.up = 0;
#pragma unroll
    for (int h = 0; h < 8 / PER; ++h) {
        float a = TWO23 + (float)q8_signs(WB, PER);
#pragma unroll
        for (int i = 0; i < PER; ++i) a = fmaf(q[h * PER + i], (float)(1u << (WB * i)), a);
        c.up |= (uint64_t)((__float_as_uint(a) ^ q8_signs(WB, PER)) & ((1u << (WB * PER)) - 1u)) << (h * PER * WB);
    }
    float a = TWO23 + (float)q8_signs(U, 4);
#pragma unroll
    for (int g = 0; g < 4; ++g) a = fmaf(f[g], (float)(1u << (U * g)), a);
    c.sh = (__float_as_uint(a) ^ q8_signs(U, 4)) & ((1u << (4 * U)) - 1u);
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
