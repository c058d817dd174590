// The steps on either side of the weight-only decode path in the reference's harness
// (tests/harness_batchsweep.py:77-111, 210-243): the W+A decode GEMV, whose activations are quantised at
// run time into the same MSAQ-signed format as the weights, and the one-off dequantisation of a packed
// weight to bf16 that the reference's prefill feeds to a dense GEMM.
//
// Behaviour replaced: quant_act_msaq_kernel (csrc/wa_gemm.cu:82-108), wa_gemv / wa_gemv_batched
// (csrc/w_gemv.cu:846-1098) and ms_dequant_bf16_kernel (csrc/w_gemv.cu:1242-1275) of the reference.
//
// W+A on this hardware is the weight-only kernel on other inputs: the quantised activation q * 2^e (|q| <=
// 127) is an exact bf16 value, and an exact bf16 value within 2^7 of its block maximum is exact in the
// 16-bit block fixed point the integer-MMA GEMV stages its activations in.  So Y = sum_blocks 2^(ea+ew) *
// intdot(qx, qw), the reference's W+A result, comes out of the same kernels fed the dequantised
// activations; only the activation quantiser is new.
#include "msaq_common.cuh"
#include "sm100_ptx.cuh"

namespace msaq {
namespace {

// One warp per (row, 32-block): the MSAQ-signed int8 word of each element, the block exponent, and (for the
// GEMV that follows) the word's value as bf16.
__global__ void __launch_bounds__(256)
quant_act_kernel(const __nv_bfloat16* __restrict__ X, int8_t* __restrict__ qX, int8_t* __restrict__ sa_exp,
                 __nv_bfloat16* __restrict__ Xdq, int64_t blocks, int64_t NB, Fmt f) {
    chain_release();
    chain_wait();
    const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= blocks) return;
    const int64_t i = w * BLOCK + lane;                       // rows are contiguous: element (m, blk*32 + lane)
    int up, sh;
    const int e = quantize_lane(__bfloat162float(X[i]), lane, f, &up, &sh);
    const int word = up * (1 << f.u) + sh;
    if (qX) qX[i] = (int8_t)word;
    if (sa_exp && lane == 0) sa_exp[w] = (int8_t)e;
    if (Xdq) Xdq[i] = __float2bfloat16_rn((float)word * exp2_int(e));     // exact: at most 8 significant bits
}

// Bits [32i, 32i+32) of the sign bits of n dense codes of `width` bits.
__host__ __device__ constexpr uint32_t sign_bits(int width, int n, int i) {
    uint32_t p = 0;
    for (int b = width - 1; b < width * n; b += width)
        if (b >= 32 * i && b < 32 * i + 32) p |= 1u << (b - 32 * i);
    return p;
}

// The 32 dequantised weights of COLS adjacent columns and one K block as bf16 into Wbf[K][OUT], consecutive threads on
// consecutive columns.  Bound by HBM (25 to 29 bytes in, 64 out).  With the format known at compile time every field is
// cut out with constant shifts, and a code becomes a float through the mantissa: q + 128 + 2^(u-1), which is not negative,
// added to the bits of 2^23 reads as 2^23 plus that, and one fused multiply-add removes the offset and applies the scale
// exactly (at most eight significant bits, so the upper half of the word is the bf16 value).  4096 x 14336 u4, us:
// run-time shifts and an int-to-float conversion per code 160, this one 36 with the shared codes read byte by byte, 27 (0.93 of the
// measured copy rate) with whole words of four columns.
template <int U, int LG_GS, int COLS>
__global__ void __launch_bounds__(128)
dequant_bf16_kernel(const int8_t* __restrict__ scale_exp, const uint8_t* __restrict__ upper_cm,
                    const uint8_t* __restrict__ shared_cm, __nv_bfloat16* __restrict__ Wbf, int64_t OUT) {
    chain_release();
    chain_wait();
    constexpr int WB = 8 - U, UW = WB, NG = 32 >> LG_GS, SB = (NG * U + 7) / 8;      // words of upper, bytes of shared codes
    const int64_t o = ((int64_t)blockIdx.x * 128 + threadIdx.x) * COLS;
    const int64_t blk = blockIdx.y;
    if (o >= OUT) return;
    uint32_t uw[COLS][UW + 1], sw[COLS][3];
    float sc[COLS], off[COLS], post[COLS];
    bool huge = false;
    // the columns' bytes are adjacent: four columns come as whole words (the launcher checks the alignment)
    const int64_t base0 = blk * OUT + o;
    uint32_t se4 = 0u, sraw[SB];
    if constexpr (COLS == 4) {
        se4 = *reinterpret_cast<const uint32_t*>(scale_exp + base0);
#pragma unroll
        for (int i = 0; i < SB; ++i) sraw[i] = reinterpret_cast<const uint32_t*>(shared_cm + base0 * SB)[i];
        const uint4* src = reinterpret_cast<const uint4*>(upper_cm + base0 * (4 * UW));
#pragma unroll
        for (int i = 0; i < UW; ++i) {
            const uint4 x = src[i];
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) uw[(4 * i + k) / UW][(4 * i + k) % UW] = w[k];
        }
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        sw[c][0] = sw[c][1] = sw[c][2] = 0u;
        if constexpr (COLS == 4) {
#pragma unroll
            for (int i = 0; i < SB; ++i) {
                const int at = c * SB + i;
                sw[c][i >> 2] |= (sraw[at >> 2] >> ((at & 3) * 8) & 0xFFu) << ((i & 3) * 8);
            }
        } else {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(upper_cm + base0 * (4 * UW));
#pragma unroll
            for (int i = 0; i < UW; ++i) uw[c][i] = src[i];
#pragma unroll
            for (int i = 0; i < SB; ++i) sw[c][i >> 2] |= (uint32_t)shared_cm[base0 * SB + i] << ((i & 3) * 8);
        }
        uw[c][UW] = 0u;
#pragma unroll
        for (int i = 0; i < UW; ++i) uw[c][i] ^= sign_bits(WB, 32, i);               // every code offset binary
#pragma unroll
        for (int i = 0; i < 2; ++i) sw[c][i] ^= sign_bits(U, NG, i);
        // 2^23 * 2^e overflows above e = 104: such a block is scaled in two steps
        const int e = COLS == 4 ? (int)(int8_t)(se4 >> (8 * c)) : (int)scale_exp[base0];
        huge = huge || e > 100;
        sc[c] = exp2_int(e > 100 ? e - 64 : e);
        off[c] = -(8388608.0f + 128.0f + (float)(1 << (U - 1))) * sc[c];
        post[c] = e > 100 ? 18446744073709551616.0f : 1.0f;
    }
    uint16_t* dst = reinterpret_cast<uint16_t*>(Wbf) + blk * BLOCK * OUT + o;
#pragma unroll
    for (int k = 0; k < BLOCK; ++k) {
        uint32_t v[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const int pu = k * WB, ps = (k >> LG_GS) * U;
            const uint32_t fu = (pu & 31) + WB <= 32 ? uw[c][pu >> 5] >> (pu & 31)
                                                     : __funnelshift_r(uw[c][pu >> 5], uw[c][(pu >> 5) + 1], pu & 31);
            const uint32_t fs = (ps & 31) + U <= 32 ? sw[c][ps >> 5] >> (ps & 31)
                                                    : __funnelshift_r(sw[c][ps >> 5], sw[c][(ps >> 5) + 1], ps & 31);
            const uint32_t bits = ((fu & ((1u << WB) - 1u)) << U) + ((fs & ((1u << U) - 1u)) | 0x4B000000u);
            float f = fmaf(__uint_as_float(bits), sc[c], off[c]);
            if (huge) f *= post[c];
            v[c] = __float_as_uint(f);
        }
        if constexpr (COLS == 4)
            *reinterpret_cast<uint2*>(dst + (int64_t)k * OUT) =
                make_uint2(__byte_perm(v[0], v[1], 0x7632), __byte_perm(v[2], v[3], 0x7632));
        else
            dst[(int64_t)k * OUT] = (uint16_t)(v[0] >> 16);
    }
}

template <int U, int LG_GS>
void launch_dequant(const int8_t* se, const uint8_t* up, const uint8_t* sh, void* Wbf, int64_t OUT, int64_t nb, cudaStream_t st) {
    __nv_bfloat16* w = static_cast<__nv_bfloat16*>(Wbf);
    if (OUT % 4 == 0 && !((reinterpret_cast<uintptr_t>(Wbf) & 7) | (reinterpret_cast<uintptr_t>(up) & 15) |
                          (reinterpret_cast<uintptr_t>(sh) & 3) | (reinterpret_cast<uintptr_t>(se) & 3)))
        launch_chained(dequant_bf16_kernel<U, LG_GS, 4>, dim3((unsigned)((OUT + 511) / 512), (unsigned)nb), dim3(128), 0, st, se, up, sh, w, OUT);
    else
        launch_chained(dequant_bf16_kernel<U, LG_GS, 1>, dim3((unsigned)((OUT + 127) / 128), (unsigned)nb), dim3(128), 0, st, se, up, sh, w, OUT);
}

template <int U>
void launch_dequant_gs(const int8_t* se, const uint8_t* up, const uint8_t* sh, void* Wbf, int64_t OUT, int64_t nb, int lg, cudaStream_t st) {
    switch (lg) {
        case 1: launch_dequant<U, 1>(se, up, sh, Wbf, OUT, nb, st); break;
        case 2: launch_dequant<U, 2>(se, up, sh, Wbf, OUT, nb, st); break;
        case 3: launch_dequant<U, 3>(se, up, sh, Wbf, OUT, nb, st); break;
        case 4: launch_dequant<U, 4>(se, up, sh, Wbf, OUT, nb, st); break;
        default: launch_dequant<U, 5>(se, up, sh, Wbf, OUT, nb, st); break;
    }
}

int launch_quant(const void* X, int8_t* qX, int8_t* sa, void* Xdq, int64_t M, int64_t K, int u, int gs, void* stream) {
    Fmt f;
    if (!make_fmt(u, gs, &f)) return fail(MSAQ_ERR_UNSUPPORTED, "unsupported format u=%d gs=%d", u, gs);
    if (!X) return fail(MSAQ_ERR_ARG, "X is null");
    if (M <= 0 || K <= 0 || K % BLOCK) return fail(MSAQ_ERR_ARG, "M must be positive and K a positive multiple of 32");
    const int64_t blocks = M * (K / BLOCK);
    launch_chained(quant_act_kernel, dim3((unsigned)((blocks + 7) / 8)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                   static_cast<const __nv_bfloat16*>(X), qX, sa, static_cast<__nv_bfloat16*>(Xdq), blocks, K / BLOCK, f);
    count_launch();
    return check_launch("quant_act");
}

}  // namespace
}  // namespace msaq

using namespace msaq;

extern "C" int msaq_quant_act(const void* X, int8_t* qX, int8_t* sa_exp, int64_t M, int64_t K, int u, int gs, void* stream) {
    if (!qX || !sa_exp) return fail(MSAQ_ERR_ARG, "null pointer");
    return launch_quant(X, qX, sa_exp, nullptr, M, K, u, gs, stream);
}

extern "C" size_t msaq_wa_gemv_workspace(int64_t M, int64_t OUT, int64_t NB, int u, int gs) {
    const DeviceScope device;
    const size_t g = msaq_wonly_gemv_workspace(M, OUT, NB, u, gs);
    if (g == 0) return 0;
    return ((g + 255) & ~(size_t)255) + (((size_t)M * NB * BLOCK * 2 + 255) & ~(size_t)255);
}

extern "C" int msaq_wa_gemv_batched(const void* X, const int8_t* scale_exp, const uint8_t* upper_cm,
                                    const uint8_t* shared_cm, void* Y, float* Y_f32, int64_t M, int64_t OUT, int64_t NB,
                                    int u, int gs, void* workspace, size_t workspace_bytes, void* stream) {
    const DeviceScope device;
    if (M <= 0 || OUT <= 0 || NB <= 0) return fail(MSAQ_ERR_ARG, "M, OUT and NB must be positive");
    const size_t tail = ((size_t)M * NB * BLOCK * 2 + 255) & ~(size_t)255;
    const size_t g = gemv_workspace_front(M, OUT, NB, u, gs, tail, workspace_bytes), need = g + tail;
    if (!workspace || workspace_bytes < need)
        return fail(MSAQ_ERR_WORKSPACE, "workspace of %zu bytes needed, %zu given", need, workspace ? workspace_bytes : (size_t)0);
    void* xdq = static_cast<uint8_t*>(workspace) + g;
    if (int rc = launch_quant(X, nullptr, nullptr, xdq, M, NB * BLOCK, u, gs, stream)) return rc;
    return msaq_wonly_gemv_batched(xdq, scale_exp, upper_cm, shared_cm, Y, Y_f32, M, OUT, NB, u, gs, workspace, g, stream);
}

extern "C" int msaq_wa_gemv(const void* x, const int8_t* scale_exp, const uint8_t* upper_cm, const uint8_t* shared_cm,
                            void* y, float* y_f32, int64_t OUT, int64_t NB, int u, int gs, void* workspace,
                            size_t workspace_bytes, void* stream) {
    return msaq_wa_gemv_batched(x, scale_exp, upper_cm, shared_cm, y, y_f32, 1, OUT, NB, u, gs, workspace, workspace_bytes,
                                stream);
}

extern "C" int msaq_dequant_bf16(const int8_t* scale_exp, const uint8_t* upper_cm, const uint8_t* shared_cm, void* Wbf,
                                 int64_t OUT, int64_t K, int u, int gs, void* stream) {
    Fmt f;
    if (!make_fmt(u, gs, &f)) return fail(MSAQ_ERR_UNSUPPORTED, "unsupported format u=%d gs=%d", u, gs);
    if (!scale_exp || !upper_cm || !shared_cm || !Wbf) return fail(MSAQ_ERR_ARG, "null pointer");
    if (OUT <= 0 || K <= 0 || K % BLOCK) return fail(MSAQ_ERR_ARG, "K must be a positive multiple of 32");
    if (K / BLOCK > 65535) return fail(MSAQ_ERR_ARG, "K exceeds the supported range");
    if (reinterpret_cast<uintptr_t>(upper_cm) & 3) return fail(MSAQ_ERR_ARG, "upper_cm must be 4-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (u == 4) launch_dequant_gs<4>(scale_exp, upper_cm, shared_cm, Wbf, OUT, K / BLOCK, f.lg_gs, st);
    else if (u == 3) launch_dequant_gs<3>(scale_exp, upper_cm, shared_cm, Wbf, OUT, K / BLOCK, f.lg_gs, st);
    else launch_dequant_gs<2>(scale_exp, upper_cm, shared_cm, Wbf, OUT, K / BLOCK, f.lg_gs, st);
    count_launch();
    return check_launch("dequant_bf16");
}
