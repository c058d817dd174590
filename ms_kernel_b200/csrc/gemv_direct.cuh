// Weight-only GEMV at gs = 2 for few rows without partial sums in global memory: small and medium matrices, where the fixed
// cost of a launch is most of the time.
//
// The pipelined kernels (gemv_mma.cuh, gemv_reg.cuh) share a column tile among thread blocks and pay for it at their end:
// partial sums stored, counted with an atomic and read back, three trips to L2 one after another, behind a ring
// that takes a copy's latency to fill.  Here a thread block (or, where there are few columns, a cluster of them, which adds up
// through distributed shared memory) owns 16 * CG columns over the whole of K.  Its sixteen warps take every sixteenth
// 32-block each, load the packed codes straight into the registers they are decoded from -- runs of 256, 128 and 16
// bytes per block and 16 columns at u = 4, whole sectors -- one block ahead of the arithmetic, and add their sums up
// through shared memory.  No staging launch runs in front: a warp prepares the activations of its own blocks.
//   gemv_direct_int_kernel   u = 4, up to four rows, with or without a fused prologue: integer MMA on 16-bit block fixed
//                            point, the arithmetic and the staged values of gemv_mma.cuh / gemv_xprep_kernel
//   gemv_direct_bf16_kernel  the rest up to 16 rows, plain activations: the exact bf16 arithmetic of gemv_reg.cuh
#pragma once

#include "gemv_reg.cuh"

namespace msaq {

constexpr int GD_WARPS = 16;
constexpr int GD_THREADS = GD_WARPS * 32;
constexpr int GD_MAX_M = 16;
constexpr int GD_MAX_CLUSTER = 8;

// thread blocks per SM: as many as the registers of the codes in flight allow
__host__ __device__ constexpr int gd_int_per_sm(int cg) { return cg == 1 ? 2 : 1; }

struct GemvDirectArgs {
    const int8_t* scale_exp;
    const uint8_t* upper_cm;
    const uint8_t* shared_cm;
    const __nv_bfloat16* X;      // rows at X + m * ldx, 16-byte aligned
    const void* R;               // XP_ADD_NORM: the addend, bf16 or fp32, [rows][K]
    __nv_bfloat16* h_out;        // XP_ADD_NORM: the sum
    __nv_bfloat16* y;            // [rows][OUT]
    float* y_f32;                // optional
    const __nv_bfloat16* res;    // optional: y = bf16(res + bf16(W x))
    int rows, OUT, NB, ldx, r_is_f32, early;
    int cs;                      // thread blocks per cluster, which share their columns
    float eps;
    PeerPush push;               // world == 0: ordinary outputs
};

__device__ __forceinline__ uint32_t ldg32_stream(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg16_stream(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg8_stream(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int ldg_s8_stream(const void* p) {
    int v;
    asm volatile("ld.global.nc.L1::no_allocate.s8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ uint2 ldg64_stream(const void* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// ---- cluster: the thread blocks that share a set of columns ----------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t saddr, uint32_t rank) {
    float v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
                 : "=f"(v) : "r"(saddr), "r"(rank) : "memory");
    return v;
}

// The end of a thread block: the warps' sums red[warp][row][column] are added in warp order, the cluster's in rank order
// (the same bits on every run), and the outputs written.  `part`: rows * COLS floats of shared memory.
template <int ROWS, int COLS, int WARPS = GD_WARPS>
__device__ __forceinline__ void gd_finish(const GemvDirectArgs& a, const float (*red)[ROWS][COLS], float* part, int c0) {
    const int tid = threadIdx.x;
    __syncthreads();
    if (a.cs > 1) {
        for (int i = tid; i < a.rows * COLS; i += GD_THREADS) {
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) v += red[w][i / COLS][i % COLS];
            part[i] = v;
        }
        cluster_sync();
    }
    if (a.cs == 1 || cluster_rank() == 0) {
        for (int i = tid; i < a.rows * COLS; i += GD_THREADS) {
            const int m = i / COLS, c = i % COLS;
            float v = 0.0f;
            if (a.cs > 1) {
                float p[GD_MAX_CLUSTER];
#pragma unroll
                for (int r = 0; r < GD_MAX_CLUSTER; ++r) p[r] = r < a.cs ? ld_cluster_f32(smem_u32(part + i), r) : 0.0f;
#pragma unroll
                for (int r = 0; r < GD_MAX_CLUSTER; ++r) v += p[r];
            } else {
#pragma unroll
                for (int w = 0; w < WARPS; ++w) v += red[w][m][c];
            }
            if (c0 + c < a.OUT) {
                const int64_t o = (int64_t)m * a.OUT + c0 + c;
                if (a.push.world) {
                    gemv_push(a.push, o, v, gemv_push_seq(a.push));
                } else {
                    if (a.y_f32) a.y_f32[o] = v;
                    __nv_bfloat16 y = __float2bfloat16_rn(v);
                    if (a.res) y = __float2bfloat16_rn(__bfloat162float(a.res[o]) + __bfloat162float(y));
                    a.y[o] = y;
                }
            }
        }
    }
    if (a.cs > 1) cluster_sync();                    // shared memory stays until rank 0 has read it
}

// ---- integer arithmetic: u = 4, up to four rows, fused prologues ------------------------------------
// The packed codes of 16 columns (rows g and g + 8 of the MMA's A operand) of one 32-block.
struct GdCodes {
    uint2 w0, w1;
    uint32_t s0, s1;
    int e0, e1;
};

template <int MODE, int CG, int ROWS>
__global__ void __launch_bounds__(GD_THREADS, gd_int_per_sm(CG))
gemv_direct_int_kernel(const GemvDirectArgs a) {
    constexpr int COLS = 16 * CG;
    __shared__ __align__(8) uint8_t rec[GD_WARPS][2][ROWS * 64 + 32];     // staged planes of one 32-block, {corr, cx} of each row
    __shared__ float red[GD_WARPS][ROWS][COLS];
    __shared__ float part[ROWS * COLS];
    __shared__ float norm_red[ROWS][GD_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3, h = t >> 1, odd = t & 1;
    const int stride = GD_WARPS * a.cs, tile = blockIdx.x / a.cs, c0 = tile * COLS, K = a.NB * BLOCK;
    const int first = (a.cs > 1 ? (int)cluster_rank() : 0) * GD_WARPS + warp;      // this warp's blocks: first, first + stride, ...
    const int ngroups = min(CG, (a.OUT - c0) >> 4);
    const uint32_t sel = odd ? 0x7531u : 0x6420u, nshift = odd * 4;

    const uint8_t* pu = a.upper_cm + ((int64_t)first * a.OUT + c0 + g) * 16 + h * 8;
    const uint8_t* ps = a.shared_cm + ((int64_t)first * a.OUT + c0 + g) * 8 + h * 4;
    const int8_t* pe = a.scale_exp + (int64_t)first * a.OUT + c0 + g;
    const int64_t de = (int64_t)stride * a.OUT, du = de * 16, ds = de * 8;
    auto load = [&](GdCodes (&k)[CG]) {
#pragma unroll
        for (int q = 0; q < CG; ++q) {
            if (q < ngroups) {
                k[q].w0 = ldg64_stream(pu + q * 256);
                k[q].w1 = ldg64_stream(pu + q * 256 + 128);
                k[q].s0 = ldg32_stream(ps + q * 128);
                k[q].s1 = ldg32_stream(ps + q * 128 + 64);
                k[q].e0 = ldg_s8_stream(pe + q * 16);
                k[q].e1 = ldg_s8_stream(pe + q * 16 + 8);
            }
        }
        pu += du;
        ps += ds;
        pe += de;
    };
    // The activation element of this lane in a block (and its partner: the up projection's value, the addend) as loaded: what is
    // computed from it waits until the block's turn, or the load would be waited for where it is issued.
    struct Raw { uint32_t x, r; };
    auto load_x = [&](int kb, Raw (&raw)[ROWS]) {
        const int k = kb * BLOCK + lane;
#pragma unroll
        for (int m = 0; m < ROWS; ++m) {
            raw[m] = Raw{0u, 0u};
            if (m < a.rows) {
                const unsigned short* xr = reinterpret_cast<const unsigned short*>(a.X + (int64_t)m * a.ldx);
                raw[m].x = xr[k];
                if (MODE == XP_SILU_MUL) raw[m].r = xr[K + k];
                if (MODE == XP_ADD_NORM) {
                    const int64_t o = (int64_t)m * K + k;
                    raw[m].r = a.r_is_f32 ? static_cast<const uint32_t*>(a.R)[o] : (uint32_t)static_cast<const unsigned short*>(a.R)[o];
                }
            }
        }
    };
    auto activation = [&](int kb, int m, const Raw& raw, float inv) {
        float x = __uint_as_float(raw.x << 16);
        if (MODE == XP_SILU_MUL) {
            const float up = __uint_as_float(raw.r << 16);
            x = __bfloat162float(__float2bfloat16_rn(x / (1.0f + __expf(-x)) * up));
        }
        if (MODE == XP_ADD_NORM) {
            const float d = a.r_is_f32 ? __uint_as_float(raw.r) : __uint_as_float(raw.r << 16);
            const __nv_bfloat16 hb = __float2bfloat16_rn(x + d);
            if (tile == 0 && m < a.rows) a.h_out[(int64_t)m * K + kb * BLOCK + lane] = hb;
            x = __bfloat162float(hb);
        }
        if (MODE == XP_RMSNORM || MODE == XP_ADD_NORM) x = __bfloat162float(__float2bfloat16_rn(x * inv));
        return x;
    };

    GdCodes cur[2][CG];
    Raw xc[2][ROWS];
#pragma unroll
    for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int q = 0; q < CG; ++q) cur[d][q] = GdCodes{make_uint2(0u, 0u), make_uint2(0u, 0u), 0u, 0u, 0, 0};
    // with MSAQ_OPT_EARLY_WEIGHTS the caller vouches for the weights: they need not wait for the kernel in front
    if (a.early && first < a.NB) load(cur[0]);
    chain_wait();
    if (!a.early && first < a.NB) load(cur[0]);
    if (first < a.NB) load_x(first, xc[0]);

    float inv_rms[ROWS];
#pragma unroll
    for (int m = 0; m < ROWS; ++m) inv_rms[m] = 1.0f;
    if (MODE == XP_RMSNORM || MODE == XP_ADD_NORM) {
        // every thread block takes the norm of the whole rows, in the same order: the same bits everywhere
#pragma unroll
        for (int m = 0; m < ROWS; ++m) {
            float ss = 0.0f;
            if (m < a.rows) {
                const uint4* xr = reinterpret_cast<const uint4*>(a.X + (int64_t)m * a.ldx);
                for (int i = tid; i < K / 8; i += GD_THREADS) {
                    const uint4 hv = xr[i];
                    const uint32_t w[4] = {hv.x, hv.y, hv.z, hv.w};
                    float f[8];
#pragma unroll
                    for (int j = 0; j < 4; ++j) { f[2 * j] = bf16_lo(w[j]); f[2 * j + 1] = bf16_hi(w[j]); }
                    if (MODE == XP_ADD_NORM) {
                        const int64_t o = (int64_t)m * K + i * 8;          // 16-byte aligned: the entry point checks the bases
                        float d[8];
                        if (a.r_is_f32) {
                            const float4 d0 = *reinterpret_cast<const float4*>(static_cast<const float*>(a.R) + o);
                            const float4 d1 = *reinterpret_cast<const float4*>(static_cast<const float*>(a.R) + o + 4);
                            d[0] = d0.x; d[1] = d0.y; d[2] = d0.z; d[3] = d0.w; d[4] = d1.x; d[5] = d1.y; d[6] = d1.z; d[7] = d1.w;
                        } else {
                            const uint4 dv = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.R) + o);
                            const uint32_t dw[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) { d[2 * j] = bf16_lo(dw[j]); d[2 * j + 1] = bf16_hi(dw[j]); }
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16_rn(f[j] + d[j]));
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) ss = fmaf(f[j], f[j], ss);
                }
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) norm_red[m][warp] = ss;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < ROWS; ++m) {
            float tot = 0.0f;
#pragma unroll
            for (int w = 0; w < GD_WARPS; ++w) tot += norm_red[m][w];
            inv_rms[m] = rsqrtf(tot / (float)K + a.eps);
        }
    }

    float acc[CG][2];
#pragma unroll
    for (int q = 0; q < CG; ++q) acc[q][0] = acc[q][1] = 0.0f;
    // thread-slot and byte of this lane's element in the staged planes (the layout of gemv_xprep_kernel)
    const int slot = (2 * (lane >> 4) + ((lane >> 1) & 1)) * 8 + (lane & 1) * 4 + ((lane & 15) >> 2);
    for (int kb0 = first; kb0 < a.NB; kb0 += 2 * stride) {
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int kb = kb0 + d * stride;
            if (kb >= a.NB) break;
            if (kb + stride < a.NB) {
                load(cur[d ^ 1]);
                load_x(kb + stride, xc[d ^ 1]);
            }
            // ---- stage this block's activations: 16-bit block fixed point, two int8 planes ----
            uint8_t* r = rec[warp][d];
#pragma unroll
            for (int m = 0; m < ROWS; ++m) {
                const float x = activation(kb, m, xc[d][m], inv_rms[m]);
                const uint32_t ax = __reduce_max_sync(0xffffffffu, __float_as_uint(x) & 0x7FFFFFFFu);
                int E = (int)(ax >> 23) - 127;
                E = ax == 0u ? 0 : max(-100, min(127, E));
                const int xi = min(__float2int_rn(x * __int_as_float((14 - E + 127) << 23)), 32639);
                const int lo = (int)(int8_t)(xi & 0xFF), hi = (xi - lo) >> 8;
                r[(2 * m) * 32 + slot] = (uint8_t)hi;
                r[(2 * m + 1) * 32 + slot] = (uint8_t)lo;
                const int sx = __reduce_add_sync(0xffffffffu, xi);
                if (lane == 0) {
                    // the offset-binary shared codes add 8 per element; an Inf or NaN makes the multiplier, and the row, NaN
                    int* tc = reinterpret_cast<int*>(r + ROWS * 64 + m * 8);
                    tc[0] = -8 * sx;
                    tc[1] = ax >= 0x7F800000u ? 0x7FC00000 : (int)((uint32_t)(E - 14 + 127) << 23);
                }
            }
            __syncwarp();                 // (the other buffer is free: every lane is past its reads of it)
            const uint32_t rb = smem_u32(r);
            uint2 bq = make_uint2(0u, 0u), tc = make_uint2(0u, 0u);
            if (g < 2 * ROWS) bq = lds64<0>(rb + g * 32 + t * 8);
            if (t < ROWS) tc = lds64<ROWS * 64>(rb + t * 8);
            const uint32_t B[2] = {bq.x, bq.y};
            const float cx = __uint_as_float(tc.y);
#pragma unroll
            for (int q = 0; q < CG; ++q) {
                if (q < ngroups) {
                    const GdCodes& k = cur[d][q];
                    const uint32_t m0 = and_xor(k.s0 >> nshift, 0x0F0F0F0Fu, 0x08080808u);
                    const uint32_t m1 = and_xor(k.s1 >> nshift, 0x0F0F0F0Fu, 0x08080808u);
                    const uint32_t x0 = prmt(k.w0.x, k.w0.y, sel), x1 = prmt(k.w1.x, k.w1.y, sel);
                    uint32_t A[4];
                    A[0] = and_or(x0 << 4, 0xF0F0F0F0u, m0);
                    A[1] = and_or(x1 << 4, 0xF0F0F0F0u, m1);
                    A[2] = and_or(x0, 0xF0F0F0F0u, m0);
                    A[3] = and_or(x1, 0xF0F0F0F0u, m1);
                    const float sw0 = __int_as_float(k.e0 * (1 << 23) + (127 << 23));
                    const float sw1 = __int_as_float(k.e1 * (1 << 23) + (127 << 23));
                    int D[4];
                    mma_s8_16832_c(D, A, B, (int)tc.x);
                    acc[q][0] = fmaf((float)(D[0] * 256 + D[1]) * cx, sw0, acc[q][0]);
                    acc[q][1] = fmaf((float)(D[2] * 256 + D[3]) * cx, sw1, acc[q][1]);
                }
            }
        }
    }
    if (t < ROWS) {
#pragma unroll
        for (int q = 0; q < CG; ++q) {
            red[warp][t][q * 16 + g] = acc[q][0];
            red[warp][t][q * 16 + g + 8] = acc[q][1];
        }
    }
    gd_finish<ROWS, COLS>(a, red, part, c0);
}

// ---- exact bf16 arithmetic: any u, up to 16 rows, plain activations --------------------------------
template <int U, int MT, int CG>
__global__ void __launch_bounds__(GD_THREADS, 1)
gemv_direct_bf16_kernel(const GemvDirectArgs a) {
    constexpr int COLS = 16 * CG, UB = gr_ub(U), SB = gr_sb(U), ROWS = 8 * MT;
    constexpr int HALVES = MT > 1 ? 2 : 1, WARPS = GD_WARPS / HALVES;        // 16 rows: half of the warps add theirs to the others'
    __shared__ float red[WARPS][ROWS][COLS];
    __shared__ float part[ROWS * COLS];
    __shared__ __align__(16) uint32_t consts[GrConst<U>::N];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int stride = GD_WARPS * a.cs, tile = blockIdx.x / a.cs, c0 = tile * COLS;
    const int first = (a.cs > 1 ? (int)cluster_rank() : 0) * GD_WARPS + warp;
    const int ngroups = min(CG, (a.OUT - c0) >> 4);
    const GrLane ln = gr_lane<U>(t);
    if (tid == 0) GrConst<U>::store(consts);

    const int64_t col = (int64_t)first * a.OUT + c0 + g;
    const uint8_t* pu = a.upper_cm + col * UB + ln.up_off;
    const uint8_t* ps = a.shared_cm + col * SB + ln.sh_off;
    const int8_t* pe = a.scale_exp + col;
    const int64_t step = (int64_t)stride * a.OUT;
    auto load = [&](GrRaw (&k)[CG][2]) {
#pragma unroll
        for (int q = 0; q < CG; ++q) {
            if (q < ngroups) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {                        // rows g and g + 8 of the fragment
                    const int c = q * 16 + i * 8;
                    GrRaw& r = k[q][i];
                    r.w0 = ldg32_stream(pu + c * UB);
                    if (U != 4) r.w1 = ldg32_stream(pu + c * UB + 4);
                    if (U == 2) r.s0 = ldg8_stream(ps + c * SB);
                    else r.s0 = ldg16_stream(ps + c * SB);
                    if (U == 3) r.s1 = ldg16_stream(ps + c * SB - ln.sh_off + ln.sh_off2);
                    r.e = ldg_s8_stream(pe + c);
                }
            }
        }
        pu += step * UB;
        ps += step * SB;
        pe += step;
    };
    auto load_x = [&](int kb, uint4 (&v)[MT]) {
#pragma unroll
        for (int n = 0; n < MT; ++n) {
            v[n] = make_uint4(0u, 0u, 0u, 0u);
            if (n * 8 + g < a.rows) v[n] = *reinterpret_cast<const uint4*>(a.X + (int64_t)(n * 8 + g) * a.ldx + kb * BLOCK + t * 8);
        }
    };

    GrRaw cur[2][CG][2];
    uint4 xc[2][MT];
#pragma unroll
    for (int d = 0; d < 2; ++d)
#pragma unroll
        for (int q = 0; q < CG; ++q) cur[d][q][0] = cur[d][q][1] = GrRaw{0u, 0u, 0u, 0u, 0};
    if (a.early && first < a.NB) load(cur[0]);
    chain_wait();
    if (!a.early && first < a.NB) load(cur[0]);
    if (first < a.NB) load_x(first, xc[0]);
    __syncthreads();
    const GrConst<U> kc(smem_u32(consts));

    float acc[CG][gr_accs(MT)][4];
#pragma unroll
    for (int q = 0; q < CG; ++q)
#pragma unroll
        for (int n = 0; n < gr_accs(MT); ++n) acc[q][n][0] = acc[q][n][1] = acc[q][n][2] = acc[q][n][3] = 0.0f;
    for (int kb0 = first; kb0 < a.NB; kb0 += 2 * stride) {
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int kb = kb0 + d * stride;
            if (kb >= a.NB) break;
            if (kb + stride < a.NB) {
                load(cur[d ^ 1]);
                load_x(kb + stride, xc[d ^ 1]);
            }
            uint32_t b[MT][4];
#pragma unroll
            for (int n = 0; n < MT; ++n) {
                const uint4 x = gr_finite_or_nan<U, MT>(xc[d][n]);
                b[n][0] = prmt(x.x, x.z, 0x5410u);
                b[n][1] = prmt(x.x, x.z, 0x7632u);
                b[n][2] = prmt(x.y, x.w, 0x5410u);
                b[n][3] = prmt(x.y, x.w, 0x7632u);
            }
#pragma unroll
            for (int q = 0; q < CG; ++q) {
                if (q < ngroups) {
                    uint32_t w0[4], w1[4];
                    gr_decode<U>(cur[d][q][0], ln, kc, w0);
                    gr_decode<U>(cur[d][q][1], ln, kc, w1);
                    gr_mma<MT, gr_accs(MT)>(acc[q], w0, w1, b);
                }
            }
        }
    }
    if constexpr (MT == 1) {
#pragma unroll
        for (int q = 0; q < CG; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[q][0][i] += acc[q][1][i];
    }
#pragma unroll
    for (int half = 0; half < HALVES; ++half) {
        if (half) __syncthreads();
        if (warp / WARPS == HALVES - 1 - half) {
#pragma unroll
            for (int q = 0; q < CG; ++q)
#pragma unroll
                for (int n = 0; n < MT; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int m = n * 8 + 2 * t + (i & 1);
                        float* r = &red[warp % WARPS][m][q * 16 + g + (i >> 1) * 8];
                        if (m < a.rows) *r = half ? *r + acc[q][n][i] : acc[q][n][i];
                    }
        }
    }
    gd_finish<ROWS, COLS, WARPS>(a, red, part, c0);
}

// gemv_direct.cu.  Column groups per thread block and thread blocks per cluster for these sizes, and the model's cycles; false:
// not one wave.
bool gemv_direct_pick(int64_t M, int64_t OUT, int64_t NB, int u, int* cg, int* cs, int64_t* cycles);
int gemv_direct_launch(const GemvDirectArgs& a, int u, int mode, int cg, cudaStream_t st);

}  // namespace msaq
