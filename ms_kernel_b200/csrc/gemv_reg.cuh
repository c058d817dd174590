// Weight-only GEMV for small batches on register operands, Y[M][OUT] = X[M][K] * dequant(W)^T at gs = 2, up to 64 rows (which
// sizes: reg_serves() in gemv.cu).
//
// What bounds it is the widening of the codes up to 16 rows, the rate of the warp-level MMA above (eight cycles each), then HBM.
// The tensor-memory kernel (gemv_umma.cuh) pays for the same widening a trip through shared memory, a proxy fence and two
// barrier hand-offs per unit with one thread block per SM, and its 128-row activation tile is mostly padding at these
// batches.  Here a lane widens the codes of its own MMA fragment in registers and nothing else touches them:
//   * the weights are the 16-row A operand of mma.m16n8k16 (bf16 in, fp32 out), eight activation rows the B operand;
//   * the sum over K may take its terms in any order, so lane t of a row's four takes the eight CONTIGUOUS elements
//     8t..8t+7 of a 32-block -- one aligned run of the packed bytes -- as the pairs (j, j + 4), j = 0..3, and
//     the activations are read from shared memory as they lie in X (one 16-byte load per eight rows, four byte
//     permutes): no staging kernel runs in front;
//   * the code q * 2^e is exact in bf16 (see gr_decode_row), so products are exact in fp32 and one accumulator runs over
//     the thread block's whole K range: no work per 32-block behind the MMA;
//   * one thread block per SM, on the schedule and the per-warp tile hand-off of gemv_mma.cuh.
// Measured (28672 x 4096, u = 4, 16 rows: 52.2 -> 37.4 us, of which copies and fixed costs alone take 22 us): 88 instructions in
// all per 16 x 32 weights, ALU pipe 44 % and FMA pipe 37 % busy.  Copies of a stage are issued by lanes in one instruction, four K blocks
// to a stage: a copy-issuing warp spends about 0.4 us on a stage whatever its size (two K blocks: 41.6 us), which is also
// why each team has its own (one for both: 42.4 us).
//
// Algorithm replaced: csrc/w_gemv.cu:173-487 of the reference (its wide and batched kernels at u = 2, 3 and at M > 8).
#pragma once

#include "gemv_mma.cuh"

namespace msaq {

constexpr int GR_MAX_M = 64;                       // activation rows per launch
// 128-column groups per tile, by n-tiles of eight activation rows.  Eighteen warps leave a thread 96 registers: one and two n-tiles fit
// with two groups, four n-tiles (17 to 32 rows) spill 240 to 300 bytes of it, eight, with one group, 20 to 60.
__host__ __device__ constexpr int gr_groups_of(int mt) { return mt <= 4 ? 2 : 1; }
__host__ __device__ constexpr int gr_tc(int mt) { return gr_groups_of(mt) * GM_GROUP; }
constexpr int GR_KB = 4;                           // K blocks per ring stage
// bytes between activation rows of a stage: 64 beyond the data, so that the 16-byte loads of two neighbouring rows fall
// into different halves of the banks
constexpr int GR_XROW = GR_KB * 64 + 64;
__host__ __device__ constexpr int gr_ub(int u) { return 4 * (8 - u); }      // bytes of upper and of shared codes per 32-block
__host__ __device__ constexpr int gr_sb(int u) { return 2 * u; }
// Teams of eight consumer warps with a copy-issuing warp and a ring each, taking alternate units: one thread block per SM
// with two teams has as many warps in flight as two thread blocks and leaves half the partial sums.
constexpr int GR_TEAMS = 2;
constexpr int GR_THREADS = GR_TEAMS * (GM_WARPS + 1) * 32;
__host__ __device__ constexpr int gr_sub_bytes(int u, int mt) { return gr_tc(mt) * (gr_ub(u) + gr_sb(u) + 1); }    // one K block of a tile
__host__ __device__ constexpr int gr_stage_bytes(int u, int mt) { return GR_KB * gr_sub_bytes(u, mt) + mt * 8 * GR_XROW; }
// the accumulators that the other teams hand to the first
__host__ __device__ constexpr int gr_merge_bytes(int mt) { return (GR_TEAMS - 1) * GM_WARPS * gr_groups_of(mt) * mt * 512; }

__device__ __forceinline__ uint32_t hfma2_bf16(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// D(16x8, f32) += A(16x16, bf16, row) * B(16x8, bf16, col)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <int OFF>
__device__ __forceinline__ uint32_t lds_u16(uint32_t base) {
    uint32_t v;
    asm volatile("ld.shared.u16 %0, [%1+%2];" : "=r"(v) : "r"(base), "n"(OFF));
    return v;
}

// A lane's place in a row's packed block: byte offsets of its codes and the bit shifts that align them.
struct GrLane {
    uint32_t up_off, up_shift, sh_off, sh_off2, sh_shift;
};
template <int U>
__device__ __forceinline__ GrLane gr_lane(int t) {
    if constexpr (U == 4) return {4u * t, 0u, 2u * t, 0u, 0u};                            // 32 bits; 16 bits
    else if constexpr (U == 3) {                                                          // 40 bits at byte 5t; 12 bits at bit 12t
        const uint32_t a = (3u * t) >> 2;
        return {4u * t, 8u * t, 2u * a, 2u * min(a + 1u, 2u), 12u * t - 16u * a};
    } else return {(6u * t) & ~3u, 16u * (t & 1), 1u * t, 0u, 0u};                        // 48 bits at byte 6t; 8 bits at byte t
}

// Eight weights of one row as bf16 pairs: w[j] = elements (8t + j, 8t + j + 4) of the 32-block.
//
// q = up * 2^u + sh.  A code with its sign bit flipped, dropped into the mantissa of bf16 128.0, reads as 128 + 2^(b-1) + code
// (b its width).  h = (sh + 64) * 2^e and then h + (up - 64 / 2^u) * 2^(u+e) are formed with one fused multiply-add each; every
// value on the way is an integer of at most eight significant bits times a power of two, so nothing is rounded.  The 64 that goes
// from one part to the other keeps the offsets, -(64 + 2^(u-1)) * 2^e among them, inside bf16 over the whole range of block
// exponents that finite weights have (up to 121; with -(128 + 2^(u-1)) * 2^e weights of 2^127 and more came out as Inf or NaN).
// The constants of the decode below, read back from shared memory once: as literals they are put into registers again at
// every use (LOP3 and HFMA2 take one immediate at most), which doubles the instructions of a step.
template <int U>
struct GrConst {
    static constexpr int WB = 8 - U;
    static constexpr int N = 9;
    uint32_t um, ux, sm, sx, uoff, soff, two_u, one, neg0;
    __device__ static __forceinline__ constexpr uint32_t value(int i) {
        switch (i) {
            case 0: return ((1u << WB) - 1u) * 0x00010001u;                          // an upper code in each half
            case 1: return 0x43004300u | (0x00010001u << (WB - 1));                  // bf16 128.0, and the code's sign bit
            case 2: return ((1u << U) - 1u) * 0x00010001u;
            case 3: return 0x43004300u | (0x00010001u << (U - 1));
            case 4: return (U == 4 ? 0xC30Cu : U == 3 ? 0xC318u : 0xC330u) * 0x00010001u;     // -(128 + 2^(WB-1) + 64 / 2^U)
            case 5: return (U == 4 ? 0xC290u : U == 3 ? 0xC288u : 0xC284u) * 0x00010001u;     // -(64 + 2^(U-1))
            case 6: return ((127u + U) << 7) * 0x00010001u;                          // 2^U
            case 7: return 0x3F803F80u;
            default: return 0x80008000u;                                             // -0: the neutral addend
        }
    }
    // by one thread, all of them immediates (a thread per constant looks its own up in constant memory: 0.1 us of a launch)
    __device__ static __forceinline__ void store(uint32_t* consts) {
#pragma unroll
        for (int i = 0; i < N; ++i) consts[i] = value(i);
    }
    __device__ __forceinline__ explicit GrConst(uint32_t a) {
        uint32_t* const v[N] = {&um, &ux, &sm, &sx, &uoff, &soff, &two_u, &one, &neg0};
#pragma unroll
        for (int i = 0; i < N; ++i) asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(*v[i]) : "r"(a + 4 * i) : "memory");
    }
};

// A lane's share of a row's packed block as loaded: u = 4: w0, s0; u = 3: both words and both half-words; u = 2: both words, s0.
struct GrRaw {
    uint32_t w0, w1, s0, s1;
    int e;
};

template <int U>
__device__ __forceinline__ void gr_decode(const GrRaw& in, const GrLane& ln, const GrConst<U>& k, uint32_t (&w)[4]) {
    constexpr int WB = 8 - U;
    const uint32_t s = (uint32_t)(in.e * 0x00800080 + 0x3F803F80);                    // 2^e twice
    const uint32_t su = hfma2_bf16(s, k.two_u, k.neg0), ns = hfma2_bf16(s, k.soff, k.neg0);

    uint32_t f[4];                       // upper codes j (low half) and j + 4 (high half), other bits arbitrary
    if constexpr (U == 4) {
        f[0] = in.w0; f[1] = in.w0 >> 4; f[2] = in.w0 >> 8; f[3] = in.w0 >> 12;
    } else {
        const uint32_t lo = __funnelshift_r(in.w0, in.w1, ln.up_shift), hi = in.w1 >> ln.up_shift;  // bits 0..31, 32.. of this lane's run
        const uint32_t up4 = __funnelshift_r(lo, hi, 4 * WB);                               // codes 4..7
        const uint32_t c = prmt(lo, up4, 0x5410u);                                          // low halves
        f[0] = c;
        f[1] = c >> WB;
        if constexpr (WB == 5) {
            f[2] = c >> 10;
            f[3] = prmt(lo, up4, 0x6521u) >> 7;                                             // bits 8..23 of each: code 3 at bit 7
        } else {
            const uint32_t d = prmt(lo, up4, 0x6521u);
            f[2] = d >> 4;                                                                  // code 2 at bit 12 = 8 + 4
            f[3] = d >> 10;
        }
    }
    uint32_t g;                          // shared codes 0, 1 (low half) and 2, 3 (high half)
    if constexpr (U == 4) g = prmt(in.s0, 0u, 0x4140u);
    else if constexpr (U == 3) {
        const uint32_t v = prmt(in.s0, in.s1, 0x5410u) >> ln.sh_shift & 0xFFFu;
        g = v | (v << 10);
    } else g = in.s0 | (in.s0 << 12);
    const uint32_t h0 = hfma2_bf16(and_xor(g, k.sm, k.sx), s, ns), h1 = hfma2_bf16(and_xor(g >> U, k.sm, k.sx), s, ns);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = hfma2_bf16(hfma2_bf16(and_xor(f[j], k.um, k.ux), k.one, k.uoff), su, j < 2 ? h0 : h1);
}

// The same from shared memory: ub, sb, eb are the addresses of this lane's codes and of the row's scale, OFF* constant
// distances from there.
template <int U, int OFFU, int OFFS, int OFFE>
__device__ __forceinline__ void gr_decode_row(uint32_t ub, uint32_t sb, uint32_t eb, const GrLane& ln, const GrConst<U>& k,
                                              uint32_t (&w)[4]) {
    GrRaw r;
    r.e = lds_s8<OFFE>(eb);
    r.w0 = lds32<OFFU>(ub);
    r.w1 = U == 4 ? 0u : lds32<OFFU + 4>(ub);
    r.s1 = 0u;
    if constexpr (U == 2) asm volatile("ld.shared.u8 %0, [%1+%2];" : "=r"(r.s0) : "r"(sb), "n"(OFFS));
    else r.s0 = lds_u16<OFFS>(sb);
    if constexpr (U == 3) r.s1 = lds_u16<OFFS>(sb - ln.sh_off + ln.sh_off2);
    gr_decode<U>(r, ln, k, w);
}

// u = 4 up to eight rows: an Inf becomes NaN, and with it the whole output row, as in the integer kernels that share these
// row counts (their fixed point cannot hold it), so that the result does not depend on the kernel a size falls to.  Four more
// instructions per 32-block and eight rows.
template <int U, int MT>
__device__ __forceinline__ uint4 gr_finite_or_nan(uint4 x) {
    if constexpr (U == 4 && MT == 1) {
        x.x = hfma2_bf16(x.x, 0u, x.x);
        x.y = hfma2_bf16(x.y, 0u, x.y);
        x.z = hfma2_bf16(x.z, 0u, x.z);
        x.w = hfma2_bf16(x.w, 0u, x.w);
    }
    return x;
}

// K block J of a stage: its activation fragments and the weights of the warp's groups, in the order that leaves fewer registers
// in use.  Every group is computed: columns beyond the matrix (a ragged last tile) come out as garbage that is not stored.
template <int U, int MT, int J, int N>
__device__ __forceinline__ void gr_activation(uint32_t xb, uint32_t (&b)[4]) {
    const uint4 x = gr_finite_or_nan<U, MT>(lds128<N * 8 * GR_XROW + J * 64>(xb));
    b[0] = prmt(x.x, x.z, 0x5410u);
    b[1] = prmt(x.x, x.z, 0x7632u);
    b[2] = prmt(x.y, x.w, 0x5410u);
    b[3] = prmt(x.y, x.w, 0x7632u);
}
template <int U, int MT, int J, int N>
__device__ __forceinline__ void gr_activations(uint32_t xb, uint32_t (&b)[MT][4]) {
    if constexpr (N < MT) {
        gr_activation<U, MT, J, N>(xb, b[N]);
        gr_activations<U, MT, J, N + 1>(xb, b);
    }
}
template <int U, int MT, int J, int Q>
__device__ __forceinline__ void gr_weights(uint32_t ub, uint32_t sb, uint32_t eb, const GrLane& ln, const GrConst<U>& k,
                                           uint32_t (&w0)[4], uint32_t (&w1)[4]) {
    constexpr int SUBJ = J * gr_sub_bytes(U, MT), UB = gr_ub(U), SB = gr_sb(U);
    constexpr int OU = SUBJ + Q * GM_GROUP * UB, OS = SUBJ + Q * GM_GROUP * SB, OE = SUBJ + Q * GM_GROUP;
    gr_decode_row<U, OU, OS, OE>(ub, sb, eb, ln, k, w0);
    gr_decode_row<U, OU + 8 * UB, OS + 8 * SB, OE + 8>(ub, sb, eb, ln, k, w1);
}
// The products of one group with N n-tiles: the first sixteen elements of the block against all of them, then the second, so
// that no MMA waits for the one before it.  A single n-tile has two accumulators for that (added up at the end).
__host__ __device__ constexpr int gr_accs(int mt) { return mt == 1 ? 2 : mt; }
template <int N, int NACC>
__device__ __forceinline__ void gr_mma(float (*acc)[4], const uint32_t (&w0)[4], const uint32_t (&w1)[4], const uint32_t (&b)[N][4]) {
#pragma unroll
    for (int n = 0; n < N; ++n) mma_bf16_16816(acc[n], w0[0], w1[0], w0[1], w1[1], b[n][0], b[n][1]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_bf16_16816(acc[NACC > N ? n + 1 : n], w0[2], w1[2], w0[3], w1[3], b[n][2], b[n][3]);
}
template <int U, int MT, int J, int Q>
__device__ __forceinline__ void gr_groups(uint32_t ub, uint32_t sb, uint32_t eb, const GrLane& ln, const GrConst<U>& k,
                                          const uint32_t (&b)[MT][4], float (&acc)[gr_groups_of(MT)][gr_accs(MT)][4]) {
    if constexpr (Q < gr_groups_of(MT)) {
        uint32_t w0[4], w1[4];
        gr_weights<U, MT, J, Q>(ub, sb, eb, ln, k, w0, w1);
        gr_mma<MT, gr_accs(MT)>(acc[Q], w0, w1, b);
        gr_groups<U, MT, J, Q + 1>(ub, sb, eb, ln, k, b, acc);
    }
}
template <int U, int MT, int J, int N>
__device__ __forceinline__ void gr_rows(uint32_t xb, const uint32_t (&w0)[4], const uint32_t (&w1)[4], float (&acc)[MT][4]) {
    if constexpr (N < MT) {                                                   // four n-tiles at a time
        uint32_t b[4][4];
        gr_activation<U, MT, J, N>(xb, b[0]);
        gr_activation<U, MT, J, N + 1>(xb, b[1]);
        gr_activation<U, MT, J, N + 2>(xb, b[2]);
        gr_activation<U, MT, J, N + 3>(xb, b[3]);
        gr_mma<4, 4>(&acc[N], w0, w1, b);
        gr_rows<U, MT, J, N + 4>(xb, w0, w1, acc);
    }
}
template <int U, int MT, int J>
__device__ __forceinline__ void gr_blocks(int nblk, uint32_t ub, uint32_t sb, uint32_t eb, uint32_t xb, const GrLane& ln,
                                          const GrConst<U>& k, float (&acc)[gr_groups_of(MT)][gr_accs(MT)][4]) {
    if constexpr (J < GR_KB) {
        if (J < nblk) {
            if constexpr (gr_groups_of(MT) > 1) {
                uint32_t b[MT][4];
                gr_activations<U, MT, J, 0>(xb, b);
                gr_groups<U, MT, J, 0>(ub, sb, eb, ln, k, b, acc);
            } else {
                uint32_t w0[4], w1[4];
                gr_weights<U, MT, J, 0>(ub, sb, eb, ln, k, w0, w1);
                gr_rows<U, MT, J, 0>(xb, w0, w1, acc[0]);
            }
        }
        gr_blocks<U, MT, J + 1>(nblk, ub, sb, eb, xb, ln, k, acc);
    }
}

struct GemvRegArgs {
    const int8_t* scale_exp;
    const uint8_t* upper_cm;
    const uint8_t* shared_cm;
    const __nv_bfloat16* X;      // row m0 of [M][K], 16-byte aligned
    float* partial;              // [max_slots][rows][OUT]
    unsigned long long* tile_counters;
    int* sticky;
    __nv_bfloat16* y;
    float* y_f32;                // optional
    const __nv_bfloat16* res;    // optional (up to eight rows): y = bf16(res + bf16(W x)); may be y itself
    int m0, rows, OUT, NB;
    GemvSchedule sch;            // sch.nb counts units of GR_KB K blocks
    uint32_t max_polls;
    int skip_stage;
    int combine;                 // split tiles are added up by gemv_umma_combine_kernel instead of the last warp to arrive
};

int gemv_reg_launch(const GemvRegArgs& a, int u, int mt, cudaStream_t st);      // gemv_reg.cu

template <int U, int MT>
__global__ void __launch_bounds__(GR_THREADS, 1)
gemv_reg_kernel(const GemvRegArgs a) {
    extern __shared__ __align__(128) uint8_t gr_smem[];
    __shared__ __align__(8) uint64_t bar_full_all[GR_TEAMS * GM_MAX_STAGES];
    __shared__ __align__(8) uint64_t bar_empty_all[GR_TEAMS * GM_MAX_STAGES];
    __shared__ unsigned int marker_sh[GM_WARPS];
    __shared__ __align__(16) uint32_t consts[GrConst<U>::N];

    constexpr int UB = gr_ub(U), SB = gr_sb(U), GR_GROUPS = gr_groups_of(MT), GR_TC = gr_tc(MT);
    constexpr int OFF_SH = GR_TC * UB, OFF_SC = GR_TC * (UB + SB), SUB = gr_sub_bytes(U, MT), OFF_X = GR_KB * SUB;
    constexpr int STAGE = gr_stage_bytes(U, MT);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GemvSchedule sch = a.sch;
    const long long n_lo = sch.lo(blockIdx.x), n_hi = sch.lo(blockIdx.x + 1);
    const int n_iter = (int)(n_hi - n_lo);
    int c = (int)(n_lo / sch.nb), blk = (int)(n_lo % sch.nb);        // tile, unit within the tile
    const int team = warp < GR_TEAMS * GM_WARPS ? warp / GM_WARPS : warp - GR_TEAMS * GM_WARPS;
    // each team has a ring of its own
    const uint32_t smem0 = smem_u32(gr_smem) + team * sch.stages * STAGE;
    uint64_t* const bar_full = bar_full_all + team * sch.stages;
    uint64_t* const bar_empty = bar_empty_all + team * sch.stages;

    if (tid == 32) GrConst<U>::store(consts);
    if (tid == 0) {
        for (int s = 0; s < GR_TEAMS * sch.stages; ++s) {
            mbar_init(smem_u32(&bar_full_all[s]), 1 + 32);       // the bulk copies' transaction, and the lanes' own copies
            mbar_init(smem_u32(&bar_empty_all[s]), GM_WARPS);
        }
        mbar_init_fence();
    }
    __syncthreads();
    chain_wait();

    if (warp >= GR_TEAMS * GM_WARPS) {
        // ------------------------------ producer warp: lanes share out a stage's copies ------------------------------
        const bool inject = a.skip_stage >= 0 && blockIdx.x == 0;
        const int64_t K = (int64_t)a.NB * BLOCK;
        // Lane 3j + p issues the copy of plane p of K block j, all in the same instruction: one lane after another needs
        // some hundred cycles for each.
        const int sub_blk = lane / 3, plane = lane - 3 * sub_blk;
        const uint8_t* const src_plane = plane == 0 ? a.upper_cm : plane == 1 ? a.shared_cm : reinterpret_cast<const uint8_t*>(a.scale_exp);
        const int per_col = plane == 0 ? UB : plane == 1 ? SB : 1;
        const uint32_t dst_off = sub_blk * SUB + (plane == 0 ? 0 : plane == 1 ? OFF_SH : OFF_SC);
        int s = 0, issued = 0;
        uint32_t ph = 1;                           // passes at once on a fresh barrier
        blk += team;
        for (int it = team; it < n_iter; it += GR_TEAMS) {
            while (blk >= sch.nb) { blk -= sch.nb; ++c; }
            bool stop = inject && it == a.skip_stage;
            if (!stop && !mbar_wait_bounded(smem_u32(&bar_empty[s]), ph, a.max_polls)) {
                report_wait_failure(a.sticky, WAIT_FAIL_GEMV_MMA);
                stop = true;
            }
            if (__any_sync(0xffffffffu, stop)) break;
            const int o0 = c * GR_TC, cv = min(GR_TC, a.OUT - o0);
            const int b0 = blk * GR_KB, nblk = min(GR_KB, a.NB - b0);
            const uint32_t bar = smem_u32(&bar_full[s]), base = smem0 + s * STAGE;
            if (lane == 0) mbar_expect_tx(bar, (uint32_t)(nblk * cv * (UB + SB + 1)));
            __syncwarp();
            if (lane < 3 * nblk) {
                const int64_t col = (int64_t)(b0 + sub_blk) * a.OUT + o0;
                bulk_g2s(base + dst_off, src_plane + col * per_col, (uint32_t)(cv * per_col), bar);
            }
            // the activations go lane by lane: a bulk copy per row would make the copy engine's rate (about a hundred
            // cycles a copy) the limit
            for (int i = lane; i < a.rows * (GR_KB * 4); i += 32) {
                const int m = i / (GR_KB * 4), ch = i % (GR_KB * 4);
                if (ch < nblk * 4) cp_async16(base + OFF_X + m * GR_XROW + ch * 16, a.X + m * K + b0 * BLOCK + ch * 8);
            }
            cp_async_arrive(bar);
            ++issued;
            blk += GR_TEAMS;
            if (++s == sch.stages) { s = 0; ph ^= 1u; }
        }
        // leave only when every copy has landed (see gemv_u4gs2_mma_kernel)
        for (int i = max(0, issued - sch.stages); i < issued; ++i)
            mbar_wait_bounded(smem_u32(&bar_full[i % sch.stages]), (uint32_t)(i / sch.stages) & 1u, a.max_polls);
        return;
    }

    // -------------------------------- consumers --------------------------------
    const int cw = warp % GM_WARPS;
    const int g = lane >> 2, t = lane & 3, r0 = cw * 16 + g;                 // columns r0 and r0 + 8 of each group
    const GrLane ln = gr_lane<U>(t);
    const GrConst<U> kc(smem_u32(consts));
    const uint32_t aU = smem0 + r0 * UB + ln.up_off, aS = smem0 + OFF_SH + r0 * SB + ln.sh_off, aE = smem0 + OFF_SC + r0;
    const uint32_t aX = smem0 + OFF_X + g * GR_XROW + t * 16;
    float acc[GR_GROUPS][gr_accs(MT)][4];
#pragma unroll
    for (int q = 0; q < GR_GROUPS; ++q)
#pragma unroll
        for (int n = 0; n < gr_accs(MT); ++n) acc[q][n][0] = acc[q][n][1] = acc[q][n][2] = acc[q][n][3] = 0.0f;
    bool aborted = false;
    int s = 0, seg = 0, next = team;                                         // ring stage and index of this team's next unit
    uint32_t ph = 0;
    for (int left = n_iter; left > 0; ++c, blk = 0) {                        // one tile after another
        // the (tile, warp) counter's marker, fetched long before the hand-off needs it
        if (!a.combine && team == 0 && lane == 0)
            marker_sh[cw] = *reinterpret_cast<volatile unsigned int*>(a.tile_counters + c * GM_WARPS + cw);
        const int cv = min(GR_TC, a.OUT - c * GR_TC);
        const int nq = (cv - cw * 16 + GM_GROUP - 1) / GM_GROUP;              // groups in which this warp has columns
        const int units = min(left, sch.nb - blk);
        left -= units;
        const int base = seg - blk;                                           // unit index of the tile's first unit
        seg += units;
        for (; next < seg; next += GR_TEAMS) {
            const int kleft = a.NB - (next - base) * GR_KB;                   // K blocks from here to the tile's end
            if (!aborted) aborted = !mbar_wait_bounded(smem_u32(&bar_full[s]), ph, a.max_polls);
            if (__any_sync(0xffffffffu, aborted)) {                           // one decision per warp: the MMAs are warp-wide
                if (aborted) report_wait_failure(a.sticky, WAIT_FAIL_GEMV_MMA);
                aborted = true;
            } else {
                const uint32_t so = s * STAGE;
                gr_blocks<U, MT, 0>(kleft, aU + so, aS + so, aE + so, aX + so, ln, kc, acc);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bar_empty[s]));
            if (++s == sch.stages) { s = 0; ph ^= 1u; }
        }
        if constexpr (MT == 1) {
#pragma unroll
            for (int q = 0; q < GR_GROUPS; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    acc[q][0][i] += acc[q][1][i];
                    acc[q][1][i] = 0.0f;
                }
        }
        {
            // the teams' sums come together: warp cw of each of the others hands its accumulators to warp cw of the first
            float4* mb = reinterpret_cast<float4*>(gr_smem + GR_TEAMS * sch.stages * STAGE) + cw * (GR_GROUPS * MT) * 32 + lane;
            constexpr int TEAM_F4 = GM_WARPS * GR_GROUPS * MT * 32;
            if (team) {
#pragma unroll
                for (int q = 0; q < GR_GROUPS; ++q)
#pragma unroll
                    for (int n = 0; n < MT; ++n) {
                        const float bad = aborted ? __int_as_float(0x7FC00000) : 0.0f;
                        mb[(team - 1) * TEAM_F4 + (q * MT + n) * 32] =
                            make_float4(acc[q][n][0] + bad, acc[q][n][1] + bad, acc[q][n][2] + bad, acc[q][n][3] + bad);
                        acc[q][n][0] = acc[q][n][1] = acc[q][n][2] = acc[q][n][3] = 0.0f;
                    }
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + cw), "n"(GR_TEAMS * 32) : "memory");
            if (!team) {
#pragma unroll
                for (int q = 0; q < GR_GROUPS; ++q)
#pragma unroll
                    for (int n = 0; n < MT; ++n)
#pragma unroll
                        for (int o = 0; o < GR_TEAMS - 1; ++o) {
                            const float4 v = mb[o * TEAM_F4 + (q * MT + n) * 32];
                            acc[q][n][0] += v.x; acc[q][n][1] += v.y; acc[q][n][2] += v.z; acc[q][n][3] += v.w;
                        }
            }
            if (left > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + cw), "n"(GR_TEAMS * 32) : "memory");    // the buffer is used again
            if (team) continue;
        }
        // ---- end of this thread block's run over tile c: the outputs, or a partial and perhaps the tile's sum ----
        {
            const int first = sch.first_cta(c), nslots = sch.last_cta(c) - first + 1;
            const int slot = blockIdx.x - first, o0 = c * GR_TC;
            const float nan = __int_as_float(0x7FC00000);
#pragma unroll
            for (int q = 0; q < GR_GROUPS; ++q) {
                if (q < nq) {
#pragma unroll
                    for (int n = 0; n < MT; ++n) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int m = n * 8 + 2 * t + (i & 1);
                            const float v = aborted ? nan : acc[q][n][i];
                            if (m < a.rows) {
                                const int o = o0 + q * GM_GROUP + r0 + (i >> 1) * 8;
                                if (nslots == 1) {
                                    const int64_t yo = (int64_t)(a.m0 + m) * a.OUT + o;
                                    __nv_bfloat16 y = __float2bfloat16_rn(v);
                                    if (MT == 1 && a.res) y = __float2bfloat16_rn(__bfloat162float(a.res[yo]) + __bfloat162float(y));
                                    a.y[yo] = y;
                                    if (a.y_f32) a.y_f32[yo] = v;
                                } else {
                                    a.partial[((int64_t)slot * a.rows + m) * a.OUT + o] = v;
                                }
                            }
                            acc[q][n][i] = 0.0f;
                        }
                    }
                }
            }
            if (nq > 0 && nslots > 1 && !a.combine) {
                __syncwarp();
                GemvMmaArgs h{};                                              // the hand-off's part of the arguments
                h.sticky = a.sticky; h.max_polls = a.max_polls;
                unsigned int arrived = 0;
                if (lane == 0) arrived = gemv_count_arrival(h, a.tile_counters + c * GM_WARPS + cw, marker_sh[cw]);
                arrived = __shfl_sync(0xffffffffu, arrived, 0);
                if (arrived == (unsigned int)nslots) {
                    __threadfence();
                    // four adjacent outputs per item, S lanes to an item where there are few (see gemv_mma.cuh): the order
                    // of the additions depends on the shape alone
                    const int64_t sstride4 = (int64_t)a.rows * a.OUT / 4;
                    const int items = a.rows * nq * 4;
                    int S = 1;
                    while (S < 8 && items * S * 2 <= 32) S *= 2;
                    const int per = 32 / S;
                    for (int base = 0; base < items; base += per) {
                        const int item = base + lane / S, part = lane % S;
                        const bool live = item < items;
                        const int m = live ? item / (nq * 4) : 0, rem = live ? item % (nq * 4) : 0;
                        const int64_t e = (int64_t)m * a.OUT + o0 + (rem >> 2) * GM_GROUP + cw * 16 + (rem & 3) * 4;
                        const float4* src = reinterpret_cast<const float4*>(a.partial + e);
                        float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (live) {
                            for (int k0 = part; k0 < nslots; k0 += 8 * S) {
                                float4 v[8];
#pragma unroll
                                for (int k = 0; k < 8; ++k)
                                    v[k] = (k0 + k * S < nslots) ? __ldcg(src + (k0 + k * S) * sstride4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                                for (int k = 0; k < 8; ++k) { sum.x += v[k].x; sum.y += v[k].y; sum.z += v[k].z; sum.w += v[k].w; }
                            }
                        }
                        for (int o = S >> 1; o; o >>= 1) {
                            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
                            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
                            sum.z += __shfl_xor_sync(0xffffffffu, sum.z, o);
                            sum.w += __shfl_xor_sync(0xffffffffu, sum.w, o);
                        }
                        if (live && part == 0) {
                            const int64_t y0 = (int64_t)a.m0 * a.OUT + e;
                            if (a.y_f32) *reinterpret_cast<float4*>(a.y_f32 + y0) = sum;
                            if (MT == 1 && a.res) {        // the projection rounds to bf16 first, as the unfused add sees it
                                const uint2 rb = *reinterpret_cast<const uint2*>(a.res + y0);
                                sum.x = bf16_lo(rb.x) + __bfloat162float(__float2bfloat16_rn(sum.x));
                                sum.y = bf16_hi(rb.x) + __bfloat162float(__float2bfloat16_rn(sum.y));
                                sum.z = bf16_lo(rb.y) + __bfloat162float(__float2bfloat16_rn(sum.z));
                                sum.w = bf16_hi(rb.y) + __bfloat162float(__float2bfloat16_rn(sum.w));
                            }
                            const __nv_bfloat162 lo = __floats2bfloat162_rn(sum.x, sum.y), hi = __floats2bfloat162_rn(sum.z, sum.w);
                            *reinterpret_cast<uint2*>(a.y + y0) =
                                make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                        }
                    }
                    if (lane == 0) reinterpret_cast<unsigned int*>(a.tile_counters + c * GM_WARPS + cw)[1] = 0u;
                }
            }
        }
    }
}

}  // namespace msaq
