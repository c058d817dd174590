// The weight packer at gs = 2, the group size of the tuned GEMVs: W [OUT][K] to all five planes.
//
// Bound by HBM: two (or four) bytes of weight in, 49/32 bytes of planes out.  A thread block takes 128 rows of four K
// blocks; four lanes share a 32-block (quant8.cuh), so a warp reads 64-byte runs and writes the column-major planes as
// they come; the bytes of the row-major planes go through shared memory and leave as 128-byte rows.  One thread per
// 32-block with byte stores (kv_pack.cu, still the packer of the other group sizes) reads 64 bytes per lane a row apart
// and scatters single bytes: 14336 x 4096 bf16 to u = 4, 485 -> 72 us.
// Behaviour: ms_lib/pack.py:101-137 of the reference (`pack_weight`).
#include "quant8.cuh"
#include "sm100_ptx.cuh"

namespace msaq {
namespace {

constexpr int WP_ROWS = 128, WP_BLKS = 4, WP_THREADS = 256;
constexpr int WP_STRIDE = WP_ROWS + 4;               // bytes per staged plane row: the four lanes of a block hit different banks

template <int U, bool BF16>
__global__ void __launch_bounds__(WP_THREADS)
weight_pack_kernel(const void* __restrict__ W, int8_t* __restrict__ scale_exp, uint8_t* __restrict__ upper,
                   uint8_t* __restrict__ shared, uint8_t* __restrict__ upper_cm, uint8_t* __restrict__ shared_cm, int64_t OUT,
                   int nb) {
    chain_release();
    chain_wait();
    constexpr int WB = 8 - U, UB = 4 * WB, SB = 2 * U, PLANE_ROWS = UB + SB + 1;
    __shared__ __align__(16) uint8_t stage[WP_BLKS][PLANE_ROWS][WP_STRIDE];
    const int tid = threadIdx.x, lane = tid & 31, p = tid & 3, r = tid >> 2;
    const int64_t o0 = (int64_t)blockIdx.x * WP_ROWS;
    const int b0 = blockIdx.y * WP_BLKS, nblk = min(WP_BLKS, nb - b0);
    const int64_t K = (int64_t)nb * BLOCK;

#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        const int oo = half * 64 + r;
        const int64_t o = o0 + oo;
        const bool in = o < OUT;
        const int64_t at = o * K + (int64_t)b0 * BLOCK + p * 8;
        uint4 raw[WP_BLKS][BF16 ? 1 : 2];
#pragma unroll
        for (int j = 0; j < WP_BLKS; ++j)
#pragma unroll
            for (int i = 0; i < (BF16 ? 1 : 2); ++i) {
                raw[j][i] = make_uint4(0u, 0u, 0u, 0u);
                if (in && j < nblk) raw[j][i] = __ldcs(static_cast<const uint4*>(W) + (at + j * BLOCK) / (BF16 ? 8 : 4) + i);
            }
#pragma unroll
        for (int j = 0; j < WP_BLKS; ++j) {
            if (j >= nblk) break;                                            // uniform over the thread block
            float v[8];
            if constexpr (BF16) {
                const uint32_t w[4] = {raw[j][0].x, raw[j][0].y, raw[j][0].z, raw[j][0].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { v[2 * i] = bf16_lo(w[i]); v[2 * i + 1] = bf16_hi(w[i]); }
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    v[4 * i] = __uint_as_float(raw[j][i].x); v[4 * i + 1] = __uint_as_float(raw[j][i].y);
                    v[4 * i + 2] = __uint_as_float(raw[j][i].z); v[4 * i + 3] = __uint_as_float(raw[j][i].w);
                }
            }
            const Codes8 c = quant8<U>(v);
            const int64_t slot = (int64_t)(b0 + j) * OUT + o;
            if (upper_cm) quant8_store<U>(c, lane, in, upper_cm + slot * UB, shared_cm + slot * SB);
#pragma unroll
            for (int k = 0; k < WB; ++k) stage[j][p * WB + k][oo] = (uint8_t)(c.up >> (8 * k));
            if constexpr (U == 4) {
                stage[j][UB + 2 * p][oo] = (uint8_t)c.sh;
                stage[j][UB + 2 * p + 1][oo] = (uint8_t)(c.sh >> 8);
            } else if constexpr (U == 3) {
                const uint32_t nsh = __shfl_down_sync(0xffffffffu, c.sh, 1);
                const uint32_t h = (c.sh >> (4 * p)) | (nsh << (12 - 4 * p));
                if (p < 3) {
                    stage[j][UB + 2 * p][oo] = (uint8_t)h;
                    stage[j][UB + 2 * p + 1][oo] = (uint8_t)(h >> 8);
                }
            } else {
                stage[j][UB + p][oo] = (uint8_t)c.sh;
            }
            if (p == 0) stage[j][UB + SB][oo] = (uint8_t)(int8_t)c.e;
        }
    }
    __syncthreads();
    const int cols = (int)min((int64_t)WP_ROWS, OUT - o0);
    for (int row = tid >> 5; row < nblk * PLANE_ROWS; row += WP_THREADS / 32) {
        const int j = row / PLANE_ROWS, i = row % PLANE_ROWS;
        const int64_t blk = b0 + j;
        uint8_t* dst = i < UB ? (upper ? upper + (blk * UB + i) * OUT : nullptr)
                     : i < UB + SB ? (shared ? shared + (blk * SB + i - UB) * OUT : nullptr)
                                   : (scale_exp ? reinterpret_cast<uint8_t*>(scale_exp) + blk * OUT : nullptr);
        if (!dst) continue;
        dst += o0;
        if (!(reinterpret_cast<uintptr_t>(dst) & 3) && cols == WP_ROWS) {
            reinterpret_cast<uint32_t*>(dst)[lane] = *reinterpret_cast<const uint32_t*>(&stage[j][i][4 * lane]);
        } else {
            for (int k = lane; k < cols; k += 32) dst[k] = stage[j][i][k];
        }
    }
}

}  // namespace

// Whether the kernel serves these planes: 16-byte reads of W, word stores of upper_cm, half-word stores of shared_cm.
bool weight_pack_usable(const void* W, const void* upper_cm, const void* shared_cm, int64_t OUT, int64_t nb, int gs) {
    return gs == 2 && !(reinterpret_cast<uintptr_t>(W) & 15) && !(reinterpret_cast<uintptr_t>(upper_cm) & 3) &&
           !(reinterpret_cast<uintptr_t>(shared_cm) & 1) && !upper_cm == !shared_cm &&
           (nb + WP_BLKS - 1) / WP_BLKS <= 65535 && nb <= INT32_MAX / BLOCK && (OUT + WP_ROWS - 1) / WP_ROWS <= INT32_MAX;
}

int weight_pack_gs2(const void* W, int w_is_bf16, int8_t* scale_exp, uint8_t* upper, uint8_t* shared, uint8_t* upper_cm,
                    uint8_t* shared_cm, int64_t OUT, int64_t nb, int u, cudaStream_t st) {
    const dim3 grid((unsigned)((OUT + WP_ROWS - 1) / WP_ROWS), (unsigned)((nb + WP_BLKS - 1) / WP_BLKS)), block(WP_THREADS);
#define MSAQ_GO(U, B) launch_chained(weight_pack_kernel<U, B>, grid, block, 0, st, W, scale_exp, upper, shared, upper_cm, shared_cm, \
                                     OUT, (int)nb)
    if (w_is_bf16) { if (u == 4) MSAQ_GO(4, true); else if (u == 3) MSAQ_GO(3, true); else MSAQ_GO(2, true); }
    else { if (u == 4) MSAQ_GO(4, false); else if (u == 3) MSAQ_GO(3, false); else MSAQ_GO(2, false); }
#undef MSAQ_GO
    count_launch();
    return check_launch("weight_pack");
}

}  // namespace msaq
