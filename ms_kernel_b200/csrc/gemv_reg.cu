// Launches of the register-operand GEMV (gemv_reg.cuh); the plan and the choice of kernel are gemv.cu's.
#include "gemv_reg.cuh"

namespace msaq {
namespace {

template <int U, int MT>
int launch_reg(const GemvRegArgs& a, cudaStream_t st) {
    static int configured[64] = {};                      // largest dynamic smem size set per device
    const int smem = GR_TEAMS * a.sch.stages * gr_stage_bytes(U, MT) + gr_merge_bytes(MT);
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && configured[dev] < smem) {
        if (cudaFuncSetAttribute(gemv_reg_kernel<U, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return fail(MSAQ_ERR_CUDA, "cannot reserve %d bytes of shared memory", smem);
        configured[dev] = smem;
    }
    launch_chained(gemv_reg_kernel<U, MT>, dim3(a.sch.grid), dim3(GR_THREADS), (size_t)smem, st, a);
    count_launch();
    return check_launch("gemv_reg");
}

template <int U>
int launch_reg_mt(const GemvRegArgs& a, int mt, cudaStream_t st) {
    return mt == 1 ? launch_reg<U, 1>(a, st) : mt == 2 ? launch_reg<U, 2>(a, st) : mt == 4 ? launch_reg<U, 4>(a, st) : launch_reg<U, 8>(a, st);
}

}  // namespace

int gemv_reg_launch(const GemvRegArgs& a, int u, int mt, cudaStream_t st) {
    return u == 4 ? launch_reg_mt<4>(a, mt, st) : u == 3 ? launch_reg_mt<3>(a, mt, st) : launch_reg_mt<2>(a, mt, st);
}

}  // namespace msaq
