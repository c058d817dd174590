// Launches of the GEMVs without partial sums in global memory (gemv_direct.cuh); gemv.cu chooses the kernel.
#include "gemv_direct.cuh"

namespace msaq {
namespace {

int launch_direct(void (*kernel)(GemvDirectArgs), int cg, const GemvDirectArgs& a, cudaStream_t st) {
    const unsigned tiles = (unsigned)((a.OUT + 16 * cg - 1) / (16 * cg));
    launch_chained_cluster(kernel, dim3(tiles * a.cs), dim3(GD_THREADS), 0, (unsigned)a.cs, st, a);
    count_launch();
    return check_launch("gemv_direct");
}

template <int MODE>
int launch_int(const GemvDirectArgs& a, int cg, cudaStream_t st) {
    switch (a.rows) {
        case 1: return launch_direct(cg == 1 ? gemv_direct_int_kernel<MODE, 1, 1> : gemv_direct_int_kernel<MODE, 4, 1>, cg, a, st);
        case 2: return launch_direct(cg == 2 ? gemv_direct_int_kernel<MODE, 2, 2> : gemv_direct_int_kernel<MODE, 4, 2>, cg, a, st);
        default: return launch_direct(cg == 2 ? gemv_direct_int_kernel<MODE, 2, 4> : gemv_direct_int_kernel<MODE, 4, 4>, cg, a, st);
    }
}

template <int U, int MT>
int launch_bf16(const GemvDirectArgs& a, int cg, cudaStream_t st) {
    switch (cg) {
        case 2: return launch_direct(gemv_direct_bf16_kernel<U, MT, 2>, cg, a, st);
        case 3: return launch_direct(gemv_direct_bf16_kernel<U, MT, 3>, cg, a, st);
        default: return launch_direct(gemv_direct_bf16_kernel<U, MT, U == 4 ? 4 : 3>, cg, a, st);
    }
}

template <int U>
int launch_bf16_rows(const GemvDirectArgs& a, int cg, cudaStream_t st) {
    return a.rows <= 8 ? launch_bf16<U, 1>(a, cg, st) : launch_bf16<U, 2>(a, cg, st);
}

bool integer(int64_t M, int u) { return u == 4 && M <= 4; }

}  // namespace

// Cycles of one launch, as far as they depend on the choice, fitted to measurements from 512 x 512 to 4096 x 28672: an
// iteration of a thread block (a 32-block per warp) costs its instructions -- `stage` for the activations, `group` per 16
// columns, sixteen warps on four schedulers, `resident` thread blocks to an SM -- or a load's latency, and a cluster costs its
// barriers.  So wide thread blocks in clusters win where the activations are expensive and K is long (4096 x 14336, one row,
// us: one group 19.2, four groups and two thread blocks to a cluster 14.0), narrow ones without where it is short (2048 x
// 2048: 3.5 against 4.9).  Clusters that do not fit the GPCs wait for a second round (1216 x 18688,
// 19 clusters of seven: 14.6 us, 76 of three: 11.1 us; the occupancy query counts 148, 74, 45, 33, 26, 22, 15 and 15 clusters of one
// to eight thread blocks, one to an SM; GPCs differ by a few SMs from part to part, hence a little less here).
bool gemv_direct_pick(int64_t M, int64_t OUT, int64_t NB, int u, int* cg, int* cs, int64_t* cycles) {
    static const int int1[] = {1, 4, 0}, int4[] = {2, 4, 0}, bf4[] = {2, 3, 4, 0}, bf3[] = {2, 3, 0};
    const int* widths = integer(M, u) ? (M == 1 ? int1 : int4) : u == 4 ? bf4 : bf3;
    const int64_t stage = integer(M, u) ? 55 * M : 20, group = integer(M, u) ? 45 : (u == 4 ? 95 : u == 3 ? 115 : 105) + (M > 8 ? 15 : 0);
    static const int fit[GD_MAX_CLUSTER + 1] = {0, 148, 74, 44, 32, 24, 20, 14, 14};
    int64_t best = INT64_MAX;
    for (const int* w = widths; *w; ++w) {
        const int64_t per_sm = integer(M, u) ? gd_int_per_sm(*w) : 1, tiles = (OUT + 16 * *w - 1) / (16 * *w);
        for (int n = 1; n <= GD_MAX_CLUSTER; ++n) {
            if (tiles > (n == 1 ? sm_count() : fit[n]) * per_sm) break;
            if (n > 1 && NB < 2 * GD_WARPS * n) break;
            const int64_t resident = (tiles * n + sm_count() - 1) / sm_count(), iterations = (NB + GD_WARPS * n - 1) / (GD_WARPS * n);
            const int64_t issue = 4 * resident * (stage + *w * group) * 5 / 4;
            const int64_t cost = iterations * (issue > 700 ? issue : 700) + (n > 1 ? 1500 + 300 * n : 0);
            if (cost < best) {
                best = cost;
                *cg = *w;
                *cs = n;
            }
        }
    }
    *cycles = best;
    return best != INT64_MAX;
}

int gemv_direct_launch(const GemvDirectArgs& a, int u, int mode, int cg, cudaStream_t st) {
    if (integer(a.rows, u)) {
        switch (mode) {
            case XP_RMSNORM: return launch_int<XP_RMSNORM>(a, cg, st);
            case XP_SILU_MUL: return launch_int<XP_SILU_MUL>(a, cg, st);
            case XP_ADD_NORM: return launch_int<XP_ADD_NORM>(a, cg, st);
            default: return launch_int<XP_PLAIN>(a, cg, st);
        }
    }
    return u == 4 ? launch_bf16_rows<4>(a, cg, st) : u == 3 ? launch_bf16_rows<3>(a, cg, st) : launch_bf16_rows<2>(a, cg, st);
}

}  // namespace msaq
