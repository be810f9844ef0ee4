// Plain FP64 table contraction: R_g = G_g Y_g^T for every multipole group g,
// where row i of G_g is w*rho of the group's i-th pair and row j of Y_g is
// Y^k of its j-th pair (the slater_rk_poisson sum of atomx
// numerics/bspline/slater.py:130 evaluated for a whole table at once).
//
// The table is symmetric in (ac)<->(bd): the caller lists 128x128 tiles with
// tile_j >= tile_i, and a block takes one 64x64 quarter of a listed tile
// (rkb_dgemm.cuh; FP64 tensor pipe, sm_100a has no FP64 tcgen05 kind).  Quarters
// below the diagonal of a diagonal tile are not computed.  Every entry above the
// diagonal is stored twice, as computed and transposed, so the tables are symmetric
// to the bit and do not depend on the tile size.
#include "rkb_dgemm.cuh"

namespace rkb {
namespace fp64tab {

constexpr int TILE = 128;  // the task list's tiles

template <class T>
__global__ void __launch_bounds__(dgemm::THREADS, 3)
contract_kernel(const double *__restrict__ G, const double *__restrict__ Y, long ld, long kdim,
                const long *__restrict__ grp_kdim, const long *__restrict__ grp_row0, const long *__restrict__ grp_n,
                const long *__restrict__ grp_out, const int *__restrict__ tasks, double *__restrict__ out) {
    extern __shared__ __align__(16) double smem[];
    constexpr int SUB = TILE / T::SIDE;  // sub-tiles per side
    const long t = blockIdx.x / (SUB * SUB);
    const int sub = (int)(blockIdx.x % (SUB * SUB)), si = sub / SUB, sj = sub % SUB;
    const int g = tasks[3 * t], ti = tasks[3 * t + 1], tj = tasks[3 * t + 2];
    if (ti == tj && si > sj) return;
    const long n = grp_n[g];
    const long i0 = (long)ti * TILE + si * T::SIDE, j0 = (long)tj * TILE + sj * T::SIDE;
    if (i0 >= n || j0 >= n) return;
    const long row0 = grp_row0[g];
    const double *o = T::run(G + row0 * ld, ld, i0, n, Y + row0 * ld, ld, j0, n,
                             (int)((grp_kdim ? grp_kdim[g] : kdim) / dgemm::BK), smem);
    constexpr int WS = T::SIDE / 2, RPW = 32 / WS;  // rows a warp stores at a time
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane / WS, lc = lane % WS;
    const long i1 = i0 + warp / 2 * WS, j1 = j0 + warp % 2 * WS;
    double *R = out + grp_out[g];
    if (j1 + lc < n)
#pragma unroll 8
        for (int r = lr; r < WS; r += RPW)
            if (i1 + r < n && i1 + r <= j1 + lc) R[(i1 + r) * n + j1 + lc] = o[r * T::OLD + lc];
    if (i1 + lc < n)
#pragma unroll 8
        for (int c = lr; c < WS; c += RPW)
            if (j1 + c < n && i1 + lc < j1 + c) R[(j1 + c) * n + i1 + lc] = o[lc * T::OLD + c];
}

}  // namespace fp64tab
}  // namespace rkb

using namespace rkb;

static int launch_contract(const double *d_g, const double *d_y, long ld, long kdim, const long *d_grp_kdim,
                           const long *d_grp_row0, const long *d_grp_n, const long *d_grp_out, const int *d_tasks,
                           long n_tasks, double *d_out, void *stream) {
    if (n_tasks == 0) return RKB_OK;
    RKB_CHECK_ARG(n_tasks < (1L << 27), "too many tiles (%ld)", n_tasks);
    auto launch = [&](auto tile) {
        using T = decltype(tile);
        constexpr long SUB = fp64tab::TILE / T::SIDE;
        RKB_CUDA(set_smem(fp64tab::contract_kernel<T>, (int)T::SMEM));
        fp64tab::contract_kernel<T><<<(unsigned)(SUB * SUB * n_tasks), dgemm::THREADS, T::SMEM, as_stream(stream)>>>(
            d_g, d_y, ld, kdim, d_grp_kdim, d_grp_row0, d_grp_n, d_grp_out, d_tasks, d_out);
        return (int)RKB_OK;
    };
    const int st = dgemm::small_problem(4 * n_tasks) ? launch(dgemm::Tile32()) : launch(dgemm::Tile64());
    if (st) return st;
    RKB_LAUNCHED("fp64tab::contract_kernel");
    return RKB_OK;
}

extern "C" int rkb_table_contract_fp64(const double *d_g, const double *d_y, long ld, long kdim,
                                       const long *d_grp_row0, const long *d_grp_n, const long *d_grp_out,
                                       const int *d_tasks, long n_tasks, double *d_out, void *stream) {
    RKB_CHECK_ARG(kdim >= 0 && kdim % dgemm::BK == 0 && ld >= kdim && ld % 2 == 0,
                  "contraction length %ld must be a multiple of %d and <= ld (%ld, even)", kdim, dgemm::BK, ld);
    return launch_contract(d_g, d_y, ld, kdim, nullptr, d_grp_row0, d_grp_n, d_grp_out, d_tasks, n_tasks, d_out,
                           stream);
}

extern "C" int rkb_table_contract_fp64_groups(const double *d_g, const double *d_y, long ld, long max_kdim,
                                              const long *d_grp_kdim, const long *d_grp_row0, const long *d_grp_n,
                                              const long *d_grp_out, const int *d_tasks, long n_tasks,
                                              double *d_out, void *stream) {
    RKB_CHECK_ARG(d_grp_kdim != nullptr, "per-group contraction lengths are required");
    RKB_CHECK_ARG(max_kdim >= 0 && ld >= max_kdim && ld % 2 == 0, "contraction lengths must be <= ld (%ld, even)",
                  ld);
    return launch_contract(d_g, d_y, ld, max_kdim, d_grp_kdim, d_grp_row0, d_grp_n, d_grp_out, d_tasks, n_tasks,
                           d_out, stream);
}
