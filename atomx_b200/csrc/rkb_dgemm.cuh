// FP64 GEMM tile C = A B^T on the DMMA pipe, shared by the table contraction and
// the cell engine's GEMMs.
//
// A block of four warps, 2 x 2 over the tile, each with a WS x WS accumulator tile
// (DMMA m8n8k4): 64 x 64 tiles with WS = 32, 32 x 32 with WS = 16.  Operands come
// through a 3-stage cp.async ring.  Every entry is summed in the same order, four
// columns at a time from the first, whatever the tile: tables do not depend on how
// many of them share a launch.
//
// Bound by the DMMA pipe (16 clocks an instruction and SM sub-partition).  128 x 128
// tiles with one block of eight warps per SM reached 81 % of cuBLAS DGEMM on large
// tables: both warps of a sub-partition stop at every stage barrier and the
// epilogue overlaps nothing.  Three small blocks per SM stop at different times,
// and the finer tiles leave fewer SMs idle on small problems.  Z=70 tables (N = 896,
// 1.6e8 unique entries): 9.91 -> 8.37 ms, 34.2 TF/s, 0.97 of cuBLAS; 222 x 2048 x 2048:
// 313 -> 95 us; 24 x 1080 x 1088: 162 -> 28 us (cuBLAS 89 and 27 us).
#pragma once

#include "rkb_common.cuh"
#include "rkb_dmma.cuh"

namespace rkb {
namespace dgemm {

constexpr int BK = 16, LDS = BK + 4, STAGES = 3, THREADS = 128;

template <int WS>
struct Tile {
    static constexpr int SIDE = 2 * WS;                            // rows and columns of the tile
    static constexpr int F = WS / 8;                               // 8 x 8 fragments per warp and side
    static constexpr int STAGE = 2 * SIDE * LDS;                   // doubles
    static constexpr int OLD = WS + 1, OUT = 4 * WS * OLD;         // the warps' output blocks
    static constexpr size_t SMEM = sizeof(double) * (STAGES * STAGE > OUT ? STAGES * STAGE : OUT);

    static __device__ __forceinline__ void load(double *s, const double *__restrict__ g, long ld, long row0, long nrows,
                                                long k0) {
#pragma unroll
        for (int it = 0; it < SIDE / 16; ++it) {
            const int c = threadIdx.x + it * THREADS;
            const int row = c >> 3, col = (c & 7) * 2;
            const bool ok = row0 + row < nrows;
            cp_async16(s + row * LDS + col, g + (ok ? row0 + row : row0) * ld + k0 + col, ok ? 16 : 0);
        }
    }

    // The tile at rows i0 of A (M rows) and j0 of B (N rows), nk steps of BK columns.
    // Returns this warp's WS x WS block (rows of OLD doubles in shared memory, visible to
    // the warp), at rows WS * (warp / 2) and columns WS * (warp % 2) of the tile.
    static __device__ __forceinline__ const double *run(const double *__restrict__ A, long lda, long i0, long M,
                                                        const double *__restrict__ B, long ldb, long j0, long N, int nk,
                                                        double *smem) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
        double acc[F][F][2];
#pragma unroll
        for (int a = 0; a < F; ++a)
#pragma unroll
            for (int b = 0; b < F; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) {
            if (s < nk) {
                load(smem + s * STAGE, A, lda, i0, M, (long)s * BK);
                load(smem + s * STAGE + SIDE * LDS, B, ldb, j0, N, (long)s * BK);
            }
            cp_async_commit();
        }
        int st = 0, pf = STAGES - 1;
        for (int kb = 0; kb < nk; ++kb) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            if (kb + STAGES - 1 < nk) {
                load(smem + pf * STAGE, A, lda, i0, M, (long)(kb + STAGES - 1) * BK);
                load(smem + pf * STAGE + SIDE * LDS, B, ldb, j0, N, (long)(kb + STAGES - 1) * BK);
            }
            cp_async_commit();
            const double *a_s = smem + st * STAGE + (warp / 2 * WS + fr) * LDS + fc;
            const double *b_s = smem + st * STAGE + (SIDE + warp % 2 * WS + fr) * LDS + fc;
#pragma unroll
            for (int k = 0; k < BK; k += 4) {
                double af[F], bf[F];
#pragma unroll
                for (int a = 0; a < F; ++a) af[a] = a_s[a * 8 * LDS + k];
#pragma unroll
                for (int b = 0; b < F; ++b) bf[b] = b_s[b * 8 * LDS + k];
#pragma unroll
                for (int a = 0; a < F; ++a)
#pragma unroll
                    for (int b = 0; b < F; ++b) dmma(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
            }
            if (++st == STAGES) st = 0;
            if (++pf == STAGES) pf = 0;
        }
        cp_async_wait<0>();
        __syncthreads();  // the ring is free: output blocks take its place
        double *o = smem + warp * (WS * OLD);
#pragma unroll
        for (int a = 0; a < F; ++a)
#pragma unroll
            for (int b = 0; b < F; ++b) {
                o[(a * 8 + fr) * OLD + b * 8 + fc * 2] = acc[a][b][0];
                o[(a * 8 + fr) * OLD + b * 8 + fc * 2 + 1] = acc[a][b][1];
            }
        __syncwarp();
        return o;
    }
};

using Tile64 = Tile<32>;
using Tile32 = Tile<16>;

// Below two 64 x 64 tiles per SM the 32 x 32 tiles keep more of the chip at work.
inline bool small_problem(long tiles64) { return tiles64 < 2L * sm_count(); }

}  // namespace dgemm
}  // namespace rkb
