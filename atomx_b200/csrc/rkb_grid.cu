// Arbitrary-grid trapezoid Y^k on the device (atomx numerics/quadrature.py).
//
// atomx's yk_on_grid / yk_pair_dot_batch_on_grid (quadrature.py:234-372) act
// with the Coulomb Green kernel r_<^k / r_>^(k+1) on a density sampled on an
// arbitrary increasing grid, by two cumulative trapezoid scans in
// block-scaled frames: within frame b the tables hold rk_i = (r_i/a_b)^k and
// inverse_i = (r_i/a_b)^-(k+1) / a_b, and a carried moment changes frame by
// the factor transfer[b] = (a_b / a_(b+1))^k <= 1 (quadrature.py:190-231).
//
//   inward:  acc_i = sum over intervals j >= i of 0.5 (b_j + b_(j+1)) dr_j,
//            b_j = rho_j inverse_j, rescaled by transfer at each frame
//            change; y_i = acc_i (y_(n-1) = 0)
//   outward: inner_i = sum over intervals j <= i of 0.5 (a_(j-1) + a_j) dr,
//            a_j = rho_j rk_j, likewise rescaled;
//            y_i = inner_i inverse_i + rk_i y_i,  y_0 = y_0 rk_0
//
// With h_i half the interval between points i and i + 1 (h_(-1) = h_(n-1) = 0), w_i = h_(i-1) +
// h_i, and t_i = 1 except at a frame's first point, where it is the transfer, both
// are first-order recurrences in one point's value at a time:
//
//   inward:  A_i = t_(i+1) A_(i+1) + w_i b_i,   acc_i = t_(i+1) A_(i+1) + h_i b_i
//   outward: B_i = t_i B_(i-1) + w_i a_i,       inner_i = t_i B_(i-1) + h_(i-1) a_i
//
// The reference runs them serially per row.  Here one CTA owns a row and cuts it into
// tiles of TILE points, a warp per tile: a first pass sums every tile's terms, a scan over
// the tiles gives each its two carries, and a second pass scans inside the tiles and
// forms y and its dots with up to FUSED consumers; a row with more puts y into shared
// memory, and a warp per consumer dots it from there.  No tile waits for another, and all
// loads are coalesced (consecutive lanes, consecutive points).  Sums are formed without
// subtractions: a difference of partial sums would cancel on grids whose terms grow
// along the row.  The summation order differs from the serial one, so results agree
// with the reference to rounding, not bit for bit.
//
// Bound by instruction issue (two passes of nine loads and about fifteen FP64
// operations a point, two warp scans in the second).  4000 rows x 20 000 points with 2
// consumers: tile after tile with block-wide scans and y in memory 2.87 ms, this form
// 1.07 ms (tiles of 64, 192, 256 points: 1.2 to 1.4 ms).  More consumers than FUSED by
// taking the second pass again: 4000 rows x 300 points with 40 841 us, 500 rows x 20 000
// points with 64 2.27 ms, from shared memory 131 us and 0.72 ms (from device memory, tile
// after tile, 0.49 and 1.99 ms).  A block takes a warp per tile, up to eight: 4000 rows x
// 300 points with 2 consumers 77 us, with eight warps 135 us.
#include "rkb_common.cuh"

namespace rkb {
namespace grid {

constexpr int THREADS = 256, WARPS = THREADS / 32;  // at most; a short row takes a warp per tile
constexpr int CH = 4, TILE = 32 * CH;  // chunks of 32 points per tile
constexpr int FUSED = 4;               // consumers dotted in one second pass
constexpr int Y_TILES = 64;            // tiles of y that shared memory holds for more consumers
constexpr unsigned FULL = 0xffffffffu;

struct Tables {
    const double *r, *rk, *inverse;  // rk / inverse: the row's multipole, n values
    const long *cuts;                // frame starts, ncuts values (cuts[ncuts-1] = n)
    long ncuts;
    const double *transfer;          // the row's multipole, ncuts-2 values
    long n, i_cut;
};

// Density of a row: a sampled rho, or P_a P_b + Q_a Q_b formed on the
// fly (quadrature.py:313-352 forms it in the same way).
struct DensRow {
    const double *rho;
    __device__ __forceinline__ DensRow from(long i) const { return DensRow{rho + i}; }
    __device__ __forceinline__ double operator()(int i) const { return __ldg(rho + i); }
};
struct DensPair {
    const double *Pa, *Qa, *Pb, *Qb;
    __device__ __forceinline__ DensPair from(long i) const { return DensPair{Pa + i, Qa + i, Pb + i, Qb + i}; }
    __device__ __forceinline__ double operator()(int i) const {
        return __dadd_rn(__dmul_rn(__ldg(Pa + i), __ldg(Pb + i)), __dmul_rn(__ldg(Qa + i), __ldg(Qb + i)));
    }
};

// Index of the first frame start (frames 1 .. ncuts-2) at or beyond p, or ncuts - 1.
__device__ __forceinline__ long frame_from(const Tables &T, long p) {
    long lo = 1, hi = T.ncuts - 1;
    while (lo < hi) {
        const long mid = (lo + hi) / 2;
        if (T.cuts[mid] >= p) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}
__device__ __forceinline__ double transfer_at(const Tables &T, long p) {  // of the frame that starts at p, else 1
    const long q = frame_from(T, p);
    return q < T.ncuts - 1 && T.cuts[q] == p ? T.transfer[q - 1] : 1.0;
}

// A factor >= 0, kept above zero: the product of many frames' factors may underflow where the
// serial scan, which applies them one by one, keeps an infinite sum infinite.
__device__ __forceinline__ double above_zero(double m) {
    return __hiloint2double(max(__double2hiint(m), 0x00100000), __double2loint(m));
}

// x -> m x + s composed along the lanes: lane l receives the map of lanes 0..l in order
// (UP), or of lanes 31..l (down).
template <bool UP>
__device__ __forceinline__ void scan_maps(double &m, double &s, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double m2 = UP ? __shfl_up_sync(FULL, m, o) : __shfl_down_sync(FULL, m, o);
        const double s2 = UP ? __shfl_up_sync(FULL, s, o) : __shfl_down_sync(FULL, s, o);
        if (UP ? lane >= o : lane + o < 32) {
            s = fma(s2, m, s);
            m = above_zero(m * m2);
        }
    }
}
template <bool UP>
__device__ __forceinline__ double scan_sums(double s, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double s2 = UP ? __shfl_up_sync(FULL, s, o) : __shfl_down_sync(FULL, s, o);
        if (UP ? lane >= o : lane + o < 32) s += s2;
    }
    return s;
}

// What the recurrences need of the points base + 32 c + lane of a tile (zeros outside the
// row).  EDGE: the tile may reach beyond the row or hold its first point.
template <bool EDGE, class Dens>
__device__ __forceinline__ void tile_points(const Tables &T, const Dens &rho, long base, int lane, double (&a)[CH],
                                            double (&b)[CH], double (&hl)[CH], double (&hr)[CH], double (&inv)[CH],
                                            double (&rk)[CH]) {
    const long p0 = base + lane;
    const Dens d = rho.from(p0);
    const double *r = T.r + p0, *pi = T.inverse + p0, *pk = T.rk + p0;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        if (EDGE && p0 + 32 * c >= T.n) {
            a[c] = b[c] = hl[c] = hr[c] = inv[c] = rk[c] = 0.0;
            continue;
        }
        const double x = __ldg(r + 32 * c), v = d(32 * c);
        inv[c] = __ldg(pi + 32 * c);
        rk[c] = __ldg(pk + 32 * c);
        hl[c] = EDGE && p0 + 32 * c == 0 ? 0.0 : .5 * (x - __ldg(r + 32 * c - 1));
        hr[c] = EDGE && p0 + 32 * c + 1 >= T.n ? 0.0 : .5 * (__ldg(r + 32 * c + 1) - x);
        b[c] = v * inv[c];
        a[c] = v * rk[c];
    }
}

// A tile's sums A and B, without its carries.
template <bool EDGE, class Dens>
__device__ __forceinline__ void tile_sums(const Tables &T, const Dens &rho, long base, bool cut, int lane, double &si,
                                          double &so) {
    double a[CH], b[CH], hl[CH], hr[CH], inv[CH], rk[CH];
    tile_points<EDGE>(T, rho, base, lane, a, b, hl, hr, inv, rk);
    si = so = 0.0;
    if (!EDGE || !cut) {
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const double w = hl[c] + hr[c];
            si = fma(b[c], w, si);
            so = fma(a[c], w, so);
        }
        si = warp_sum(si);
        so = warp_sum(so);
        return;
    }
#pragma unroll 1
    for (int k = 0; k < CH; ++k) {
        double bk = 0.0, ak = 0.0;  // chunk CH-1-k from the top, chunk k from the bottom
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            if (c == CH - 1 - k) bk = b[c] * (hl[c] + hr[c]);
            if (c == k) ak = a[c] * (hl[c] + hr[c]);
        }
        double mi = transfer_at(T, base + 32 * (CH - 1 - k) + lane + 1), mo = transfer_at(T, base + 32 * k + lane);
        scan_maps<false>(mi, bk, lane);
        si = __shfl_sync(FULL, fma(mi, si, bk), 0);
        scan_maps<true>(mo, ak, lane);
        so = __shfl_sync(FULL, fma(mo, so, ak), 31);
    }
}

// y at a tile's points from its carries A (at base + TILE) and B (at base - 1).
template <bool EDGE, class Dens>
__device__ __forceinline__ void tile_y(const Tables &T, const Dens &rho, long base, bool cut, int lane, double A,
                                       double B, double (&y)[CH]) {
    double a[CH], b[CH], hl[CH], hr[CH], inv[CH], rk[CH];
    tile_points<EDGE>(T, rho, base, lane, a, b, hl, hr, inv, rk);
#pragma unroll
    for (int c = CH - 1; c >= 0; --c) {
        double s = b[c] * (hl[c] + hr[c]), t = 1.0;
        if (EDGE && cut) {
            t = transfer_at(T, base + 32 * c + lane + 1);
            double m = t;
            scan_maps<false>(m, s, lane);
            s = fma(m, A, s);
        } else {
            s = A + scan_sums<false>(s, lane);
        }
        double above = __shfl_down_sync(FULL, s, 1);
        if (lane == 31) above = A;
        A = __shfl_sync(FULL, s, 0);
        // nothing lies behind the last point (and its h_i = 0 times an infinite density is no zero)
        y[c] = EDGE && base + 32 * c + lane + 1 >= T.n ? 0.0 : rk[c] * fma(hr[c], b[c], t * above);
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        double s = a[c] * (hl[c] + hr[c]), t = 1.0;
        if (EDGE && cut) {
            t = transfer_at(T, base + 32 * c + lane);
            double m = t;
            scan_maps<true>(m, s, lane);
            s = fma(m, B, s);
        } else {
            s = B + scan_sums<true>(s, lane);
        }
        double below = __shfl_up_sync(FULL, s, 1);
        if (lane == 0) below = B;
        B = __shfl_sync(FULL, s, 31);
        if (!EDGE || base + 32 * c + lane) y[c] = fma(inv[c], fma(hl[c], a[c], t * below), y[c]);
    }
}

// Exclusive carries of the tiles' maps x -> m x + s in order of the scan: s[c] is replaced by
// the value that tile c starts from.  One warp; tiles with a frame start have their
// multiplier looked up.
template <bool UP>
__device__ void carry_scan(const Tables &T, double *sums, int ntiles, int lane) {
    double carry = 0.0;
    for (int k = 0; k < ntiles; k += 32) {
        const int i = UP ? k + lane : ntiles - 1 - k - (31 - lane);
        double m = 1.0, s = 0.0;
        if (i >= 0 && i < ntiles) {
            s = sums[i];
            // outward: frame starts in [base, base + TILE); inward: in (base, base + TILE]
            const long first = (long)i * TILE + (UP ? 0 : 1);
            for (long q = frame_from(T, first); q < T.ncuts - 1 && T.cuts[q] < first + TILE; ++q) m = above_zero(m * T.transfer[q - 1]);
        }
        scan_maps<UP>(m, s, lane);
        const double after = fma(m, carry, s);  // the value behind this lane's tile
        double before = UP ? __shfl_up_sync(FULL, after, 1) : __shfl_down_sync(FULL, after, 1);
        if (lane == (UP ? 0 : 31)) before = carry;
        if (i >= 0 && i < ntiles) sums[i] = before;
        carry = __shfl_sync(FULL, after, UP ? 31 : 0);
    }
}

struct BatchArgs {
    const double *PA, *QA, *PB, *QB, *rho;
    long ld, rho_ld;
    const long *rows_a, *rows_b, *rows_k;
    const unsigned char *rows_ok;
    long nrows;
    const double *W;  // consumer weight rows (ld w_ld), or null: write y instead
    long w_ld;
    const long *cons_ptr, *cons_rho;
    const double *r, *RK, *inverse, *transfers;
    const long *cuts;
    long n, ncuts, ntr, i_cut;
    double *val;  // consumer dots
    double *y;    // y rows (ld y_ld) when W is null
    long y_ld;
    int y_tiles;  // rows with more than FUSED consumers take y through shared memory, that many tiles at a time (or 0)
};

template <bool DOTS>
__global__ void __launch_bounds__(THREADS, 3) grid_rows_kernel(const __grid_constant__ BatchArgs a, double *scratch) {
    extern __shared__ double tiles_sh[];
    __shared__ double dots_sh[WARPS * FUSED];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int ntiles = (int)((a.n + TILE - 1) / TILE), live = (int)(a.i_cut / TILE) + 1;  // tiles with an output
    double *in = scratch ? scratch + 2L * ntiles * blockIdx.x : tiles_sh, *out = in + ntiles;
    double *y_sh = tiles_sh + (scratch ? 0 : 2 * ntiles);
    for (long m = blockIdx.x; m < a.nrows; m += gridDim.x) {
        if (a.rows_ok && !a.rows_ok[m]) continue;
        const long s0 = DOTS ? a.cons_ptr[m] : 0, s1 = DOTS ? a.cons_ptr[m + 1] : 1;
        if (s0 == s1) continue;
        const long k = a.rows_k[m];
        const Tables T{a.r, a.RK + k * a.n, a.inverse + k * a.n, a.cuts, a.ncuts, a.transfers + k * a.ntr, a.n, a.i_cut};
        const auto rho = [&] {
            if constexpr (DOTS) {
                const long x = a.rows_a[m] * a.ld, z = a.rows_b[m] * a.ld;
                return DensPair{a.PA + x, a.QA + x, a.PB + z, a.QB + z};
            } else {
                return DensRow{a.rho + m * a.rho_ld};
            }
        }();
        // a tile at the row's ends or with a frame start in [base, base + TILE] takes the general form
        auto has_cut = [&](long base) {
            const long q = frame_from(T, base);
            return q < T.ncuts - 1 && T.cuts[q] <= base + TILE;
        };
        // ---- the tiles' sums
        for (int c = warp; c < ntiles; c += warps) {
            const long base = (long)c * TILE;
            const bool cut = has_cut(base);
            double si, so;
            if (cut || base == 0 || base + TILE >= T.n) tile_sums<true>(T, rho, base, cut, lane, si, so);
            else tile_sums<false>(T, rho, base, false, lane, si, so);
            if (lane == 0) {
                in[c] = si;
                out[c] = so;
            }
        }
        __syncthreads();
        if (warp == 0) carry_scan<false>(T, in, ntiles, lane);
        if (warp == 1) carry_scan<true>(T, out, ntiles, lane);
        __syncthreads();
        // ---- many consumers: y into shared memory, and a warp per consumer
        if (DOTS && a.y_tiles && s1 - s0 > FUSED) {
            for (int c0 = 0; c0 < live; c0 += a.y_tiles) {
                for (int c = c0 + warp; c < min(live, c0 + a.y_tiles); c += warps) {
                    const long base = (long)c * TILE;
                    const bool cut = has_cut(base);
                    double y[CH];
                    if (cut || base == 0 || base + TILE >= T.n) tile_y<true>(T, rho, base, cut, lane, in[c], out[c], y);
                    else tile_y<false>(T, rho, base, false, lane, in[c], out[c], y);
#pragma unroll
                    for (int j = 0; j < CH; ++j) y_sh[(c - c0) * TILE + 32 * j + lane] = y[j];
                }
                __syncthreads();
                const long first = (long)c0 * TILE;
                const int pts = (int)min((long)a.y_tiles * TILE, a.i_cut + 1 - first);
                for (long s = s0 + warp; s < s1; s += warps) {
                    const double *w = a.W + a.cons_rho[s] * a.w_ld + first;
                    double part = 0.0;
#pragma unroll 4
                    for (int i = lane; i < pts; i += 32) part = fma(__ldg(w + i), y_sh[i], part);
                    part = warp_sum(part);
                    if (lane == 0) a.val[s] = c0 ? a.val[s] + part : part;
                }
                __syncthreads();
            }
            continue;
        }
        // ---- y, and its dots with FUSED consumers at a time
        for (long s = s0; s < s1; s += FUSED) {
            const double *w[FUSED];
            double part[FUSED];
            if (DOTS)
#pragma unroll
                for (int q = 0; q < FUSED; ++q) {
                    w[q] = a.W + a.cons_rho[s + q < s1 ? s + q : s] * a.w_ld + lane;
                    part[q] = 0.0;
                }
            for (int c = warp; c < live; c += warps) {
                const long base = (long)c * TILE;
                const bool cut = has_cut(base);
                double y[CH];
                if (cut || base == 0 || base + TILE >= T.n) tile_y<true>(T, rho, base, cut, lane, in[c], out[c], y);
                else tile_y<false>(T, rho, base, false, lane, in[c], out[c], y);
                const bool whole = base + TILE <= a.i_cut + 1;
#pragma unroll
                for (int j = 0; j < CH; ++j) {
                    if (!whole && base + 32 * j + lane > a.i_cut) continue;
                    if (!DOTS) a.y[m * a.y_ld + base + 32 * j + lane] = y[j];
                    else
#pragma unroll
                        for (int q = 0; q < FUSED; ++q)
                            if (q == 0 || s + q < s1) part[q] = fma(__ldg(w[q] + base + 32 * j), y[j], part[q]);
                }
            }
            if (!DOTS) break;
#pragma unroll
            for (int q = 0; q < FUSED; ++q) {
                part[q] = warp_sum(part[q]);
                if (lane == 0) dots_sh[warp * FUSED + q] = part[q];
            }
            __syncthreads();
            if (threadIdx.x < FUSED && s + threadIdx.x < s1) {
                double v = 0.0;
                for (int x = 0; x < warps; ++x) v += dots_sh[x * FUSED + threadIdx.x];
                a.val[s + threadIdx.x] = v;
            }
            __syncthreads();
        }
        __syncthreads();  // the carries are overwritten by the next row
    }
}

}  // namespace grid
}  // namespace rkb

using namespace rkb;

static int grid_common_checks(long n, long ncuts, long ntr, long i_cut) {
    RKB_CHECK_ARG(n >= 1, "empty grid");
    RKB_CHECK_ARG(ncuts >= 2 && ntr >= ncuts - 2, "invalid frame tables (ncuts=%ld, transfers=%ld)", ncuts, ntr);
    RKB_CHECK_ARG(i_cut >= 0 && i_cut <= n - 1, "i_cut %ld outside [0, %ld]", i_cut, n - 1);
    return RKB_OK;
}

// max_cons: the most consumers of a row, or -1 if that is not known here.
template <bool DOTS>
static int launch_rows(grid::BatchArgs &a, long max_cons, cudaStream_t st) {
    auto kern = grid::grid_rows_kernel<DOTS>;
    const long tiles = ceil_div(a.n, grid::TILE);
    const int warps = tiles < 2 ? 2 : tiles < grid::WARPS ? (int)tiles : grid::WARPS;  // the carries take two
    const long most = 8L * sm_count() * grid::WARPS / warps;
    long ctas = a.nrows < most ? a.nrows : most;
    size_t bytes = sizeof(double) * 2 * (size_t)tiles;  // the tiles' sums and carries
    const bool fits = bytes <= 200 * 1024;
    // Shared memory for y costs L1 (4000 rows x 5000 points with two consumers: 457 us, 477 with it), so it is
    // taken where rows have, or may have, more consumers than one second pass serves.
    const long live = a.i_cut / grid::TILE + 1;
    const int y_tiles = live < grid::Y_TILES ? (int)live : grid::Y_TILES;
    const size_t y_bytes = sizeof(double) * grid::TILE * (size_t)y_tiles;
    size_t smem = fits ? bytes : 0;
    if (DOTS && (max_cons < 0 || max_cons > grid::FUSED) && smem + y_bytes <= 200 * 1024) {
        a.y_tiles = y_tiles;
        smem += y_bytes;
    }
    double *scratch = nullptr;
    RKB_CUDA(set_smem(kern, (int)smem));
    if (!fits) {  // above 1 638 400 points they go to device memory (n / 8 bytes a CTA): fewer CTAs where that is short
        cudaError_t e;
        while ((e = cudaMallocAsync(reinterpret_cast<void **>(&scratch), bytes * ctas, st)) == cudaErrorMemoryAllocation &&
               ctas > 1) {
            cudaGetLastError();
            ctas = (ctas + 3) / 4;
        }
        RKB_CUDA(e);
    }
    kern<<<(unsigned)ctas, 32 * warps, smem, st>>>(a, scratch);
    const cudaError_t e = cudaGetLastError(), f = scratch ? cudaFreeAsync(scratch, st) : cudaSuccess;
    if (e != cudaSuccess) return cuda_status(e, "grid_rows_kernel");
    RKB_CUDA(f);
    return RKB_OK;
}

extern "C" int rkb_grid_yk_rows(const double *d_rho, long rho_ld, const long *d_rows_k, long nrows,
                                const double *d_r, long n, const double *d_RK, const double *d_inverse,
                                const long *d_cuts, long ncuts, const double *d_transfers, long ntr, long i_cut,
                                double *d_y, long y_ld, void *stream) {
    int st = grid_common_checks(n, ncuts, ntr, i_cut);
    if (st != RKB_OK) return st;
    RKB_CHECK_ARG(y_ld >= n && rho_ld >= n, "row strides must be >= n");
    if (nrows == 0) return RKB_OK;
    grid::BatchArgs a = {};
    a.rho = d_rho; a.rho_ld = rho_ld; a.rows_k = d_rows_k; a.nrows = nrows;
    a.r = d_r; a.RK = d_RK; a.inverse = d_inverse; a.transfers = d_transfers; a.cuts = d_cuts;
    a.n = n; a.ncuts = ncuts; a.ntr = ntr; a.i_cut = i_cut; a.y = d_y; a.y_ld = y_ld;
    return launch_rows<false>(a, 0, as_stream(stream));
}

extern "C" int rkb_grid_pair_dot_batch_cons(const double *d_PA, const double *d_QA, const double *d_PB,
                                       const double *d_QB, long ld, const long *d_rows_a, const long *d_rows_b,
                                       const long *d_rows_k, const unsigned char *d_rows_ok, long nrows,
                                       const double *d_W, long w_ld, const long *d_cons_ptr,
                                       const long *d_cons_rho, const double *d_r, long n, const double *d_RK,
                                       const double *d_inverse, const long *d_cuts, long ncuts,
                                       const double *d_transfers, long ntr, long i_cut, double *d_val,
                                       long max_cons, void *stream) {
    int st = grid_common_checks(n, ncuts, ntr, i_cut);
    if (st != RKB_OK) return st;
    RKB_CHECK_ARG(ld >= n && w_ld >= i_cut + 1, "row strides too small (ld=%ld, w_ld=%ld)", ld, w_ld);
    RKB_CHECK_ARG(max_cons >= -1, "invalid number of consumers");
    if (nrows == 0) return RKB_OK;
    grid::BatchArgs a = {};
    a.PA = d_PA; a.QA = d_QA; a.PB = d_PB; a.QB = d_QB; a.ld = ld; a.rows_a = d_rows_a; a.rows_b = d_rows_b;
    a.rows_k = d_rows_k; a.rows_ok = d_rows_ok; a.nrows = nrows; a.W = d_W; a.w_ld = w_ld;
    a.cons_ptr = d_cons_ptr; a.cons_rho = d_cons_rho; a.r = d_r; a.RK = d_RK; a.inverse = d_inverse;
    a.transfers = d_transfers; a.cuts = d_cuts; a.n = n; a.ncuts = ncuts; a.ntr = ntr; a.i_cut = i_cut;
    a.val = d_val;
    return launch_rows<true>(a, max_cons, as_stream(stream));
}

extern "C" int rkb_grid_pair_dot_batch(const double *d_PA, const double *d_QA, const double *d_PB,
                                       const double *d_QB, long ld, const long *d_rows_a, const long *d_rows_b,
                                       const long *d_rows_k, const unsigned char *d_rows_ok, long nrows,
                                       const double *d_W, long w_ld, const long *d_cons_ptr,
                                       const long *d_cons_rho, const double *d_r, long n, const double *d_RK,
                                       const double *d_inverse, const long *d_cuts, long ncuts,
                                       const double *d_transfers, long ntr, long i_cut, double *d_val,
                                       double *d_work, long work_rows, void *stream) {
    RKB_CHECK_ARG(d_work != nullptr && work_rows >= 1, "a work area of at least one row is required");
    return rkb_grid_pair_dot_batch_cons(d_PA, d_QA, d_PB, d_QB, ld, d_rows_a, d_rows_b, d_rows_k, d_rows_ok, nrows, d_W,
                                        w_ld, d_cons_ptr, d_cons_rho, d_r, n, d_RK, d_inverse, d_cuts, ncuts,
                                        d_transfers, ntr, i_cut, d_val, -1, stream);
}
