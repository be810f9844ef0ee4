// Split-precision R^k engine: factored Green operator + Ozaki-II (CRT) INT8
// residue GEMMs on the 5th-generation tensor cores, recombined in FP64.
//
//   R(ac;bd) = X_ac . X_bd - Z_ac . Z_bd + left_ac . right_bd
//
// K2x  split_rows_kernel  (one warp per (pair, k) row, FP64 on CUDA cores)
//      g = w (P_a P_c + Q_a Q_c);  per body cell m >= 1:  d_m = u_m . g_m and
//      the exclusive suffix sums T_m = sum_{m'>m} d_m' (warp-shuffle scans);
//      X_m = L_mm^T g_m + c_m T_m;  Z_e = z_e . g_{cell(e)};
//      FP64 core terms left = [g_0, alpha sx, q/sx], right = [G_00 g_0, q/sx,
//      alpha sx] with alpha = v_0.g_0 and q = T_0 (the core-body coupling).
//      The FP64 row [X | Z] goes to a scratch buffer with its power-of-two
//      scale (|x| < 2^bits); split_residues_kernel then rounds it to integers
//      x~ and writes int8 residues x~ mod m_i (and the B copy with Z negated)
//      in a [modulus][row][kpad] layout, one 16-byte store per modulus.
//      Per row the kernels also record (cbound, CB_STRIDE doubles): the
//      screen bounds |g_0|, |G_00 g_0|, |alpha sx|, |q/sx| relative to the row
//      scale, and for the certificate |[X | Z]| and the FP64 diagonal
//      R_aa = |X|^2 - |Z|^2 + left.right.
//
// K3s  crt_syrk_kernel  (persistent, one CTA per SM, 20 warps)
//      warp 0: TMA producer — 128x128-byte boxes (SWIZZLE_128B) of the A and B
//              residue matrices into a STAGES-deep ring;
//      warp 1: TMEM owner + MMA issuer — tcgen05.mma.kind::i8, M=N=128, K=32,
//              int32 accumulators in a double-buffered TMEM tile;
//      warps 2, 3: the next tile's record (row scales, screen bounds, table) into
//              shared memory: beside the TMA feed an L2 read takes over a thousand
//              cycles, and the epilogue makes none;
//      warps 4-19: epilogue (4 TMEM lane quarters x 4 column groups).  Per modulus
//              one IMAD.WIDE an entry folds the int32 accumulator, unreduced, into
//              the open digit's 64-bit sum; three times a tile the digit is reduced
//              (FP64 quotient) and its CRT weight added to the entry's 72-bit
//              fraction x / M, 64 bits of it in TMEM columns 256..511 and a byte in
//              shared memory.  A finished tile's scaling,
//              core correction (when it is not screened out) and stores (the tile and
//              its transpose) run in four chunks between the next tile's first moduli,
//              so that the MMAs do not wait for them.
//      The epilogue's instructions were the limit: reducing every accumulator to its
//      residue and merging residues in pairs took about 13 instructions per entry and
//      modulus (IMAD.HI issues at a quarter rate), spilled registers went through L2,
//      and the MMAs stood still during the final phase.  Z=70 table (kdim 1024): 2.88
//      ms before, 2.47 ms now; N=2112 table (kdim 2176): 2.58 and 2.49 ms.
//      The fraction is off by 3 x 2^-73 of M at most (one rounding per digit), less than
//      the 2^-70 of a recombination in doubles; with 64 bits it would be 2^-63.4, more than
//      a split narrow for its moduli is off by itself.  The eight more bits take 0.10 ms.
//      Every mbarrier wait is bounded; on timeout the kernel records
//      RKB_ETIMEDOUT in *status, every role gives up, waits (again with a limit) for
//      the loads and MMAs that it has issued, and returns.  A non-finite entry is only
//      recorded (its row has zero residues and a NaN scale): the launch runs to its end.
#include <cuda.h>

#include <cfloat>

#include <mutex>
#include <numeric>

#include "rkb_common.cuh"

namespace rkb {
namespace split {

constexpr int MAXMOD = 12;
// Doubles per row of the cbound array: [0] |g_0|, [1] |G_00 g_0|, [2] |alpha sx|,
// [3] |q/sx| (each times 2^-e of the row scale), [4] |[X | Z]|, [5] R_aa, [6..7] 0.
constexpr int CB_STRIDE = 8;

// The per-row record: screen bounds relative to 2^-e (infinite for a zero
// row, which is never screened), the row norm and the FP64 diagonal.
__device__ __forceinline__ void write_row_record(double *cb, double amax, int ex, double n_g0, double n_gg,
                                                 double a_sx, double q_sx, double xsq, double zsq, double g0gg) {
    const double rel = amax > 0.0 ? ldexp(1.0, -ex) : INFINITY;
    cb[0] = sqrt(n_g0) * rel;
    cb[1] = sqrt(n_gg) * rel;
    cb[2] = fabs(a_sx) * rel;
    cb[3] = fabs(q_sx) * rel;
    cb[4] = sqrt(xsq + zsq);
    cb[5] = xsq - zsq + g0gg + 2.0 * a_sx * q_sx;
    cb[6] = 0.0;
    cb[7] = 0.0;
}

// =========================================================================
// K2x — transform, quantise, residues
// =========================================================================
struct RowsArgs {
    const double *P, *Q;
    long orb_ld;
    const long *pairs, *row_pair;
    const int *row_k;
    long nrows;
    const double *w;
    int nv, ng;
    const double *ktab;
    const long *koff;  // by k
    int bits, n_mod;
    int mod[MAXMOD];
    uint32_t magic[MAXMOD], c20[MAXMOD], bias[MAXMOD];  // 2^32/m + 1, 2^20 mod m, m * 2^20
    double inv_mod[MAXMOD];    // RN(1/m)
    signed char *resA, *resB;  // [n_mod][nrows_total][kpad]; resB may be null
    long kpad, row_base, nrows_total;
    long b_ld;   // row stride and width of resB
    int b_col0;  // first column that resB holds (cell kernel; a multiple of 128)
    double *rowscale, *left, *right, *cbound;
    double *xwork;  // scratch rows [X | Z | 0] (row stride kpad)
    int cwp;
};

__device__ __forceinline__ double rho_at(const RowsArgs &a, long q, long i) {
    long p = a.row_pair[q];
    long x = a.pairs[2 * p], c = a.pairs[2 * p + 1];
    return __dadd_rn(__dmul_rn(a.P[x * a.orb_ld + i], a.P[c * a.orb_ld + i]),
                     __dmul_rn(a.Q[x * a.orb_ld + i], a.Q[c * a.orb_ld + i]));
}

// x mod m in [0, m) for 0 <= x < 2^32 with integer operations only:
// q = hi32(x * (floor(2^32/m) + 1)) exceeds x/m by less than x/2^32 < 1, so it
// is floor(x/m) or one more, and one conditional add repairs the remainder.
__device__ __forceinline__ uint32_t umod_small(uint32_t x, uint32_t m, uint32_t magic) {
    const uint32_t q = __umulhi(x, magic);
    int r = (int)(x - q * m);
    return (uint32_t)(r + (r < 0 ? (int)m : 0));
}

// Centred int8 residue (as a byte) of an integer x = hi * 2^20 + lo, |hi| <= 2^20, 0 <= lo < 2^20.
__device__ __forceinline__ uint32_t residue_i8(int hi, uint32_t lo, uint32_t m, uint32_t magic, uint32_t c20,
                                               uint32_t bias) {
    // (hi mod m) * (2^20 mod m) + (lo mod m): every operand nonnegative and < 2^29
    const uint32_t h = umod_small((uint32_t)(hi + (int)bias), m, magic);
    const uint32_t l = umod_small(lo, m, magic);
    const uint32_t r = umod_small(h * c20 + l, m, magic);
    const int rc = (int)r - (r > 127u ? (int)m : 0);
    return (uint32_t)rc & 0xffu;
}

// One warp per row.  Shared memory per warp: g (n doubles) and the per-cell
// suffix sums (nv doubles).  Cells are processed by lane groups of ng lanes
// (lane = node of a cell), so shared and global accesses are consecutive
// across lanes.  The FP64 row [X | Z | 0...] goes to the caller's scratch
// buffer; split_residues_kernel turns it into int8 residues.
template <int NG>
__global__ void __launch_bounds__(128) split_rows_kernel(RowsArgs a) {
    const int ng = NG > 0 ? NG : a.ng;
    const int nv = a.nv;
    const long n = (long)nv * ng;
    extern __shared__ double sm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    // segment lengths rounded to even counts of doubles keep every segment 16-byte aligned
    const long np = (n + 1) & ~1L, nvp = (nv + 1) & ~1L;
    const long per_warp = np + nvp;
    double *g = sm + (long)wib * per_warp;
    double *tsuf = g + np;
    const long q = (long)blockIdx.x * (blockDim.x >> 5) + wib;
    if (q >= a.nrows) return;
    const int k = a.row_k[q];
    const double *tab = a.ktab + a.koff[k];
    const double *u = tab;
    const double *Lb = u + n;
    const double *C = Lb + (long)nv * ng * ng;
    const double *v0 = C + (long)nv * ng;
    const double *G00 = v0 + ng;
    const double sx = G00[ng * ng];
    const int nz = (int)G00[ng * ng + 1];
    const double *zt = G00 + ng * ng + 2;
    const long kbody = (long)(nv - 1) * ng;
    // lane groups: cpp cells per pass, lane -> (cell offset, node)
    const int cpp = 32 / ng;
    const int sub = lane / ng, node = lane - sub * ng;
    const bool glane = sub < cpp;

    for (long i = lane; i < n; i += 32) g[i] = __dmul_rn(a.w[i], rho_at(a, q, i));
    __syncwarp();
    // alpha = v_0 . g_0: the core multipole moment of the core-body coupling
    double alpha = 0.0;
    for (int j = lane; j < ng; j += 32) alpha = fma(v0[j], g[j], alpha);
    alpha = warp_sum(alpha);

    // cell dots d_m = u_m . g_m (m >= 1) by lane groups, segmented shuffle sums
    for (int m0 = 0; m0 < nv; m0 += cpp) {
        const int m = m0 + sub;
        double p = 0.0;
        if (glane && m >= 1 && m < nv) p = u[(long)m * ng + node] * g[(long)m * ng + node];
        // sum over the ng lanes of the group (groups never straddle: lanes >= cpp*ng idle)
        double tot = 0.0;
        for (int t = 0; t < ng; ++t) tot += __shfl_sync(0xffffffffu, p, sub * ng + t < 32 ? sub * ng + t : lane);
        if (glane && node == 0 && m < nv) tsuf[m] = (m >= 1) ? tot : 0.0;
    }
    __syncwarp();
    // exclusive suffix sums over cells: lane l owns cell (end - l) of each chunk
    const int nch = (nv + 31) >> 5;
    double carry = 0.0;
    for (int c = 0; c < nch; ++c) {
        const int m = nv - 1 - ((c << 5) + lane);
        const double d = m >= 0 ? tsuf[m] : 0.0;
        const double incl = warp_inclusive_scan(d, lane);
        const double excl = __shfl_up_sync(0xffffffffu, incl, 1);
        __syncwarp();
        if (m >= 0) tsuf[m] = lane == 0 ? carry : carry + excl;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();

    // the row [X | Z | 0...] into the scratch row, with its maximum and sums of squares
    const long grow = a.row_base + q;  // row index in the residue matrices
    double *xs = a.xwork + grow * a.kpad;
    double amax = 0.0, xsq = 0.0, zsq = 0.0;
    bool bad = false;  // fmax drops NaNs, so non-finite values are tracked apart
    for (int m0 = 1; m0 < nv; m0 += cpp) {
        const int m = m0 + sub;
        if (glane && m < nv) {
            const double *L = Lb + (long)m * ng * ng;
            const double *gm = g + (long)m * ng;
            double x = C[(long)m * ng + node] * tsuf[m];
            for (int i = node; i < ng; ++i) x = fma(L[i * ng + node], gm[i], x);
            xs[(long)(m - 1) * ng + node] = x;
            amax = fmax(amax, fabs(x));
            xsq = fma(x, x, xsq);
            bad |= !isfinite(x);
        }
    }
    for (int e = lane; e < nz; e += 32) {
        const double *ze = zt + (long)e * (ng + 1);
        const double *gm = g + (long)ze[0] * ng;
        double x = 0.0;
        for (int i = 0; i < ng; ++i) x = fma(ze[1 + i], gm[i], x);
        xs[kbody + e] = x;
        amax = fmax(amax, fabs(x));
        zsq = fma(x, x, zsq);
        bad |= !isfinite(x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    xsq = warp_sum(xsq);
    zsq = warp_sum(zsq);

    for (long c = kbody + nz + lane; c < a.kpad; c += 32) xs[c] = 0.0;
    int ex = 0;
    double inv_scale = 0.0;
    if (amax > 0.0 && isfinite(amax)) {
        frexp(amax, &ex);  // amax < 2^ex
        inv_scale = ldexp(1.0, ex - a.bits);
    }

    // FP64 core terms: left = [g_0, alpha sx, q/sx], right = [G_00 g_0, q/sx, alpha sx]
    const double a_sx = alpha * sx, q_sx = tsuf[0] / sx;  // T_0 = u_b . g_b
    bad |= !isfinite(a_sx) || !isfinite(q_sx);
    double *lf = a.left + grow * a.cwp, *rt = a.right + grow * a.cwp;
    double n1 = 0.0, n2 = 0.0, gg = 0.0;
    for (int i = lane; i < a.cwp; i += 32) {
        double gi = 0.0, sacc = 0.0;
        if (i < ng) {
            gi = g[i];
            for (int j = 0; j < ng; ++j) sacc = fma(G00[i * ng + j], g[j], sacc);
            n1 = fma(gi, gi, n1);
            n2 = fma(sacc, sacc, n2);
            gg = fma(gi, sacc, gg);
        } else if (i == ng) {
            gi = a_sx;
            sacc = q_sx;
        } else if (i == ng + 1) {
            gi = q_sx;
            sacc = a_sx;
        }
        lf[i] = gi;
        rt[i] = sacc;
    }
    n1 = warp_sum(n1);
    n2 = warp_sum(n2);
    gg = warp_sum(gg);
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        // a non-finite row gets a NaN scale: its residues are zero and every
        // entry it reaches is NaN, which the contraction reports
        a.rowscale[grow] = bad ? __longlong_as_double(0x7ff8000000000000LL) : inv_scale;
        write_row_record(a.cbound + grow * CB_STRIDE, amax, ex, n1, n2, a_sx, q_sx, xsq, zsq, gg);
    }
}


// Residues of the scaled rows: one thread per (row, 16 columns).  x = rint(X *
// 2^(bits - e_row)) is an exact integer with |x| <= 2^bits; each modulus gets
// one 16-byte store (and the B copy negates the row's Z columns).
__global__ void __launch_bounds__(256) split_residues_kernel(RowsArgs a, const int *__restrict__ z_count) {
    const long per_row = a.kpad / 16;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.nrows * per_row) return;
    const long q = t / per_row, c0 = (t - q * per_row) * 16;
    const long grow = a.row_base + q;
    const double rs = a.rowscale[grow];
    const double scale = rs > 0.0 ? 1.0 / rs : 0.0;  // an exact power of two
    const double *xs = a.xwork + grow * a.kpad + c0;
    int hi[16];
    uint32_t lo[16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
        const double2 v = *reinterpret_cast<const double2 *>(xs + j);
        double y0 = v.x * scale, y1 = v.y * scale;
        y0 = fabs(y0) <= 0x1p40 ? y0 : 0.0;  // NaN rows (and a zero scale) give zeros
        y1 = fabs(y1) <= 0x1p40 ? y1 : 0.0;
        const long long x0 = (long long)rint(y0), x1 = (long long)rint(y1);
        hi[j] = (int)(x0 >> 20);
        lo[j] = (uint32_t)(x0 & 0xfffffLL);
        hi[j + 1] = (int)(x1 >> 20);
        lo[j + 1] = (uint32_t)(x1 & 0xfffffLL);
    }
    const long kbody = (long)(a.nv - 1) * a.ng;
    const long zhi = kbody + z_count[a.row_k[q]];
    const bool anyz = a.resB != nullptr && c0 + 16 > kbody && c0 < zhi;
    for (int md = 0; md < a.n_mod; ++md) {
        const uint32_t m = (uint32_t)a.mod[md], magic = a.magic[md], c20 = a.c20[md], bias = a.bias[md];
        uint32_t w[4], wb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t va = 0u, vb = 0u;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int j = 4 * i + s;
                const uint32_t r = residue_i8(hi[j], lo[j], m, magic, c20, bias);
                va |= r << (8 * s);
                uint32_t rb = r;
                if (anyz && c0 + j >= kbody && c0 + j < zhi) {
                    int nr = -(int)(int8_t)(uint8_t)r;  // residue of -x, centred again
                    nr -= nr > 127 ? (int)m : 0;
                    rb = (uint32_t)nr & 0xffu;
                }
                vb |= rb << (8 * s);
            }
            w[i] = va;
            wb[i] = vb;
        }
        const long o = ((long)md * a.nrows_total + grow) * a.kpad + c0;
        *reinterpret_cast<uint4 *>(a.resA + o) = make_uint4(w[0], w[1], w[2], w[3]);
        if (a.resB) *reinterpret_cast<uint4 *>(a.resB + o) = make_uint4(wb[0], wb[1], wb[2], wb[3]);
    }
}


// ---------------------------------------------------------------------------
// Fused row kernel (rows whose body fits in registers): one warp per row, no
// shared memory and no FP64 workspace.  Cells are taken from the last to the
// first in passes of CPP = 32/NG cells (lane = (cell offset, node)), so the
// suffix sums t_m = sum_{m'>m} u_m'.g_m' are a running carry; each lane keeps
// its X value of every pass in registers until the row maximum is known, then
// writes int8 residues directly.
//
// Residue layout (any column order shared by every row of a GEMM leaves the
// products unchanged): the value of pass p held by lane l goes to position
// 128*(p/4) + 4*l + (p%4), so four passes form one 32-bit word per lane and a
// warp stores 128 contiguous bytes per modulus.  Lanes without a cell (l >=
// CPP*NG, or cell 0 / below in the last pass) hold zeros.  The body therefore
// spans fused_body_width() positions; Z column e sits at body_width + e.
__host__ __device__ constexpr int fused_cpp(int ng) { return 32 / ng; }
__host__ __device__ inline long fused_passes(int nv, int ng) { return (nv - 1 + fused_cpp(ng) - 1) / fused_cpp(ng); }
__host__ __device__ inline long fused_body_width(int nv, int ng) { return 128 * ((fused_passes(nv, ng) + 3) / 4); }
constexpr int FUSED_PMAX = 32;  // passes kept in registers (body width <= 1024)
constexpr int FUSED_ZMAX = 64;  // Z columns per row (two per lane)

// Centred residue of an integer-valued double |x| <= 2^40 modulo m <= 256:
// q = round(x/m) with the 1.5*2^52 rounding constant (x*inv_m is within
// 2^-13 of x/m, and x/m is never that close to a half-integer except exactly
// at one, where either rounding is fine), r = x - q*m exactly by one fma,
// |r| <= m/2, then moved into [-128, 127].
__device__ __forceinline__ uint32_t residue_f64(double x, double m, double inv_m) {
    const double rc = 6755399441055744.0;  // 1.5 * 2^52
    const double q = __dadd_rn(__fma_rn(x, inv_m, rc), -rc);
    const double r = __fma_rn(-q, m, x);
    int ri = __double2loint(__dadd_rn(r, rc));
    ri -= ri > 127 ? (int)m : 0;
    return (uint32_t)ri & 0xffu;
}

template <int NG>
__global__ void __launch_bounds__(128) split_rows_fused_kernel(RowsArgs a) {
    constexpr int CPP = 32 / NG;
    constexpr unsigned FULL = 0xffffffffu;
    const int nv = a.nv;
    const int lane = threadIdx.x & 31;
    const long q = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= a.nrows) return;
    const int k = a.row_k[q];
    const long pr = a.row_pair[q];
    const double *Pa = a.P + a.pairs[2 * pr] * a.orb_ld, *Pc = a.P + a.pairs[2 * pr + 1] * a.orb_ld;
    const double *Qa = a.Q + a.pairs[2 * pr] * a.orb_ld, *Qc = a.Q + a.pairs[2 * pr + 1] * a.orb_ld;
    const long n = (long)nv * NG;
    const double *tab = a.ktab + a.koff[k];
    const double *u = tab;
    const double *Lb = u + n;
    const double *C = Lb + (long)nv * NG * NG;
    const double *v0 = C + (long)nv * NG;
    const double *G00 = v0 + NG;
    const double sx = G00[NG * NG];
    const int nz = (int)G00[NG * NG + 1];
    const double *zt = G00 + NG * NG + 2;
    const int sub = lane / NG, node = lane - sub * NG;
    const bool glane = sub < CPP;
    const long grow = a.row_base + q;
    auto gval = [&](long i) {
        return __dmul_rn(a.w[i], __dadd_rn(__dmul_rn(Pa[i], Pc[i]), __dmul_rn(Qa[i], Qc[i])));
    };

    // cell 0: g_0 (lanes < NG), alpha = v_0 . g_0, G_00 g_0 and their norms
    const double g0 = lane < NG ? gval(lane) : 0.0;
    const double alpha = warp_sum(lane < NG ? v0[lane] * g0 : 0.0);
    double sg = 0.0;
#pragma unroll
    for (int j = 0; j < NG; ++j) {
        const double gj = __shfl_sync(FULL, g0, j);
        if (lane < NG) sg = fma(G00[lane * NG + j], gj, sg);
    }
    const double n1 = warp_sum(g0 * g0), n2 = warp_sum(sg * sg), gg = warp_sum(g0 * sg);

    // body passes, last cell first
    const int P = (int)fused_passes(nv, NG);
    double xs[FUSED_PMAX];
    double carry = 0.0, amax = 0.0, xsq = 0.0, zsq = 0.0;
    bool bad = false;
#pragma unroll
    for (int p = 0; p < FUSED_PMAX; ++p) {
        xs[p] = 0.0;
        if (p < P) {
            const int m = nv - 1 - p * CPP - sub;
            const bool ok = glane && m >= 1;
            const long i = (long)m * NG + node;
            const double g = ok ? gval(i) : 0.0;
            double dm = ok ? u[i] * g : 0.0;
            // sum over the NG lanes of the group (every lane of the group gets it)
            {
                double tot = 0.0;
#pragma unroll
                for (int t = 0; t < NG; ++t) tot += __shfl_sync(FULL, dm, (sub * NG + t) & 31);
                dm = tot;
            }
            // carry of the cells already passed plus the higher cells of this pass
            double before = 0.0, all = 0.0;
#pragma unroll
            for (int s = 0; s < CPP; ++s) {
                const double ds = __shfl_sync(FULL, dm, s * NG);
                all += ds;
                before += s < sub ? ds : 0.0;
            }
            const double t = carry + before;
            carry += all;
            const double *L = Lb + (long)m * NG * NG;
            double x = ok ? C[i] * t : 0.0;
#pragma unroll
            for (int ii = 0; ii < NG; ++ii) {
                const double gi = __shfl_sync(FULL, g, (sub * NG + ii) & 31);
                if (ok && ii >= node) x = fma(L[ii * NG + node], gi, x);
            }
            xs[p] = x;
            amax = fmax(amax, fabs(x));
            xsq = fma(x, x, xsq);
            bad |= !isfinite(x);
        }
    }
    // core terms: left = [g_0, alpha sx, q/sx], right = [G_00 g_0, q/sx, alpha sx]
    // (the carry now holds q = u_b . g_b on every lane)
    const double a_sx = alpha * sx, q_sx = carry / sx;
    bad |= !isfinite(a_sx) || !isfinite(q_sx);
    if (lane < a.cwp) {
        a.left[grow * a.cwp + lane] = lane < NG ? g0 : (lane == NG ? a_sx : (lane == NG + 1 ? q_sx : 0.0));
        a.right[grow * a.cwp + lane] = lane < NG ? sg : (lane == NG ? q_sx : (lane == NG + 1 ? a_sx : 0.0));
    }
    // Z columns: lane e and e + 32
    double zx[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int e = lane + 32 * h;
        if (e < nz) {
            const double *ze = zt + (long)e * (NG + 1);
            const long base = (long)ze[0] * NG;
            double x = 0.0;
            for (int ii = 0; ii < NG; ++ii) x = fma(ze[1 + ii], gval(base + ii), x);
            zx[h] = x;
            amax = fmax(amax, fabs(x));
            zsq = fma(x, x, zsq);
            bad |= !isfinite(x);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(FULL, amax, o));
    xsq = warp_sum(xsq);
    zsq = warp_sum(zsq);
    bad = __any_sync(FULL, bad);
    int ex = 0;
    double scale = 0.0, inv_scale = 0.0;
    if (!bad && amax > 0.0) {
        frexp(amax, &ex);  // amax < 2^ex
        scale = ldexp(1.0, a.bits - ex);
        inv_scale = ldexp(1.0, ex - a.bits);
    }
    if (lane == 0) {
        a.rowscale[grow] = bad ? __longlong_as_double(0x7ff8000000000000LL) : inv_scale;
        write_row_record(a.cbound + grow * CB_STRIDE, amax, ex, n1, n2, a_sx, q_sx, xsq, zsq, gg);
    }

    // quantise in place (exact integers, |x| <= 2^bits) and write residues
    const double rc = 6755399441055744.0;
#pragma unroll
    for (int p = 0; p < FUSED_PMAX; ++p) xs[p] = __dadd_rn(__fma_rn(xs[p], scale, rc), -rc);
    zx[0] = __dadd_rn(__fma_rn(zx[0], scale, rc), -rc);
    zx[1] = __dadd_rn(__fma_rn(zx[1], scale, rc), -rc);
    const long bw = fused_body_width(nv, NG);
    for (int md = 0; md < a.n_mod; ++md) {
        const double m = (double)a.mod[md], inv_m = a.inv_mod[md];
        signed char *rowA = a.resA + ((long)md * a.nrows_total + grow) * a.kpad;
        signed char *rowB = a.resB ? a.resB + ((long)md * a.nrows_total + grow) * a.kpad : nullptr;
#pragma unroll
        for (int j = 0; j < FUSED_PMAX / 4; ++j) {
            if (4 * j < P) {
                uint32_t word = 0u;
#pragma unroll
                for (int s = 0; s < 4; ++s) word |= residue_f64(xs[4 * j + s], m, inv_m) << (8 * s);
                reinterpret_cast<uint32_t *>(rowA + 128 * j)[lane] = word;
                if (rowB) reinterpret_cast<uint32_t *>(rowB + 128 * j)[lane] = word;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = lane + 32 * h;
            if (e < nz) {
                const uint32_t r = residue_f64(zx[h], m, inv_m);
                rowA[bw + e] = (signed char)r;
                if (rowB) {
                    int nr = -(int)(int8_t)(uint8_t)r;  // residue of -x, centred again
                    nr -= nr > 127 ? (int)m : 0;
                    rowB[bw + e] = (signed char)nr;
                }
            }
        }
    }
}


// ---------------------------------------------------------------------------
// Cell-parallel row kernel: one block per R rows, one thread per cell.  Thread t
// owns cell m = nv-1-t (cells last to first), so a forward exclusive block
// scan of the cell dots u_m.g_m gives each cell its suffix sum t_m directly.
// The block first forms g = w*rho of its rows with coalesced loads into a
// padded shared-memory image; each thread then reads its cell's g and the
// cell-minor factor copy (entry i of every cell contiguous, so a warp's reads
// are consecutive), once for all R rows, and forms X = L_m^T g_m + C_m t_m in
// registers, in place of g.  Threads past the cells compute the Z columns.  X
// and Z go back to the image in column order, and once a block maximum has
// fixed each row's power-of-two scale, the residues are written: a thread takes
// four consecutive columns, so that a warp stores 128 contiguous bytes per
// modulus and the work is even whatever the number of cells.  Columns are in
// natural order: (m-1)*ng + node, then Z.
//
// Bound by instruction issue.  A residue costs six FP32 operations (an integer
// of 41 bits as three exact limbs; FP32 issues at twice the rate of FP64 and
// integer multiplies), and the factor tables, R rows per read, stay off L2.  One
// row per block with FP64 residues, byte stores to shared images and a copy
// out took 0.856 ms for the Z=70 rows (56 209 x 896) and 2.06 ms for N = 2112
// (44 900 rows); this form takes 0.732 and 1.25 ms.  R = 1, 2, 4 took 0.753, 0.759,
// 0.732 ms for the first and 1.37, 1.25, 1.35 ms for the second: four rows fit the
// registers up to eight nodes a cell, two beyond.
//
// Cell-minor factor table of one multipole (doubles), nv cells:
//   u[NG][nv] | C[NG][nv] | L[NG][NG][nv] (L[i][node][m])
constexpr int CELL_ZMAX = 128;  // Z columns per row of the cell kernel (one thread each, nv + Z <= 256)
__host__ __device__ constexpr int cell_rows(int ng) { return ng <= 8 ? 4 : 2; }  // R: R x ng doubles a thread
// doubles from one cell to the next in the image: odd, so that cell-strided reads do not conflict
__host__ __device__ constexpr int cell_stride(int ng) { return ng | 1; }
__host__ __device__ constexpr long cell_image(int ng, long nv, long z) {  // doubles of one row's image
    return (nv + (z + ng - 1) / ng) * cell_stride(ng);
}

struct ResidueArgs {
    float4 mod[MAXMOD];  // m, 1/m, 2^14 mod m and 2^28 mod m (nearest zero)
};

template <int NG, int R>
__device__ __forceinline__ void cell_rows_body(const RowsArgs &a, const ResidueArgs &f,
                                               const double *__restrict__ ktab_t, const long *__restrict__ koff_t,
                                               long q, long zmax, double *img, double *red) {
    constexpr int GS = cell_stride(NG);
    const int nv = a.nv;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarp = blockDim.x >> 5;
    const long ld = cell_image(NG, nv, zmax);
    const int k = a.row_k[q];
    const long n = (long)nv * NG;
    const double *tab = a.ktab + a.koff[k];
    const double *v0 = tab + n + (long)nv * NG * NG + (long)nv * NG;
    const double *G00 = v0 + NG;
    const double sx = G00[NG * NG];
    const int nz = min((int)G00[NG * NG + 1], (int)zmax);
    const double *zt = G00 + NG * NG + 2;
    const double *tt = ktab_t + koff_t[k];
    const double *ut = tt, *Ct = tt + n, *Lt = tt + 2 * n;
    const int kbody = (nv - 1) * NG, zend = kbody + nz;
    const long grow = a.row_base + q;
    // g = w * (P_a P_c + Q_a Q_c) of the rows, coalesced
    {
        const double *Pa[R], *Pc[R], *Qa[R], *Qc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const long pr = a.row_pair[q + r];
            const long x = a.pairs[2 * pr] * a.orb_ld, c = a.pairs[2 * pr + 1] * a.orb_ld;
            Pa[r] = a.P + x;
            Qa[r] = a.Q + x;
            Pc[r] = a.P + c;
            Qc[r] = a.Q + c;
        }
        for (int j = tid; j < (int)n; j += blockDim.x) {
            const int cell = j / NG, at = cell * GS + (j - cell * NG);
            const double w = __ldg(a.w + j);
#pragma unroll
            for (int r = 0; r < R; ++r)
                img[r * ld + at] = __dmul_rn(w, __dadd_rn(__dmul_rn(__ldg(Pa[r] + j), __ldg(Pc[r] + j)),
                                                          __dmul_rn(__ldg(Qa[r] + j), __ldg(Qc[r] + j))));
        }
    }
    __syncthreads();
    const int m = nv - 1 - tid;  // this thread's cell (m < 0: a Z column or idle)
    double g[R][NG], d[R];
#pragma unroll
    for (int r = 0; r < R; ++r) d[r] = 0.0;
    if (m >= 0) {
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const double u = m >= 1 ? __ldg(ut + (long)i * nv + m) : 0.0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                g[r][i] = img[r * ld + m * GS + i];
                d[r] = fma(u, g[r][i], d[r]);
            }
        }
    }
    // Z columns: thread nv + e
    const int e = tid - nv;
    double zx[R];
#pragma unroll
    for (int r = 0; r < R; ++r) zx[r] = 0.0;
    if (e >= 0 && e < nz) {
        const double *ze = zt + (long)e * (NG + 1);
        const int cz = (int)ze[0] * GS;
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            const double z = ze[1 + i];
#pragma unroll
            for (int r = 0; r < R; ++r) zx[r] = fma(z, img[r * ld + cz + i], zx[r]);
        }
    }
    // the core cell: lane (r, i) of the block's last warp forms G_00 g_0 (row i)
    double *core = red + 8 * 4 * R;  // [R][2 * NG]: g_0, G_00 g_0
    for (int o = wid == nwarp - 1 ? lane : R * NG; o < R * NG; o += 32) {
        const int r = o / NG, i = o - r * NG;
        const double *g0 = img + r * ld;
        double sacc = 0.0;
#pragma unroll
        for (int j = 0; j < NG; ++j) sacc = fma(__ldg(G00 + i * NG + j), g0[j], sacc);
        a.left[(grow + r) * a.cwp + i] = g0[i];
        a.right[(grow + r) * a.cwp + i] = sacc;
        core[r * 2 * NG + i] = g0[i];
        core[r * 2 * NG + NG + i] = sacc;
    }
    // exclusive scan of d over threads (= suffix sums over cells)
    double t_m[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double incl = warp_inclusive_scan(d[r], lane);
        if (lane == 31) red[wid * R + r] = incl;
        t_m[r] = __shfl_up_sync(0xffffffffu, incl, 1);
        if (lane == 0) t_m[r] = 0.0;
    }
    __syncthreads();  // from here on nothing reads g from the image
#pragma unroll
    for (int r = 0; r < R; ++r) {
        double before = 0.0;
        for (int w = 0; w < wid; ++w) before += red[w * R + r];
        t_m[r] = lane == 0 ? before : before + t_m[r];
    }
    uint32_t top[R];  // largest exponent field
    double xsq[R], zsq[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        top[r] = 0u;
        xsq[r] = zsq[r] = 0.0;
    }
    if (m >= 1) {
#pragma unroll
        for (int node = 0; node < NG; ++node) {
            const double C = __ldg(Ct + (long)node * nv + m);
            double xv[R];
#pragma unroll
            for (int r = 0; r < R; ++r) xv[r] = C * t_m[r];
#pragma unroll
            for (int i = node; i < NG; ++i) {
                const double L = __ldg(Lt + ((long)i * NG + node) * nv + m);
#pragma unroll
                for (int r = 0; r < R; ++r) xv[r] = fma(L, g[r][i], xv[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                img[r * ld + m * GS + node] = xv[r];
                top[r] = max(top[r], (uint32_t)__double2hiint(xv[r]) & 0x7ff00000u);
                xsq[r] = fma(xv[r], xv[r], xsq[r]);
            }
        }
    }
    if (e >= 0 && e < nz) {
        const int cell = nv + e / NG, at = cell * GS + e % NG;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            img[r * ld + at] = zx[r];
            top[r] = max(top[r], (uint32_t)__double2hiint(zx[r]) & 0x7ff00000u);
            zsq[r] = zx[r] * zx[r];
        }
    }
    // the coupling moments (cell 0's thread: t_0 = q = u_b . g_b)
    double *mom = core + 2 * NG * R;  // [R][2]: alpha sx, q / sx
    if (m == 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double alpha = 0.0;
#pragma unroll
            for (int i = 0; i < NG; ++i) alpha = fma(__ldg(v0 + i), g[r][i], alpha);
            const double a_sx = alpha * sx, q_sx = t_m[r] / sx;
            if (!isfinite(a_sx) || !isfinite(q_sx)) top[r] = 0x7ff00000u;
            mom[2 * r] = a_sx;
            mom[2 * r + 1] = q_sx;
        }
    }
    // block maximum and sums of squares (8 warps at most)
    __syncthreads();  // red[] reused
    double *rsum = red;
    uint32_t *rtop = reinterpret_cast<uint32_t *>(red + 8 * 2 * R);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t t = __reduce_max_sync(0xffffffffu, top[r]);
        const double xs = warp_sum(xsq[r]), zs = warp_sum(zsq[r]);
        if (lane == 0) {
            rsum[(wid * R + r) * 2] = xs;
            rsum[(wid * R + r) * 2 + 1] = zs;
            rtop[wid * R + r] = t;
        }
    }
    __syncthreads();
    double *scl = mom + 2 * R;  // [R]: the rows' scales 2^(bits - e)
    if (tid < R) {
        const int r = tid;
        uint32_t t = 0u;
        double xs = 0.0, zs = 0.0;
        for (int w = 0; w < nwarp; ++w) {
            t = max(t, rtop[w * R + r]);
            xs += rsum[(w * R + r) * 2];
            zs += rsum[(w * R + r) * 2 + 1];
        }
        // every |x| < 2^ex; a row below the normal range counts as zero
        const bool bad = t == 0x7ff00000u, some = t != 0u && !bad;
        const int ex = some ? (int)(t >> 20) - 1022 : 0;
        scl[r] = some ? ldexp(1.0, a.bits - ex) : 0.0;
        // a non-finite row gets a NaN scale: its residues are zero and every
        // entry it reaches is NaN, which the contraction reports
        a.rowscale[grow + r] =
            bad ? __longlong_as_double(0x7ff8000000000000LL) : (some ? ldexp(1.0, ex - a.bits) : 0.0);
        const double *g0 = core + r * 2 * NG, *gg0 = g0 + NG;
        double n1 = 0.0, n2 = 0.0, gg = 0.0;
#pragma unroll
        for (int i = 0; i < NG; ++i) {
            n1 = fma(g0[i], g0[i], n1);
            n2 = fma(gg0[i], gg0[i], n2);
            gg = fma(g0[i], gg0[i], gg);
        }
        const double a_sx = mom[2 * r], q_sx = mom[2 * r + 1];
        double *lf = a.left + (grow + r) * a.cwp, *rt = a.right + (grow + r) * a.cwp;
        lf[NG] = rt[NG + 1] = a_sx;
        lf[NG + 1] = rt[NG] = q_sx;
        for (int i = NG + 2; i < a.cwp; ++i) lf[i] = rt[i] = 0.0;
        write_row_record(a.cbound + (grow + r) * CB_STRIDE, some ? 1.0 : 0.0, ex, n1, n2, a_sx, q_sx, xs, zs, gg);
    }
    __syncthreads();
    // residues: item = (row, four columns)
    const int words = (int)(a.kpad / 4);
    for (int it = tid; it < R * words; it += blockDim.x) {
        const int r = it / words, c0 = (it - r * words) * 4;
        const double scale = scl[r];
        const double *x = img + r * ld + GS;
        const int zlive = scale != 0.0 ? zend : 0;
        float l0[4], l1[4], l2[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int c = c0 + s;
            // the scaled value rounded to an integer of at most bits + 1 bits: the low bits of the sum;
            // a zero scale (an empty or non-finite row) gives zero
            const double v = c < zlive ? x[GS == NG ? c : c + c / NG] : 0.0;
            const double y = __fma_rn(v, scale, 6755399441055744.0);  // 1.5 * 2^52
            const uint32_t lo = (uint32_t)__double2loint(y), hi = (uint32_t)__double2hiint(y);
            l0[s] = __fadd_rn(__uint_as_float((lo & 0x3fffu) | 0x4b000000u), -8388608.0f);
            l1[s] = __fadd_rn(__uint_as_float(((lo >> 14) & 0x3fffu) | 0x4b000000u), -8388608.0f);
            // (hi : lo) >> 28, signed: the sum's exponent and leading bit are 0x43380000 in hi
            l2[s] = __fadd_rn(__uint_as_float(__funnelshift_r(lo, hi, 28) + (0x4b400000u - 0x33800000u)), -12582912.0f);
        }
        signed char *pa = a.resA + (grow + r) * a.kpad + c0;
        const long slab = a.nrows_total * a.kpad;
        auto residues = [&](int md, float (&t)[4]) {
            const float4 v = f.mod[md];  // m, 1/m, 2^14 mod m, 2^28 mod m
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                // |u| < 2^22: exact; the quotient rounds to the nearest integer (or either, at a tie of an even m)
                const float u = __fmaf_rn(l2[s], v.w, __fmaf_rn(l1[s], v.z, l0[s]));
                const float qf = __fadd_rn(__fmaf_rn(u, v.y, 12582912.0f), -12582912.0f);
                t[s] = __fmaf_rn(-qf, v.x, u);  // in [-128, 128]
            }
        };
        auto byte = [](float t) { return __float_as_uint(__fadd_rn(t, 12582912.0f)); };  // in the low eight bits
        auto word = [&](const float (&t)[4]) {
            return __byte_perm(__byte_perm(byte(t[0]), byte(t[1]), 0x0040), __byte_perm(byte(t[2]), byte(t[3]), 0x0040),
                               0x5410);
        };
        if (!a.resB || c0 < a.b_col0 || c0 >= a.b_col0 + a.b_ld) {
#pragma unroll 2
            for (int md = 0; md < a.n_mod; ++md, pa += slab) {
                float t[4];
                residues(md, t);
                *reinterpret_cast<uint32_t *>(pa) = word(t);
            }
        } else {
            signed char *pb = a.resB + (grow + r) * a.b_ld + (c0 - a.b_col0);
            const long slab_b = a.nrows_total * a.b_ld;
#pragma unroll 1
            for (int md = 0; md < a.n_mod; ++md, pa += slab, pb += slab_b) {
                float t[4];
                residues(md, t);
                *reinterpret_cast<uint32_t *>(pa) = word(t);
#pragma unroll
                for (int s = 0; s < 4; ++s)  // B holds the residues of -z
                    if (c0 + s >= kbody) t[s] = -t[s];
                *reinterpret_cast<uint32_t *>(pb) = word(t);
            }
        }
    }
}

template <int NG, int R>
__global__ void __launch_bounds__(256, 2) split_rows_cell_kernel(const __grid_constant__ RowsArgs a,
                                                              const __grid_constant__ ResidueArgs f,
                                                              const double *__restrict__ ktab_t,
                                                              const long *__restrict__ koff_t, int zmax) {
    extern __shared__ __align__(16) double sm[];
    double *img = sm;                                          // [R][cell_image]
    double *red = sm + R * cell_image(NG, a.nv, zmax);           // block scratch (cell_scratch doubles)
    const long q0 = (long)blockIdx.x * R;
    if (R == 1) {
        cell_rows_body<NG, 1>(a, f, ktab_t, koff_t, q0, zmax, img, red);
        return;
    }
    bool same = q0 + R <= a.nrows;
    for (int r = 1; same && r < R; ++r) same = a.row_k[q0 + r] == a.row_k[q0];
    if (same) {
        cell_rows_body<NG, R>(a, f, ktab_t, koff_t, q0, zmax, img, red);
        return;
    }
    // the last rows, and rows at a change of multipole: one at a time
    for (long q = q0; q < a.nrows && q < q0 + R; ++q) {
        cell_rows_body<NG, 1>(a, f, ktab_t, koff_t, q, zmax, img, red);
        __syncthreads();
    }
}
// doubles of block scratch: warp sums and maxima, the core vectors and moments, the scales
constexpr int cell_scratch(int ng, int rows) { return rows * (8 * 4 + 2 * ng + 2 + 1); }

// =========================================================================
// K3s — tcgen05 INT8 residue SYRK with CRT epilogue
// =========================================================================
constexpr int BM = 128, BN = 128, BKB = 128;  // tile rows, tile cols, K bytes per stage
constexpr int STAGES = 5;
constexpr int STAGE_BYTES = (BM + BN) * BKB;  // 32 KB
constexpr int EPI_WARPS = 16;                 // 4 TMEM lane quarters x 4 column groups
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);  // columns per epilogue thread
constexpr int CTL_WARPS = 4;                  // one warpgroup: TMA, MMA, tile records (rows, columns)
constexpr int THREADS = 32 * (CTL_WARPS + EPI_WARPS);
// 640 threads launch with 96 registers each; the control warpgroup keeps 32, which
// gives the four epilogue warpgroups 112 (4 x 112 + 32 = 5 x 96).
constexpr int CTL_REGS = 32, EPI_REGS = 112;
constexpr int NACC = 2;     // int32 accumulator tiles in TMEM (128 columns each; the rest parks digits 0 and 1)
constexpr int NDIG = 3;     // CRT digits, of up to four moduli each
constexpr int FC = 8;       // columns per chunk of the final phase
constexpr int STG_LD = FC + 1;  // doubles per staged row
constexpr int LOW_WORDS = EPI_WARPS * EPI_COLS / 4 * 32;  // the fractions' lowest bytes, four columns a word
// What the epilogue needs to know of a tile, fetched ahead of it by two control warps.
struct __align__(16) TileInfo {
    double rs_row[BM], rs_col[BN];         // row scales
    double row_max[4][3], col_max[4][3];   // screen bounds of each 32-row / 32-column group
    double *out;                           // the tile's table
    long row0;
    int n, ti, tj, pad;
};
constexpr size_t SMEM_BYTES = 1024 /*align slack*/ + (size_t)STAGES * STAGE_BYTES +
                              (size_t)EPI_WARPS * 32 * STG_LD * sizeof(double) + 2 * sizeof(TileInfo) +
                              LOW_WORDS * sizeof(uint32_t) + 256 /*barriers*/;
constexpr long long WAIT_LIMIT = 4000000000LL;  // clock64 ticks (~2 s)
constexpr uint32_t IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

struct CrtArgs {
    const double *rowscale, *left, *right, *cbound;
    double corr_floor;  // skip the FP64 core correction of a warp block when its bound is below this
    int cwp, cw;
    const long *grp_row0, *grp_n, *grp_kdim, *grp_out;
    const int *grp_zc;  // first 128-column chunk that B holds for itself (null: all)
    const int *tasks;
    long n_tasks, nrows_total;
    double *out;
    int *status;
    int n_mod;
    // The CRT in two steps. Consecutive moduli (up to dig_end[g]) make a digit modulo
    // D_g < 2^32: d_g = sum_i x_i coef_i mod D_g. Then x / M = sum_g d_g F_g mod 1 with
    // F_g = f_hi 2^-32 + f_mid 2^-64 + f_lo 2^-96 + f_end 2^-112 (f_end of 16 bits).
    int dig_end[NDIG], coef[MAXMOD], D[NDIG], f_hi[NDIG], f_mid[NDIG], f_lo[NDIG], f_end[NDIG];
    double inv_D[NDIG], inv_D32[NDIG];  // 1/D, 2^32/D
    double M;  // the product of the moduli, times 2^-32
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false (and status = ETIMEDOUT) after WAIT_LIMIT clock ticks, or as soon as
// another wait has given up.  RKB_ENONFINITE in the status word ends no wait.
__device__ __forceinline__ bool mbar_wait_slow(uint64_t *bar, uint32_t parity, int *status) {
    const long long t0 = clock64();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 8; ++i)  // the status word is an L2 read: looked at between tries only
            if (mbar_try(bar, parity)) return true;
        if (*(volatile int *)status == (int)RKB_ETIMEDOUT) return false;
        if (clock64() - t0 > WAIT_LIMIT) {
            atomicExch(status, (int)RKB_ETIMEDOUT);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *status) {
    if (mbar_try(bar, parity)) return true;
    return mbar_wait_slow(bar, parity, status);
}
// The same by a whole warp, with one outcome for all its lanes: what follows a wait (shuffles,
// .aligned instructions) wants every lane.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, int *status) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, status));
}
// After a failure: wait for what is still in flight, whatever the status, with the same limit.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try(bar, parity) && clock64() - t0 <= WAIT_LIMIT) {}
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tma_load(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);   // start address (16-byte units)
    d |= (uint64_t)1u << 16;                   // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024u >> 4) << 32;         // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1u << 46;                   // descriptor version for sm_100
    d |= (uint64_t)2u << 61;                   // SWIZZLE_128B
    return d;
}
__device__ __forceinline__ void mma_i8(uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(dtmem),
        "l"(ad), "l"(bd), "r"(IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, int (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const int (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3])
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const int (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Exact int -> double by the 2^52 trick (ALU and FP64 pipes; cvt runs at a quarter of their rate).
__device__ __forceinline__ double int_to_double(int v) {
    return __dadd_rn(__hiloint2double(0x43300000, (int)((uint32_t)v ^ 0x80000000u)),
                     -(4503599627370496.0 + 2147483648.0));
}
__device__ __forceinline__ double uint_to_double(uint32_t v) {
    return __dadd_rn(__hiloint2double(0x43300000, (int)v), -4503599627370496.0);
}
// 2^8 v plus a byte
__device__ __forceinline__ double uint40_to_double(uint32_t v, uint32_t byte) {
    return __dadd_rn(__hiloint2double((int)(0x43300000u | (v >> 24)), (int)((v << 8) | byte)), -4503599627370496.0);
}
// acc mod D nearest zero. |acc| < 2^59 and D < 2^32, so the quotient's rounding error is
// far below 1 and |result| <= D/2 (1 + 2^-25).
__device__ __forceinline__ int mod_near(long long acc, int D, double inv_D, double inv_D32) {
    const double q = __fma_rn(int_to_double((int)(acc >> 32)), inv_D32, __dmul_rn(uint_to_double((uint32_t)acc), inv_D));
    return (int)((uint32_t)acc - (uint32_t)__double2loint(__dadd_rn(q, 6755399441055744.0)) * (uint32_t)D);
}

__global__ void __launch_bounds__(THREADS, 1)
    crt_syrk_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                    const __grid_constant__ CrtArgs p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *ring = base;
    double *stage_out = (double *)(ring + (size_t)STAGES * STAGE_BYTES);
    TileInfo *info = (TileInfo *)(stage_out + EPI_WARPS * 32 * STG_LD);
    uint32_t *low_all = (uint32_t *)(info + 2);
    uint64_t *bars = (uint64_t *)(low_all + LOW_WORDS);
    uint64_t *full = bars, *empty = full + STAGES, *accf = empty + STAGES, *acce = accf + NACC;
    uint64_t *inff = acce + NACC, *infe = inff + 2, *drain = infe + 2;
    uint32_t *tmem_slot = (uint32_t *)(drain + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < NACC; ++b) {
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], EPI_WARPS);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&inff[b], 2);
            mbar_init(&infe[b], EPI_WARPS);
        }
        mbar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    int *status = p.status;
    const int n_mod = p.n_mod;

    if (warp < CTL_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CTL_REGS));
        if (warp == 0) {
            // -------------------------------------------------------- TMA producer
            if (lane == 0) {
                uint32_t it = 0;
                bool ok = true;
                for (long t = blockIdx.x; t < p.n_tasks && ok; t += gridDim.x) {
                    const int g = p.tasks[3 * t], ti = p.tasks[3 * t + 1], tj = p.tasks[3 * t + 2];
                    const long row0 = p.grp_row0[g];
                    const int nk = (int)(p.grp_kdim[g] / BKB), zc = p.grp_zc ? p.grp_zc[g] : 0;
                    for (int md = 0; md < n_mod && ok; ++md) {
                        const int ya = (int)(md * p.nrows_total + row0 + (long)ti * BM);
                        const int yb = (int)(md * p.nrows_total + row0 + (long)tj * BN);
                        for (int kc = 0; kc < nk; ++kc, ++it) {
                            const int s = it % STAGES;
                            const uint32_t ph = (it / STAGES) & 1u;
                            if (!mbar_wait(&empty[s], ph ^ 1u, status)) { ok = false; break; }
                            unsigned char *sa = ring + (size_t)s * STAGE_BYTES;
                            mbar_expect_tx(&full[s], STAGE_BYTES);
                            tma_load(sa, &mapA, kc * BKB, ya, &full[s]);
                            if (kc < zc) tma_load(sa + BM * BKB, &mapA, kc * BKB, yb, &full[s]);
                            else tma_load(sa + BM * BKB, &mapB, (kc - zc) * BKB, yb, &full[s]);
                        }
                    }
                }
                // given up: the loads of the last STAGES steps may still be under way
                if (!ok)
                    for (uint32_t i = it > STAGES ? it - STAGES : 0u; i < it; ++i)
                        mbar_drain(&full[i % STAGES], (i / STAGES) & 1u);
            }
        } else if (warp == 1) {
            // -------------------------------------------------------- MMA issuer
            if (lane == 0) {
                uint32_t it = 0, buf = 0, aph = 0;  // accumulator buffer and its phase
                bool ok = true;
                for (long t = blockIdx.x; t < p.n_tasks && ok; t += gridDim.x) {
                    const int nk = (int)(p.grp_kdim[p.tasks[3 * t]] / BKB);
                    for (int md = 0; md < n_mod && ok; ++md) {
                        if (!mbar_wait(&acce[buf], aph ^ 1u, status)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t dt = tmem + buf * (uint32_t)BN;
                        for (int kc = 0; kc < nk; ++kc, ++it) {
                            const int s = it % STAGES;
                            const uint32_t ph = (it / STAGES) & 1u;
                            if (!mbar_wait(&full[s], ph, status)) { ok = false; break; }
                            tc_fence_after();
                            const uint32_t sa = smem_u32(ring + (size_t)s * STAGE_BYTES);
                            const uint64_t ad = sw128_desc(sa), bd = sw128_desc(sa + BM * BKB);
#pragma unroll
                            for (int kk = 0; kk < BKB / 32; ++kk)
                                mma_i8(dt, ad + (uint64_t)(2 * kk), bd + (uint64_t)(2 * kk), (kc | kk) != 0 ? 1u : 0u);
                            mma_commit(&empty[s]);
                        }
                        if (ok) mma_commit(&accf[buf]);
                        if (++buf == NACC) { buf = 0; aph ^= 1u; }
                    }
                }
                if (!ok) {  // given up: wait for the MMAs issued
                    mma_commit(drain);
                    mbar_drain(drain, 0);
                }
            }
        } else {
            // -------------------------------------------------------- tile records: warp 2 rows, warp 3 columns
            const bool rows = warp == 2;
            uint32_t buf = 0, ph = 0;
            for (long t = blockIdx.x; t < p.n_tasks; t += gridDim.x) {
                const int g = p.tasks[3 * t], ti = p.tasks[3 * t + 1], tj = p.tasks[3 * t + 2];
                const long row0 = p.grp_row0[g];
                const int n = (int)p.grp_n[g];
                if (!mbar_wait_warp(&infe[buf], ph ^ 1u, status)) break;
                TileInfo &I = info[buf];
                double *rs = rows ? I.rs_row : I.rs_col, *mx = rows ? I.row_max[0] : I.col_max[0];
                int i = (rows ? ti : tj) * BM + lane;
#pragma unroll 1
                for (int q = 0; q < 4; ++q, i += 32, mx += 3) {
                    const bool in = i < n;
                    rs[32 * q + lane] = in ? __ldg(p.rowscale + row0 + i) * (rows ? p.M : 1.0) : 0.0;
#pragma unroll 1
                    for (int v = 0; v < 3; ++v) {  // |g0| or |G00 g0|, |alpha sx|, |q/sx|
                        const int f = v ? v + 1 : !rows;
                        double m = in ? __ldg(p.cbound + (row0 + i) * CB_STRIDE + f) : 0.0;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
                        if (lane == 0) mx[v] = m;
                    }
                }
                if (rows && lane == 0) {
                    I.out = p.out + p.grp_out[g];
                    I.row0 = row0;
                    I.n = n;
                    I.ti = ti;
                    I.tj = tj;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&inff[buf]);
                if ((buf ^= 1u) == 0u) ph ^= 1u;
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
        const int ew = warp - CTL_WARPS;
        const int quarter = warp & 3;       // TMEM lane quarter this warp may access
        const int cgrp = ew >> 2;           // column group of the tile
        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cgrp * EPI_COLS);
        double *stg = stage_out + (size_t)ew * 32 * STG_LD;
        const int tiles = (int)((p.n_tasks - blockIdx.x + gridDim.x - 1) / gridDim.x);
        // x / M mod 1 of this thread's row: words of 2^-64 and, BN columns on, of 2^-32 in TMEM, and the
        // bytes of 2^-72 of four columns in a word of shared memory that no other thread touches
        const uint32_t park = tbase + (uint32_t)(NACC * BN);
        uint32_t *low = low_all + ew * (EPI_COLS / 4 * 32) + lane;
        double *row = stg + lane * STG_LD;
        // One chunk of FC columns of a finished tile: scaling, correction and stores.
        auto finish = [&](const TileInfo &I, int c) {
            const int a0 = I.ti * BM + quarter * 32, bc = I.tj * BN + cgrp * EPI_COLS + c, a = a0 + lane;
            const double rs_a = I.rs_row[quarter * 32 + lane];  // with M folded in
            const double *rs_b = I.rs_col + cgrp * EPI_COLS + c;
            tmem_wait_st();
#pragma unroll
            for (int h = 0; h < FC; h += 4) {
                int lo[4], hi[4];
                tmem_ld4(park + (uint32_t)(c + h), lo);
                tmem_ld4(park + (uint32_t)(BN + c + h), hi);
                const uint32_t bytes = low[(c + h) * 8];
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    row[h + j] = __fma_rn(uint40_to_double((uint32_t)lo[j], (bytes >> (8 * j)) & 0xffu), 0x1p-40,
                                          int_to_double(hi[j])) * (rs_a * rs_b[h + j]);
            }
            // Correction screen for this warp's 32 x EPI_COLS block: with per-row bounds
            // relative to each row's scale, |left_a . right_b| <= 2^(e_a+e_b) *
            // (|g0_a| |G00 g0_b| + |alpha_a sx| |q_b/sx| + |q_a/sx| |alpha_b sx|).
            // Below corr_floor the term is far under the split's own error and is skipped.
            const double *rm = I.row_max[quarter], *cm = I.col_max[cgrp];
            const int n = I.n;
            if (!(rm[0] * cm[0] + rm[1] * cm[2] + rm[2] * cm[1] <= p.corr_floor) && a < n) {
                const double *la = p.left + (I.row0 + a) * p.cwp;
                const double *rb = p.right + (I.row0 + bc) * p.cwp;
#pragma unroll 1
                for (int j = 0; j < min(FC, n - bc); ++j, rb += p.cwp) {
                    double corr = 0.0;
#pragma unroll 2
                    for (int i = 0; i < p.cw; ++i) corr = fma(__ldg(la + i), __ldg(rb + i), corr);
                    row[j] += corr;
                }
            }
            __syncwarp();
            uint32_t top = 0u;  // largest exponent field of this thread's entries
            const int sub = lane / FC, col = lane % FC;
            const double *seg = stg + sub * STG_LD + col;
            if (a0 + 32 <= n && bc + FC <= n) {
                // the transposed tile: lanes hold consecutive a, 256 contiguous bytes a store;
                // the tile itself: row segments of FC columns, 32 / FC rows a store
                double *T = I.out + (long)bc * n + a, *R = I.out + (long)(a0 + sub) * n + bc + col;
                const bool mirror = I.ti != I.tj;
#pragma unroll
                for (int j = 0; j < FC; ++j, T += n) {
                    const double v = row[j];
                    top = max(top, (uint32_t)__double2hiint(v) & 0x7ff00000u);
                    if (mirror) *T = v;
                }
#pragma unroll
                for (int rr = 0; rr < 32; rr += 32 / FC, R += (long)(32 / FC) * n) *R = seg[rr * STG_LD];
            } else {
#pragma unroll 1
                for (int j = 0; j < FC; ++j)
                    if (a < n && bc + j < n) {
                        const double v = row[j];
                        top = max(top, (uint32_t)__double2hiint(v) & 0x7ff00000u);
                        if (I.ti != I.tj) I.out[(long)(bc + j) * n + a] = v;
                    }
#pragma unroll 1
                for (int rr = 0; rr < 32; rr += 32 / FC)
                    if (a0 + rr + sub < n && bc + col < n)
                        I.out[(long)(a0 + rr + sub) * n + bc + col] = seg[rr * STG_LD];
            }
            if (top == 0x7ff00000u) atomicCAS(status, 0, (int)RKB_ENONFINITE);
            __syncwarp();
        };
        uint32_t it = 0;  // accumulators taken
        bool ok = true;
#pragma unroll 1
        for (int k = 0; k < tiles; ++k) {
            // The chunks of the tile before wait for the first digit of this one, in whose
            // shadow (the MMAs run on) they are finished.
            int late = k ? 0 : EPI_COLS;
            if (k && !mbar_wait_warp(&inff[(k - 1) & 1], (uint32_t)((k - 1) >> 1) & 1u, status)) { ok = false; break; }
#pragma unroll 1
            for (int dg = 0, md = 0; dg < NDIG; ++dg) {
                long long acc[EPI_COLS];  // the open digit's sum
#pragma unroll
                for (int c = 0; c < EPI_COLS; ++c) acc[c] = 0;
                const int end = p.dig_end[dg];
#pragma unroll 1
                for (; md < end; ++md, ++it) {
                    if (!mbar_wait_warp(&accf[it & 1u], (it >> 1) & 1u, status)) { ok = false; break; }
                    tc_fence_after();
                    const int coef = p.coef[md];
                    const uint32_t src = tbase + (it & 1u) * (uint32_t)BN;
#pragma unroll
                    for (int c = 0; c < EPI_COLS; c += 8) {
                        int v[8];
                        tmem_ld8(src + (uint32_t)c, v);
                        tmem_wait_ld();
                        if (c + 8 == EPI_COLS) {  // the accumulator is read: the next modulus may overwrite it
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&acce[it & 1u]);
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[c + j] += (long long)v[j] * coef;
                    }
                    if (late < EPI_COLS) {
                        finish(info[(k - 1) & 1], late);
                        late += FC;
                    }
                }
                if (!ok) break;
                if (dg == 0 && k) {
#pragma unroll 1
                    for (; late < EPI_COLS; late += FC) finish(info[(k - 1) & 1], late);
                    if (lane == 0) mbar_arrive(&infe[(k - 1) & 1]);
                }
                // f += d F mod 1, rounded to 2^-72
                const int D = p.D[dg], fh = p.f_hi[dg], fm = p.f_mid[dg], fl = p.f_lo[dg], fe = p.f_end[dg];
                const double inv_D = p.inv_D[dg], inv_D32 = p.inv_D32[dg];
                tmem_wait_st();
#pragma unroll
                for (int c = 0; c < EPI_COLS; c += 4) {
                    int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
                    uint32_t bytes = 0u, t[4];
                    if (dg) {
                        tmem_ld4(park + (uint32_t)c, lo);
                        tmem_ld4(park + (uint32_t)(BN + c), hi);
                        bytes = low[c * 8];
                        tmem_wait_ld();
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int d = mod_near(acc[c + j], D, inv_D, inv_D32);
                        // units of 2^-96: the byte so far in bits 24..31, half a unit of it below; the product
                        // with the weight's end needs d to 16 bits only (off by 2^-81)
                        long long e = (long long)(d >> 16) * fe + __byte_perm(bytes, 0x00800000u, 0x0644u | (j << 12));
                        e += (long long)d * fl;
                        long long f = ((long long)hi[j] << 32) | (uint32_t)lo[j];
                        f += (long long)d * fm + ((long long)((uint32_t)d * (uint32_t)fh) << 32) + (e >> 32);
                        lo[j] = (int)f;
                        hi[j] = (int)(f >> 32);
                        t[j] = (uint32_t)e;
                    }
                    tmem_st4(park + (uint32_t)c, lo);
                    tmem_st4(park + (uint32_t)(BN + c), hi);
                    low[c * 8] = __byte_perm(__byte_perm(t[0], t[1], 0x0073), __byte_perm(t[2], t[3], 0x0073), 0x5410);
                }
            }
            if (!ok) break;
        }
        if (ok && tiles > 0 && mbar_wait_warp(&inff[(tiles - 1) & 1], (uint32_t)((tiles - 1) >> 1) & 1u, status)) {
#pragma unroll 1
            for (int c = 0; c < EPI_COLS; c += FC) finish(info[(tiles - 1) & 1], c);
        }
        tmem_wait_st();
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ------------------------------------------------------------- host helpers
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)f;
    }
    return fn;
}

static int inverse_mod(int a, int m) {  // a and m coprime, m >= 2 (extended Euclid)
    int r0 = m, r1 = a % m, t0 = 0, t1 = 1;
    while (r1 > 1) {
        const int q = r0 / r1, r2 = r0 - q * r1, t2 = t0 - q * t1;
        r0 = r1, r1 = r2, t0 = t1, t1 = t2;
    }
    return t1 < 0 ? t1 + m : t1;
}

// The CRT constants of the contraction (CrtArgs); 4..MAXMOD pairwise coprime moduli in [2, 256].
static int crt_weights(const int *moduli, int n_mod, CrtArgs &p) {
    RKB_CHECK_ARG(n_mod >= 4 && n_mod <= MAXMOD, "split contraction takes 4..%d moduli (got %d)", MAXMOD, n_mod);
    for (int i = 0; i < n_mod; ++i) {
        RKB_CHECK_ARG(moduli[i] >= 2 && moduli[i] <= 256, "moduli must lie in [2, 256]");
        for (int j = 0; j < i; ++j)
            RKB_CHECK_ARG(std::gcd(moduli[j], moduli[i]) == 1, "moduli %d and %d have a common factor", moduli[j],
                          moduli[i]);
    }
    const __int128 one = (__int128)1 << 126;
    for (int g = 0, i0 = 0; g < NDIG; ++g) {
        const int i1 = i0 + (n_mod - i0 + NDIG - g - 1) / (NDIG - g);  // 4 to 12 moduli in three even parts
        unsigned long long D = 1, c = 0;
        for (int i = i0; i < i1; ++i) D *= moduli[i];
        for (int i = i0; i < i1; ++i) {
            // coef_i = (D/m_i) ((D/m_i)^-1 mod m_i), nearest zero: 1 mod m_i, 0 mod the digit's others
            const int m = moduli[i];
            const unsigned long long r = D / m, e = r * inverse_mod((int)(r % m), m) % D;
            p.coef[i] = (int)(2 * e >= D ? (long long)e - (long long)D : (long long)e);
            int rest = 1 % m;  // M/D mod m
            for (int j = 0; j < n_mod; ++j)
                if (j < i0 || j >= i1) rest = rest * (moduli[j] % m) % m;
            c = (c + e * inverse_mod(rest, m)) % D;
        }
        // F = ((M/D)^-1 mod D) / D in [-1/2, 1/2)
        const __int128 cs = 2 * c >= D ? (__int128)c - (__int128)D : (__int128)c, Ds = (__int128)D;
        const __int128 f = one / Ds * cs + one % Ds * cs / Ds;
        // 112 bits; every word but the first is read as signed
        const __int128 v = (f + ((__int128)1 << 13)) >> 14;
        p.f_end[g] = (int)(int16_t)(uint16_t)v;
        const __int128 w = (v - p.f_end[g]) >> 16;
        p.f_lo[g] = (int)(uint32_t)w;
        const uint64_t t = (uint64_t)(w >> 32) + ((uint32_t)w >> 31);
        p.f_mid[g] = (int)(uint32_t)t;
        p.f_hi[g] = (int)((uint32_t)(t >> 32) + ((uint32_t)t >> 31));
        p.D[g] = (int)(uint32_t)D;
        p.inv_D[g] = 1.0 / (double)D;
        p.inv_D32[g] = 4294967296.0 / (double)D;
        p.dig_end[g] = i0 = i1;
    }
    return RKB_OK;
}

static int make_map(CUtensorMap *map, const void *ptr, long kpad, long rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) {
        set_error("cuTensorMapEncodeTiled is unavailable from the CUDA driver");
        return RKB_EUNSUPPORTED;
    }
    cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)kpad};
    cuuint32_t box[2] = {(cuuint32_t)BKB, (cuuint32_t)BM};
    cuuint32_t es[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d) for a %ld x %ld residue matrix", (int)r, rows, kpad);
        return RKB_EINVAL;
    }
    return RKB_OK;
}

}  // namespace split
}  // namespace rkb

using namespace rkb;
using namespace rkb::split;

extern "C" int rkb_split_rows(const double *d_Pv, const double *d_Qv, long orb_ld, const long *d_pairs,
                              const long *d_row_pair, const int *d_row_k, long nrows, const double *d_w, int nv,
                              int ng, const double *d_ktab, const long *d_koff, int bits, int n_mod,
                              const int *moduli, signed char *d_resA, signed char *d_resB, long kpad,
                              long row_base, long nrows_total, double *d_rowscale, double *d_left,
                              double *d_right, double *d_cbound, int cwp, double *d_xwork,
                              const int *d_zcount, void *stream) {
    RKB_CHECK_ARG(nv >= 2 && ng >= 1 && ng <= RKB_MAX_NG, "invalid grid (nv=%d, ng=%d)", nv, ng);
    RKB_CHECK_ARG(bits >= 8 && bits <= 50, "bits must be in [8, 50] (got %d)", bits);
    RKB_CHECK_ARG(n_mod >= 1 && n_mod <= MAXMOD, "1..%d moduli supported (got %d)", MAXMOD, n_mod);
    RKB_CHECK_ARG(kpad % BKB == 0 && kpad >= (long)(nv - 1) * ng, "kpad must be a multiple of %d >= body width",
                  BKB);
    RKB_CHECK_ARG(cwp >= ng + 2, "correction width must be >= ng + 2");
    RKB_CHECK_ARG(d_cbound != nullptr, "the correction-bound array is required");
    RKB_CHECK_ARG(row_base >= 0 && row_base + nrows <= nrows_total, "row range outside the residue matrices");
    if (nrows == 0) return RKB_OK;
    RowsArgs a;
    a.P = d_Pv; a.Q = d_Qv; a.orb_ld = orb_ld; a.pairs = d_pairs; a.row_pair = d_row_pair; a.row_k = d_row_k;
    a.nrows = nrows; a.w = d_w; a.nv = nv; a.ng = ng; a.ktab = d_ktab; a.koff = d_koff; a.bits = bits;
    a.n_mod = n_mod;
    for (int i = 0; i < MAXMOD; ++i) {
        const int m = i < n_mod ? moduli[i] : 256;
        RKB_CHECK_ARG(m >= 2 && m <= 256, "moduli must lie in [2, 256]");
        a.mod[i] = m;
        a.magic[i] = (uint32_t)((1ULL << 32) / (unsigned long long)m + 1ULL);
        a.c20[i] = (uint32_t)((1u << 20) % (uint32_t)m);
        a.bias[i] = (uint32_t)m << 20;  // hi + bias >= 0 for |hi| <= 2^20
        a.inv_mod[i] = 1.0 / (double)m;
    }
    a.resA = d_resA; a.resB = d_resB; a.kpad = kpad; a.row_base = row_base; a.nrows_total = nrows_total;
    a.rowscale = d_rowscale; a.left = d_left; a.right = d_right; a.cbound = d_cbound; a.cwp = cwp;
    a.xwork = d_xwork;
    RKB_CHECK_ARG(d_xwork != nullptr && d_zcount != nullptr, "the row workspace and Z counts are required");
    RKB_CHECK_ARG(bits <= 40, "the residue path handles |x| <= 2^40 (bits <= 40)");
    RKB_CHECK_ARG(kpad % 16 == 0, "kpad must be a multiple of 16");
    const long np = ((long)nv * ng + 1) & ~1L, nvp = ((long)nv + 1) & ~1L;
    const size_t per_warp = (size_t)(np + nvp) * sizeof(double);
    const int warps = 4;
    size_t smem = (size_t)warps * per_warp;
    RKB_CHECK_ARG(smem <= 200 * 1024, "grid too large for the split row kernel");
    dim3 grid((unsigned)ceil_div(nrows, warps)), block(32 * warps);
    cudaStream_t st = as_stream(stream);
    RKB_CHECK_ARG(((uintptr_t)d_resA % 16) == 0 && (d_resB == nullptr || ((uintptr_t)d_resB % 16) == 0),
                  "residue buffers must be 16-byte aligned");
#define RKB_SR_CASE(NGV)                                                                              \
    case NGV: {                                                                                       \
        RKB_CUDA(set_smem(split_rows_kernel<NGV>, (int)smem));                                         \
        split_rows_kernel<NGV><<<grid, block, smem, st>>>(a);                                         \
        break;                                                                                        \
    }
    switch (ng) {
        RKB_SR_CASE(5) RKB_SR_CASE(7) RKB_SR_CASE(8) RKB_SR_CASE(9) RKB_SR_CASE(11)
        default: {
            RKB_CUDA(set_smem(split_rows_kernel<0>, (int)smem));
            split_rows_kernel<0><<<grid, block, smem, st>>>(a);
        }
    }
#undef RKB_SR_CASE
    RKB_LAUNCHED("split_rows_kernel");
    const long nthreads = nrows * (kpad / 16);
    split_residues_kernel<<<(unsigned)ceil_div(nthreads, 256), 256, 0, st>>>(a, d_zcount);
    RKB_LAUNCHED("split_residues_kernel");
    return RKB_OK;
}

// Rows up to which a block takes one: with R at a time fewer blocks than SMs are left, and blocks at
// a change of multipole take their rows one after another.  R rows and one row a block in us: ng = 8
// (R = 4, 105 cells) 114 rows 36 and 17, 801 rows 38 and 28, 1 656 rows 38 and 38, 3 114 rows 56 and
// 63; ng = 11 (R = 2, 142 cells) 32 and 21, 36 and 36, 52 and 59, 89 and 96.
static long cell_single(int ng) { return 2L * cell_rows(ng) * sm_count(); }

extern "C" int rkb_split_rows_cells_z(const double *d_Pv, const double *d_Qv, long orb_ld, const long *d_pairs,
                                      const long *d_row_pair, const int *d_row_k, long nrows, const double *d_w,
                                      int nv, int ng, const double *d_ktab, const long *d_koff,
                                      const double *d_ktab_t, const long *d_koff_t, int max_z, int bits,
                                      int n_mod, const int *moduli, signed char *d_resA, signed char *d_resB,
                                      long kpad, long b_col0, long b_ld, long row_base, long nrows_total,
                                      double *d_rowscale, double *d_left, double *d_right, double *d_cbound, int cwp,
                                      void *stream) {
    RKB_CHECK_ARG(nv >= 2 && ng >= 5 && ng <= 11, "the cell row kernel takes 5 <= ng <= 11 (got %d)", ng);
    RKB_CHECK_ARG(max_z >= 0 && max_z <= CELL_ZMAX, "the cell row kernel takes <= %d Z columns (got %d)", CELL_ZMAX,
                  max_z);
    const long threads = ((long)nv + max_z + 31) / 32 * 32;
    RKB_CHECK_ARG(threads <= 256, "grid too long for the cell row kernel (%d cells + %d Z columns > 256)", nv,
                  max_z);
    RKB_CHECK_ARG(bits >= 8 && bits <= 40, "bits must be in [8, 40] (got %d)", bits);
    RKB_CHECK_ARG(n_mod >= 1 && n_mod <= MAXMOD, "1..%d moduli supported (got %d)", MAXMOD, n_mod);
    RKB_CHECK_ARG(kpad % BKB == 0 && kpad >= (long)(nv - 1) * ng + max_z, "kpad must be a multiple of %d >= %ld",
                  BKB, (long)(nv - 1) * ng + max_z);
    RKB_CHECK_ARG(cwp >= ng + 2, "correction width must be >= ng + 2");
    RKB_CHECK_ARG(d_cbound != nullptr, "the correction-bound array is required");
    RKB_CHECK_ARG(row_base >= 0 && row_base + nrows <= nrows_total, "row range outside the residue matrices");
    RKB_CHECK_ARG(((uintptr_t)d_resA % 16) == 0 && (d_resB == nullptr || ((uintptr_t)d_resB % 16) == 0),
                  "residue buffers must be 16-byte aligned");
    RKB_CHECK_ARG(d_resB == nullptr || (b_col0 % BKB == 0 && b_col0 >= 0 && b_col0 <= (long)(nv - 1) * ng &&
                                        b_ld % BKB == 0 && b_ld >= (long)(nv - 1) * ng + max_z - b_col0),
                  "B must start at a multiple of %d columns within the body and hold every Z column", BKB);
    if (nrows == 0) return RKB_OK;
    RowsArgs a = {};
    a.b_col0 = (int)b_col0; a.b_ld = b_ld;
    a.P = d_Pv; a.Q = d_Qv; a.orb_ld = orb_ld; a.pairs = d_pairs; a.row_pair = d_row_pair; a.row_k = d_row_k;
    a.nrows = nrows; a.w = d_w; a.nv = nv; a.ng = ng; a.ktab = d_ktab; a.koff = d_koff; a.bits = bits;
    a.n_mod = n_mod;
    for (int i = 0; i < MAXMOD; ++i) {
        const int m = i < n_mod ? moduli[i] : 256;
        RKB_CHECK_ARG(m >= 2 && m <= 256, "moduli must lie in [2, 256]");
        a.mod[i] = m;
        a.inv_mod[i] = 1.0 / (double)m;
    }
    a.resA = d_resA; a.resB = d_resB; a.kpad = kpad; a.row_base = row_base; a.nrows_total = nrows_total;
    a.rowscale = d_rowscale; a.left = d_left; a.right = d_right; a.cbound = d_cbound; a.cwp = cwp;
    RKB_CHECK_ARG(d_ktab_t != nullptr && d_koff_t != nullptr, "the cell-minor factor tables are required");
    const int rows = nrows <= cell_single(ng) ? 1 : cell_rows(ng);
    const size_t smem = sizeof(double) * (size_t)(rows * cell_image(ng, nv, max_z) + cell_scratch(ng, rows));
    RKB_CHECK_ARG(smem <= 200 * 1024, "row images too large for shared memory");
    ResidueArgs f = {};
    for (int i = 0; i < n_mod; ++i) {
        const int m = moduli[i];
        auto near = [m](long v) { return (float)(2 * (v % m) > m ? v % m - m : v % m); };
        f.mod[i] = make_float4((float)m, 1.0f / (float)m, near(1L << 14), near(1L << 28));
    }
    cudaStream_t st = as_stream(stream);
    const dim3 grid((unsigned)ceil_div(nrows, rows)), block((unsigned)threads);
#define RKB_CELL_LAUNCH(NGV, RV)                                                                        \
    {                                                                                                   \
        RKB_CUDA(set_smem(split_rows_cell_kernel<NGV, RV>, (int)smem));                                 \
        split_rows_cell_kernel<NGV, RV><<<grid, block, smem, st>>>(a, f, d_ktab_t, d_koff_t, max_z);    \
    }
#define RKB_CELL_CASE(NGV)                                                                              \
    case NGV:                                                                                           \
        if (rows == 1) RKB_CELL_LAUNCH(NGV, 1) else RKB_CELL_LAUNCH(NGV, cell_rows(NGV))                \
        break;
    switch (ng) {
        RKB_CELL_CASE(5) RKB_CELL_CASE(6) RKB_CELL_CASE(7) RKB_CELL_CASE(8) RKB_CELL_CASE(9) RKB_CELL_CASE(10)
        default:
            RKB_CELL_CASE(11)
    }
#undef RKB_CELL_CASE
#undef RKB_CELL_LAUNCH
    RKB_LAUNCHED("split_rows_cell_kernel");
    return RKB_OK;
}

extern "C" int rkb_split_rows_cells(const double *d_Pv, const double *d_Qv, long orb_ld, const long *d_pairs,
                                    const long *d_row_pair, const int *d_row_k, long nrows, const double *d_w,
                                    int nv, int ng, const double *d_ktab, const long *d_koff,
                                    const double *d_ktab_t, const long *d_koff_t, int max_z, int bits,
                                    int n_mod, const int *moduli, signed char *d_resA, signed char *d_resB,
                                    long kpad, long row_base, long nrows_total, double *d_rowscale, double *d_left,
                                    double *d_right, double *d_cbound, int cwp, void *stream) {
    return rkb_split_rows_cells_z(d_Pv, d_Qv, orb_ld, d_pairs, d_row_pair, d_row_k, nrows, d_w, nv, ng, d_ktab, d_koff,
                                  d_ktab_t, d_koff_t, max_z, bits, n_mod, moduli, d_resA, d_resB, kpad, 0, kpad,
                                  row_base, nrows_total, d_rowscale, d_left, d_right, d_cbound, cwp, stream);
}

extern "C" long rkb_split_fused_body_width(int nv, int ng) {
    if (nv < 2 || ng < 1 || ng > 32) return -1;
    return rkb::split::fused_body_width(nv, ng);
}

extern "C" int rkb_split_rows_fused(const double *d_Pv, const double *d_Qv, long orb_ld, const long *d_pairs,
                                    const long *d_row_pair, const int *d_row_k, long nrows, const double *d_w,
                                    int nv, int ng, const double *d_ktab, const long *d_koff, int max_z, int bits,
                                    int n_mod, const int *moduli, signed char *d_resA, signed char *d_resB,
                                    long kpad, long row_base, long nrows_total, double *d_rowscale, double *d_left,
                                    double *d_right, double *d_cbound, int cwp, void *stream) {
    RKB_CHECK_ARG(nv >= 2 && ng >= 5 && ng <= 11, "the fused row kernel takes 5 <= ng <= 11 (got %d)", ng);
    RKB_CHECK_ARG(fused_passes(nv, ng) <= FUSED_PMAX, "grid too long for the fused row kernel (%ld passes > %d)",
                  fused_passes(nv, ng), FUSED_PMAX);
    RKB_CHECK_ARG(max_z >= 0 && max_z <= FUSED_ZMAX, "the fused row kernel takes <= %d Z columns (got %d)",
                  FUSED_ZMAX, max_z);
    RKB_CHECK_ARG(bits >= 8 && bits <= 40, "bits must be in [8, 40] (got %d)", bits);
    RKB_CHECK_ARG(n_mod >= 1 && n_mod <= MAXMOD, "1..%d moduli supported (got %d)", MAXMOD, n_mod);
    RKB_CHECK_ARG(kpad % BKB == 0 && kpad >= fused_body_width(nv, ng) + max_z,
                  "kpad must be a multiple of %d >= %ld", BKB, fused_body_width(nv, ng) + max_z);
    RKB_CHECK_ARG(cwp >= ng + 2 && cwp <= 32, "correction width must be in [ng + 2, 32]");
    RKB_CHECK_ARG(d_cbound != nullptr, "the correction-bound array is required");
    RKB_CHECK_ARG(row_base >= 0 && row_base + nrows <= nrows_total, "row range outside the residue matrices");
    RKB_CHECK_ARG(((uintptr_t)d_resA % 16) == 0 && (d_resB == nullptr || ((uintptr_t)d_resB % 16) == 0),
                  "residue buffers must be 16-byte aligned");
    if (nrows == 0) return RKB_OK;
    RowsArgs a = {};
    a.P = d_Pv; a.Q = d_Qv; a.orb_ld = orb_ld; a.pairs = d_pairs; a.row_pair = d_row_pair; a.row_k = d_row_k;
    a.nrows = nrows; a.w = d_w; a.nv = nv; a.ng = ng; a.ktab = d_ktab; a.koff = d_koff; a.bits = bits;
    a.n_mod = n_mod;
    for (int i = 0; i < MAXMOD; ++i) {
        const int m = i < n_mod ? moduli[i] : 256;
        RKB_CHECK_ARG(m >= 2 && m <= 256, "moduli must lie in [2, 256]");
        a.mod[i] = m;
        a.inv_mod[i] = 1.0 / (double)m;
    }
    a.resA = d_resA; a.resB = d_resB; a.kpad = kpad; a.row_base = row_base; a.nrows_total = nrows_total;
    a.rowscale = d_rowscale; a.left = d_left; a.right = d_right; a.cbound = d_cbound; a.cwp = cwp;
    const int warps = 4;
    dim3 grid((unsigned)ceil_div(nrows, warps)), block(32 * warps);
    cudaStream_t st = as_stream(stream);
    switch (ng) {
        case 5: split_rows_fused_kernel<5><<<grid, block, 0, st>>>(a); break;
        case 6: split_rows_fused_kernel<6><<<grid, block, 0, st>>>(a); break;
        case 7: split_rows_fused_kernel<7><<<grid, block, 0, st>>>(a); break;
        case 8: split_rows_fused_kernel<8><<<grid, block, 0, st>>>(a); break;
        case 9: split_rows_fused_kernel<9><<<grid, block, 0, st>>>(a); break;
        case 10: split_rows_fused_kernel<10><<<grid, block, 0, st>>>(a); break;
        default: split_rows_fused_kernel<11><<<grid, block, 0, st>>>(a); break;
    }
    RKB_LAUNCHED("split_rows_fused_kernel");
    return RKB_OK;
}

extern "C" int rkb_split_crt_weights(const int *moduli, int n_mod, int *dig_end, int *coef, unsigned *digit, int *weight) {
    CrtArgs p;
    const int rc = crt_weights(moduli, n_mod, p);
    if (rc) return rc;
    for (int i = 0; i < n_mod; ++i) coef[i] = p.coef[i];
    for (int g = 0; g < NDIG; ++g) {
        dig_end[g] = p.dig_end[g];
        digit[g] = (unsigned)p.D[g];
        const int w[4] = {p.f_hi[g], p.f_mid[g], p.f_lo[g], p.f_end[g]};
        for (int i = 0; i < 4; ++i) weight[4 * g + i] = w[i];
    }
    return RKB_OK;
}

extern "C" int rkb_split_contract_z(const signed char *d_resA, const signed char *d_resB, long kpad, long b_ld,
                                    long nrows_total, int n_mod, const int *moduli, double M,
                                    const double *d_rowscale, const double *d_left, const double *d_right,
                                    const double *d_cbound, double corr_floor, int cw, int cwp,
                                    const long *d_grp_row0, const long *d_grp_n, const long *d_grp_kdim,
                                    const int *d_grp_zchunk, const long *d_grp_out, const int *d_tasks,
                                    long n_tasks, double *d_out, int *d_status, void *stream) {
    RKB_CHECK_ARG(d_resB == nullptr || (b_ld % BKB == 0 && b_ld > 0 && b_ld <= kpad),
                  "B's width must be a positive multiple of %d, <= kpad", BKB);
    RKB_CHECK_ARG(n_mod >= 1 && n_mod <= MAXMOD, "1..%d moduli supported (got %d)", MAXMOD, n_mod);
    RKB_CHECK_ARG(kpad % BKB == 0 && kpad > 0 && kpad <= 3456, "kpad must be a positive multiple of %d, <= 3456",
                  BKB);
    RKB_CHECK_ARG((long)n_mod * nrows_total < (1L << 31), "residue matrices too tall for 32-bit TMA rows");
    RKB_CHECK_ARG(d_status != nullptr, "a device status word is required");
    RKB_CHECK_ARG(cw <= cwp, "cw must be <= cwp");
    RKB_CHECK_ARG(d_cbound != nullptr && corr_floor >= 0.0, "correction bounds and a nonnegative floor are required");
    if (n_tasks == 0) return RKB_OK;
    CrtArgs p;
    int rc = crt_weights(moduli, n_mod, p);
    if (rc) return rc;
    double prod = 1.0;
    for (int i = 0; i < n_mod; ++i) prod *= moduli[i];
    RKB_CHECK_ARG(M >= prod * (1.0 - 1e-14) && M <= prod * (1.0 + 1e-14), "M (%g) is not the product of the moduli (%g)",
                  M, prod);
    CUtensorMap mA, mB;
    rc = make_map(&mA, d_resA, kpad, (long)n_mod * nrows_total);
    if (rc) return rc;
    rc = d_resB ? make_map(&mB, d_resB, b_ld, (long)n_mod * nrows_total) : make_map(&mB, d_resA, kpad, (long)n_mod * nrows_total);
    if (rc) return rc;
    p.rowscale = d_rowscale; p.left = d_left; p.right = d_right; p.cbound = d_cbound; p.corr_floor = corr_floor;
    p.cwp = cwp; p.cw = cw;
    p.grp_row0 = d_grp_row0; p.grp_n = d_grp_n; p.grp_kdim = d_grp_kdim; p.grp_out = d_grp_out;
    p.grp_zc = d_resB ? d_grp_zchunk : nullptr;
    p.tasks = d_tasks; p.n_tasks = n_tasks; p.nrows_total = nrows_total; p.out = d_out; p.status = d_status;
    p.n_mod = n_mod; p.M = M * 0x1p-32;
    long grid = n_tasks < sm_count() ? n_tasks : sm_count();
    cudaStream_t st = as_stream(stream);
    RKB_CUDA(set_smem(crt_syrk_kernel, (int)SMEM_BYTES));
    crt_syrk_kernel<<<(unsigned)grid, THREADS, SMEM_BYTES, st>>>(mA, mB, p);
    RKB_LAUNCHED("crt_syrk_kernel");
    return RKB_OK;
}

extern "C" int rkb_split_contract(const signed char *d_resA, const signed char *d_resB, long kpad,
                                  long nrows_total, int n_mod, const int *moduli, const int *pair_inv,
                                  const double *f_hi,
                                  const double *f_lo, double M, const double *d_rowscale, const double *d_left,
                                  const double *d_right, const double *d_cbound, double corr_floor, int cw,
                                  int cwp, const long *d_grp_row0,
                                  const long *d_grp_n, const long *d_grp_kdim, const long *d_grp_out,
                                  const int *d_tasks, long n_tasks, double *d_out, int *d_status, void *stream) {
    (void)pair_inv, (void)f_hi, (void)f_lo;
    return rkb_split_contract_z(d_resA, d_resB, kpad, kpad, nrows_total, n_mod, moduli, M, d_rowscale, d_left, d_right,
                                d_cbound, corr_floor, cw, cwp, d_grp_row0, d_grp_n, d_grp_kdim, nullptr, d_grp_out,
                                d_tasks, n_tasks, d_out, d_status, stream);
}

// ---------------------------------------------------------------------------
// Certificate of each (ion, k) table from the row records, before or after the
// contraction.  Rounding row a to the quantum h_a = 2^(e_a - bits) moves entry
// (a, b) by about h_a |[X|Z]_b| + h_b |[X|Z]_a| (a random walk of K rounding
// errors against the other row), so the Schwarz-relative error of the table
// is estimated by
//     est = max_a h_a / sqrt|R_aa|  *  max_b |[X|Z]_b| / sqrt|R_bb|
// (rows with [X|Z] = 0 carry no rounding and are skipped; a vanishing or
// non-finite diagonal gives est = inf).  Tables with est > limit are counted in
// *flagged; the host recomputes them in FP64.  One 1024-thread block per table.
namespace rkb {
namespace split {
constexpr int CERT_THREADS = 1024;

__global__ void __launch_bounds__(CERT_THREADS) certify_kernel(const long *__restrict__ grp_row0,
                                                      const long *__restrict__ grp_n,
                                                      const double *__restrict__ rowscale,
                                                      const double *__restrict__ cbound, double limit,
                                                      double *__restrict__ est, int *__restrict__ flagged) {
    __shared__ double sm1[CERT_THREADS / 32], sm2[CERT_THREADS / 32];
    __shared__ int sbad[CERT_THREADS / 32];
    const long g = blockIdx.x;
    const long row0 = grp_row0[g], n = grp_n[g];
    double m1 = 0.0, m2 = 0.0;
    bool bad = false;
    for (long i = threadIdx.x; i < n; i += blockDim.x) {
        const long r = row0 + i;
        const double nrm = cbound[r * CB_STRIDE + 4];
        if (nrm == 0.0) continue;
        const double rd = sqrt(fabs(cbound[r * CB_STRIDE + 5]));
        const double t1 = rowscale[r] / rd, t2 = nrm / rd;
        if (!(t1 <= DBL_MAX) || !(t2 <= DBL_MAX)) {
            bad = true;
        } else {
            m1 = fmax(m1, t1);
            m2 = fmax(m2, t2);
        }
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
        m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    }
    const int badw = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        sm1[wid] = m1;
        sm2[wid] = m2;
        sbad[wid] = badw;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        bool any = false;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            m1 = fmax(m1, sm1[w]);
            m2 = fmax(m2, sm2[w]);
            any |= sbad[w] != 0;
        }
        const double e = any ? INFINITY : m1 * m2;
        est[g] = e;
        if (!(e <= limit)) atomicAdd(flagged, 1);
    }
}
}  // namespace split
}  // namespace rkb

extern "C" int rkb_split_certify(const long *d_grp_row0, const long *d_grp_n, long n_groups, const double *d_rowscale,
                                 const double *d_cbound, double limit, double *d_est, int *d_flagged, void *stream) {
    RKB_CHECK_ARG(n_groups >= 0 && n_groups <= 0x7fffffffL, "invalid group count %ld", n_groups);
    RKB_CHECK_ARG(limit >= 0.0, "the certificate limit must be >= 0");
    RKB_CHECK_ARG(d_flagged != nullptr && (n_groups == 0 || (d_grp_row0 && d_grp_n && d_rowscale && d_cbound && d_est)),
                  "null argument");
    cudaStream_t st = as_stream(stream);
    RKB_CUDA(cudaMemsetAsync(d_flagged, 0, sizeof(int), st));
    if (n_groups == 0) return RKB_OK;
    certify_kernel<<<(unsigned)n_groups, CERT_THREADS, 0, st>>>(d_grp_row0, d_grp_n, d_rowscale, d_cbound, limit,
                                                               d_est, d_flagged);
    RKB_LAUNCHED("certify_kernel");
    return RKB_OK;
}

// ---------------------------------------------------------------------------
// rkb_split_rows_noalloc: rkb_split_rows whose row workspace is a fixed array
// compiled into this library instead of caller memory.  It is meant for hosts
// that cannot call cudaMalloc on this path: a C or Fortran program that links
// only this ABI and hands over buffers from its own pool, or a process that
// plans every device allocation up front and may not have cudaMalloc /
// cudaFree synchronise the device in the middle of its pipelined streams.
//
// The array holds RKB_SPLIT_ROWS_NOALLOC_MAX_DOUBLES doubles (16 MiB) on every
// GPU that loads the library, until the process exits.  The host name of a
// __device__ array is only a host-side stand-in, so its device address is
// looked up per device with cudaGetSymbolAddress, on the first call made with
// that device current; make that first call before any stream capture.
// Every call shares the one array, so calls that overlap on the GPU (other
// streams, other host threads) race and must be serialised by the caller.
// Nothing needs clearing between calls: the row kernel writes every element
// of each row [X | Z | 0] that the residue kernel later reads.
namespace rkb {
namespace split {
static __device__ __align__(256) double g_noalloc_xwork[RKB_SPLIT_ROWS_NOALLOC_MAX_DOUBLES];

constexpr int NOALLOC_MAX_DEVICES = 64;
static double *g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};
static std::mutex g_noalloc_mutex;
}  // namespace split
}  // namespace rkb

extern "C" int rkb_split_rows_noalloc(const double *d_Pv, const double *d_Qv, long orb_ld, const long *d_pairs,
                                      const long *d_row_pair, const int *d_row_k, long nrows, const double *d_w,
                                      int nv, int ng, const double *d_ktab, const long *d_koff, int bits,
                                      int n_mod, const int *moduli, signed char *d_resA, signed char *d_resB,
                                      long kpad, long row_base, long nrows_total, double *d_rowscale,
                                      double *d_left, double *d_right, double *d_cbound, int cwp,
                                      const int *d_zcount, void *stream) {
    const long cap = (long)RKB_SPLIT_ROWS_NOALLOC_MAX_DOUBLES;
    RKB_CHECK_ARG(kpad > 0 && nrows >= 0 && row_base >= 0, "invalid row range or width");
    RKB_CHECK_ARG(row_base <= cap / kpad && nrows <= cap / kpad - row_base,
                  "rows [0, %ld) of width %ld need %ld workspace doubles; the fixed workspace holds %ld "
                  "(use rkb_split_rows with a caller buffer)",
                  row_base + nrows, kpad, (row_base + nrows) * kpad, cap);
    int dev = -1;
    RKB_CUDA(cudaGetDevice(&dev));
    RKB_CHECK_ARG(dev >= 0 && dev < NOALLOC_MAX_DEVICES, "device ordinal %d out of range", dev);
    double *ws = nullptr;
    {
        std::lock_guard<std::mutex> guard(g_noalloc_mutex);
        if (g_noalloc_addr[dev] == nullptr) {
            void *addr = nullptr;
            RKB_CUDA(cudaGetSymbolAddress(&addr, g_noalloc_xwork));
            g_noalloc_addr[dev] = static_cast<double *>(addr);
        }
        ws = g_noalloc_addr[dev];
    }
    return rkb_split_rows(d_Pv, d_Qv, orb_ld, d_pairs, d_row_pair, d_row_k, nrows, d_w, nv, ng, d_ktab, d_koff,
                          bits, n_mod, moduli, d_resA, d_resB, kpad, row_base, nrows_total, d_rowscale, d_left,
                          d_right, d_cbound, cwp, ws, d_zcount, stream);
}
