// Cell (bank) R^k engine on the device: atomx numerics/bspline/convol.py.
//
// A bank holds the four-index integrals
//     rkb[i][j][ip][jp] = int int B_i B_{i+ip}(r1) r_<^k / r_>^(k+1) B_j B_{j+jp}(r2)
// of one component pair (P or Q basis on each electron), assembled from
// per-cell moments (cells far apart: the kernel factorises) and diagonal-cell
// integrals (nested Gauss quadrature).  Here every bank is stored as a dense
// matrix K[(ip, i)][(jp, j)] = rkb[i][j][ip][jp] (row ip*ns + i, column
// jp*ns + j) inside one block matrix per multipole,
//     K_full = [[K_pp, K_pq], [K_qp, K_qq]],
// so that with the banded pair densities of _density_sym laid out in the same
// index order, D(ab) = [D_P(ab) | D_Q(ab)], atomx's cell integral is the
// bilinear form R^k(ab, cd) = D(ab) K_full D(cd)^T.  Whole tables and batches
// of integrals are then FP64 GEMMs on the DMMA pipe plus gathered dots.
//
// The bank construction kernels keep the reference's operation order with
// explicitly rounded multiplies and adds (no fused multiply-add), so the banks
// equal atomx's bit for bit: moments (convol.py:58-94), diagonal cells
// (_triang_sym :136-250, _triang_pqpq :388-530), assembly (:324-381,
// :533-576).  So does the exchange contraction (_convol_case4_t :1001-1059)
// and the bilinear fold (_rkb_bilinear :1901-1942).
#include <cmath>

#include "rkb_common.cuh"
#include "rkb_dgemm.cuh"

namespace rkb {
namespace cell {

constexpr int MAX_KS = 16;
constexpr int MAX_NSUB = 64;

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }

// w r^k (k > 0), w / r^-k (k < 0), w (k = 0)
__device__ __forceinline__ double power_weight(double w, double r, int k) {
    if (k > 0) return mul(w, int_pow(r, k));
    if (k < 0) return dvd(w, int_pow(r, -k));
    return w;
}

// packed upper pair (h, hp), hp >= h, of order ks: h*ks - h(h-1)/2 + (hp - h)
__device__ __forceinline__ int packed(int h, int hp, int ks) { return h * ks - (h * (h - 1)) / 2 + (hp - h); }

__device__ __forceinline__ void unpack(int p, int ks, int &h, int &hp) {
    h = 0;
    while (p >= ks - h) {
        p -= ks - h;
        ++h;
    }
    hp = h + p;
}

// B-spline values of order ks at x in the interval starting at knot `left`
// (de Boor's recurrence, the reference's _bsplvb_inplace order).
__device__ void bsplvb(const double *__restrict__ t, int ks, double x, int left, double *b) {
    double dr[MAX_KS], dl[MAX_KS];
    b[0] = 1.0;
    for (int i = 1; i < ks; ++i) b[i] = 0.0;
    for (int j = 1; j < ks; ++j) {
        dr[j] = sub(t[left + j], x);
        dl[j] = sub(x, t[left + 1 - j]);
        double saved = 0.0;
        for (int r = 0; r < j; ++r) {
            const double term = dvd(b[r], add(dr[r + 1], dl[j - r]));
            b[r] = add(saved, mul(dr[r + 1], term));
            saved = mul(dl[j - r], term);
        }
        b[j] = saved;
    }
}

// ------------------------------------------------------------------ moments
// out[ii][iv] = sum_m B_i B_j(iv, m) * power_weight(grw, gr, k), ii = packed (i, j)
__global__ void moments_kernel(const double *__restrict__ bsp, const double *__restrict__ gr,
                               const double *__restrict__ grw, int nv, int ng, int ks, int k,
                               double *__restrict__ out) {
    const int kk = ks * (ks + 1) / 2;
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)kk * nv) return;
    const int ii = (int)(t / nv), iv = (int)(t % nv);
    int i, j;
    unpack(ii, ks, i, j);
    double s = 0.0;
    for (int m = 0; m < ng; ++m) {
        const double *b = bsp + ((long)iv * ng + m) * ks;
        const double gw = power_weight(grw[iv * ng + m], gr[iv * ng + m], k);
        s = add(s, mul(mul(b[i], b[j]), gw));
    }
    out[t] = s;
}

// ----------------------------------------------------------- diagonal cells
struct DiagSmem {
    double *bsub, *gwr, *span, *intp, *bw, *res_a, *res_b;
};

// One pass of the nested quadrature on cell iv: the inner integrals of the
// inner component's products (knots t_i, order ks_i) up to each outer node,
// then the outer sum with the outer component's products and the 1/r^(k+1)
// weight: res[ii_o][jj_i].
__device__ void diag_pass(const double *__restrict__ bsp_o, int ks_o, const double *__restrict__ t_i, int ks_i,
                          int iv, const double *__restrict__ gr, const double *__restrict__ grw, int ng, int k,
                          int n_sub, const double *__restrict__ x01, const double *__restrict__ w01, DiagSmem sm,
                          double *res) {
    const int left = ks_i - 1 + iv;
    const double xbase = t_i[left];
    for (int m = threadIdx.x; m < ng; m += blockDim.x) sm.span[m] = sub(gr[iv * ng + m], xbase);
    __syncthreads();
    for (int p = threadIdx.x; p < ng * n_sub; p += blockDim.x) {
        const int m = p / n_sub, n = p % n_sub;
        const double span = sm.span[m];
        double *b = sm.bsub + (long)p * ks_i;
        if (span < 1e-30) {
            for (int s = 0; s < ks_i; ++s) b[s] = 0.0;
            sm.gwr[p] = 0.0;
            continue;
        }
        const double gx = add(xbase, mul(span, x01[n]));
        bsplvb(t_i, ks_i, gx, left, b);
        const double w = mul(span, w01[n]);
        sm.gwr[p] = k > 0 ? mul(w, int_pow(gx, k)) : (k < 0 ? dvd(w, int_pow(gx, -k)) : w);
    }
    __syncthreads();
    const int kki = ks_i * (ks_i + 1) / 2, kko = ks_o * (ks_o + 1) / 2;
    for (int p = threadIdx.x; p < kki * ng; p += blockDim.x) {
        const int jj = p / ng, m = p % ng;
        int j, jp;
        unpack(jj, ks_i, j, jp);
        double s = 0.0;
        if (!(sm.span[m] < 1e-30)) {
            for (int n = 0; n < n_sub; ++n) {
                const double *b = sm.bsub + ((long)m * n_sub + n) * ks_i;
                s = add(s, mul(mul(b[j], b[jp]), sm.gwr[m * n_sub + n]));
            }
        }
        sm.intp[jj * ng + m] = s;
    }
    for (int p = threadIdx.x; p < kko * ng; p += blockDim.x) {
        const int ii = p / ng, m = p % ng;
        int i, ip;
        unpack(ii, ks_o, i, ip);
        const double ow = dvd(grw[iv * ng + m], int_pow(gr[iv * ng + m], k + 1));
        const double *bo = bsp_o + ((long)iv * ng + m) * ks_o;
        sm.bw[ii * ng + m] = mul(mul(bo[i], bo[ip]), ow);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < kko * kki; p += blockDim.x) {
        const int ii = p / kki, jj = p % kki;
        double s = 0.0;
        for (int m = 0; m < ng; ++m) s = add(s, mul(sm.bw[ii * ng + m], sm.intp[jj * ng + m]));
        res[p] = s;
    }
    __syncthreads();
}

// One block per cell: out[ii_l][jj_r][iv] (kk_l x kk_r x nv).
__global__ void diag_kernel(const double *__restrict__ bsp_l, const double *__restrict__ bsp_r,
                            const double *__restrict__ gr, const double *__restrict__ grw,
                            const double *__restrict__ t_l, const double *__restrict__ t_r, int nv, int ng, int ks_l,
                            int ks_r, int same, int k, int n_sub, const double *__restrict__ x01,
                            const double *__restrict__ w01, double *__restrict__ out) {
    extern __shared__ double smem[];
    const int iv = blockIdx.x;
    const int ks_max = ks_l > ks_r ? ks_l : ks_r;
    const int kkl = ks_l * (ks_l + 1) / 2, kkr = ks_r * (ks_r + 1) / 2, kkm = ks_max * (ks_max + 1) / 2;
    DiagSmem sm;
    sm.bsub = smem;
    sm.gwr = sm.bsub + (long)ng * n_sub * ks_max;
    sm.span = sm.gwr + ng * n_sub;
    sm.intp = sm.span + ng;
    sm.bw = sm.intp + kkm * ng;
    sm.res_a = sm.bw + kkm * ng;
    sm.res_b = sm.res_a + kkl * kkr;
    // left outer, right inner: a[ii_l][jj_r]
    diag_pass(bsp_l, ks_l, t_r, ks_r, iv, gr, grw, ng, k, n_sub, x01, w01, sm, sm.res_a);
    if (same) {
        for (int p = threadIdx.x; p < kkl * kkr; p += blockDim.x) {
            const int ii = p / kkr, jj = p % kkr;
            out[(long)p * nv + iv] = add(sm.res_a[ii * kkr + jj], sm.res_a[jj * kkr + ii]);
        }
        return;
    }
    // right outer, left inner: b[jj_r][ii_l]
    diag_pass(bsp_r, ks_r, t_l, ks_l, iv, gr, grw, ng, k, n_sub, x01, w01, sm, sm.res_b);
    for (int p = threadIdx.x; p < kkl * kkr; p += blockDim.x) {
        const int ii = p / kkr, jj = p % kkr;
        out[(long)p * nv + iv] = add(sm.res_a[ii * kkr + jj], sm.res_b[jj * kkl + ii]);
    }
}

// ------------------------------------------------------------------ assembly
// One thread per bank element, stored at K[(row_off + ip*ns + i)][col_off + jp*ns + j]:
// cells iv < jv contribute rising_l[ii][iv] falling_r[jj][jv], cells iv > jv
// rising_r[jj][jv] falling_l[ii][iv], iv == jv the diagonal cell; summed over
// jv, then iv, ascending.
__global__ void assemble_kernel(const double *__restrict__ rl, const double *__restrict__ fl,
                                const double *__restrict__ rr, const double *__restrict__ fr,
                                const double *__restrict__ diag, int nv, int ks_l, int ks_r, int ns,
                                double *__restrict__ out, long ld, long row_off, long col_off) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ks_l * ns * ks_r * ns) return;
    const int j = (int)(t % ns);
    const long r1 = t / ns;
    const int jp = (int)(r1 % ks_r);
    const long r2 = r1 / ks_r;
    const int i = (int)(r2 % ns), ip = (int)(r2 / ns);
    const int kkr = ks_r * (ks_r + 1) / 2;
    const int jv_lo = max(0, j - (ks_r - 1 - jp)), jv_hi = min(j, nv - 1);
    const int iv_lo = max(0, i - (ks_l - 1 - ip)), iv_hi = min(i, nv - 1);
    double acc = 0.0;
    for (int jv = jv_lo; jv <= jv_hi; ++jv) {
        const int jh = j - jv, jj = packed(jh, jh + jp, ks_r);
        for (int iv = iv_lo; iv <= iv_hi; ++iv) {
            const int ih = i - iv, ii = packed(ih, ih + ip, ks_l);
            double c;
            if (iv < jv) c = mul(rl[(long)ii * nv + iv], fr[(long)jj * nv + jv]);
            else if (iv > jv) c = mul(rr[(long)jj * nv + jv], fl[(long)ii * nv + iv]);
            else c = diag[((long)ii * kkr + jj) * nv + iv];
            acc = add(acc, c);
        }
    }
    out[(row_off + (long)ip * ns + i) * ld + col_off + (long)jp * ns + j] = acc;
}

// ---------------------------------------------------------------- densities
// Banded pair densities of _density_sym (extent ns_d, order ks; component
// vectors of stored lengths n1, n2) in bank index order:
// out[p][col_off + s*ns_k + i] = d[i][s].
__global__ void densities_kernel(const double *__restrict__ c1, const double *__restrict__ c2, long ld,
                                 const long *__restrict__ pairs, long n_pairs, int n1, int n2, int ns_d, int ns_k,
                                 int ks, double *__restrict__ out, long out_ld, long col_off) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_pairs * ks * ns_k) return;
    const int i = (int)(t % ns_k);
    const long r = t / ns_k;
    const int s = (int)(r % ks);
    const long p = r / ks;
    const double *p1 = c1 + pairs[2 * p] * ld, *p2 = c2 + pairs[2 * p + 1] * ld;
    double v = 0.0;
    if (i < min(n1, ns_d)) {
        if (s == 0) {
            if (i < n2) v = mul(p1[i], p2[i]);
        } else {
            const int ip = i + s;
            if (ip < ns_d) {
                double x = 0.0;
                if (ip < n2) x = add(x, mul(p1[i], p2[ip]));
                if (ip < n1 && i < n2) x = add(x, mul(p1[ip], p2[i]));
                v = x;
            }
        }
    }
    out[p * out_ld + col_off + (long)s * ns_k + i] = v;
}

// ------------------------------------------------------------- FP64 GEMM NT
// C[m][n] (+)= sum_x A[m][x] B[n][x], a block per tile (rkb_dgemm.cuh).
template <class T>
__device__ __forceinline__ void gemm_tile(const double *__restrict__ A, long lda, const double *__restrict__ B, long ldb,
                                          double *__restrict__ C, long ldc, long M, long N, long K, long i0, long j0,
                                          int accumulate, double *smem) {
    const double *o = T::run(A, lda, i0, M, B, ldb, j0, N, (int)(K / dgemm::BK), smem);
    constexpr int WS = T::SIDE / 2, RPW = 32 / WS;  // rows a warp stores at a time
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long j = j0 + warp % 2 * WS + lane % WS, i = i0 + warp / 2 * WS + lane / WS;
    o += lane / WS * T::OLD + lane % WS;
    if (j >= N) return;
#pragma unroll 8
    for (int r = 0; r < WS; r += RPW)
        if (i + r < M) {
            double *c = C + (i + r) * ldc + j;
            *c = accumulate ? *c + o[r * T::OLD] : o[r * T::OLD];
        }
}

template <class T>
__global__ void __launch_bounds__(dgemm::THREADS, 3)
gemm_nt_kernel(const double *__restrict__ A, long lda, const double *__restrict__ B, long ldb, double *__restrict__ C,
               long ldc, long M, long N, long K, int accumulate) {
    extern __shared__ __align__(16) double smem[];
    const long tn = (N + T::SIDE - 1) / T::SIDE;
    gemm_tile<T>(A, lda, B, ldb, C, ldc, M, N, K, blockIdx.x / tn * T::SIDE, blockIdx.x % tn * T::SIDE, accumulate, smem);
}

// Row ranges of A and C against a B each, in one launch: as launches of their own (one
// per multipole) the ranges fill a few waves of the chip badly, or less than one.
// Whole calls, launches of their own -> one launch: cell_tables of a many-electron basis
// (its GEMM 3.48 ms now) 7.41 -> 5.30 ms, a 2000-key batch (0.59 ms) 2.14 -> 1.96 ms,
// Fock blocks 2.56 -> 2.21 ms.
constexpr int MAX_GROUPS = 64;
struct GroupArgs {
    const double *B[MAX_GROUPS];
    long row0[MAX_GROUPS + 1];   // rows of A and C
    long tile0[MAX_GROUPS + 1];  // tiles before each group
    int n;
};

template <class T>
__global__ void __launch_bounds__(dgemm::THREADS, 3)
gemm_nt_groups_kernel(const double *__restrict__ A, long lda, const __grid_constant__ GroupArgs g, long ldb,
                      double *__restrict__ C, long ldc, long N, long K) {
    extern __shared__ __align__(16) double smem[];
    int q = 0;
    while (q + 1 < g.n && (long)blockIdx.x >= g.tile0[q + 1]) ++q;
    const long t = blockIdx.x - g.tile0[q], tn = (N + T::SIDE - 1) / T::SIDE;
    gemm_tile<T>(A + g.row0[q] * lda, lda, g.B[q], ldb, C + g.row0[q] * ldc, ldc, g.row0[q + 1] - g.row0[q], N, K,
                 t / tn * T::SIDE, t % tn * T::SIDE, 0, smem);
}

// ------------------------------------------------------------- gathered dots
// out[e] = sum_x L[il[e]][x] W[iw[e]][x], one warp per entry
__global__ void dots_kernel(const double *__restrict__ L, long l_ld, const double *__restrict__ W, long w_ld, long n,
                            const long *__restrict__ il, const long *__restrict__ iw, long n_ent,
                            double *__restrict__ out) {
    const long e = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (e >= n_ent) return;
    const double *x = L + il[e] * l_ld, *y = W + iw[e] * w_ld;
    double s = 0.0;
    for (long i = lane; i < n; i += 32) s = fma(x[i], y[i], s);
    s = warp_sum(s);
    if (lane == 0) out[e] = s;
}

// ----------------------------------------------------------------- exchange
// _convol_case4_t on one bank block: a[row][col] over the four families in
// the reference's order; `symmetric` computes col <= row and mirrors.  Bank
// element rkb[i][j][ip][jp] = K[(ip*ns + i) * ld + jp*ns + j].  Batch b uses
// density d + b*ns*ns, bank block K + kofs[b], output a + b*ns*ns.
__global__ void exchange_kernel(const double *__restrict__ K, long ld, const long *__restrict__ kofs,
                                const double *__restrict__ d, int ns, int ks, int ks_r, int symmetric,
                                int accumulate, double *__restrict__ a, long nbatch) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long per = (long)ns * ns;
    if (t >= per * nbatch) return;
    const long b = t / per;
    const int row = (int)((t % per) / ns), col = (int)(t % ns);
    if (symmetric && col > row) return;
    const double *Kb = K + kofs[b];
    const double *db = d + b * per;
#define RKB(i, j, ip, jp) Kb[((long)(ip) * ns + (i)) * ld + (long)(jp) * ns + (j)]
    double s = 0.0;
    for (int ip = 0; ip < ks; ++ip) {
        const int i = row - ip;
        if (i < 0) continue;
        for (int jp = 0; jp < ks_r; ++jp)
            if (col < ns - jp) s = add(s, mul(RKB(i, col, ip, jp), db[(long)i * ns + col + jp]));
    }
    for (int ip = 1; ip < ks; ++ip) {
        const int ii = row + ip;
        if (ii >= ns) continue;
        for (int jp = 0; jp < ks_r; ++jp)
            if (col < ns - jp) s = add(s, mul(RKB(row, col, ip, jp), db[(long)ii * ns + col + jp]));
    }
    for (int jp = 1; jp < ks_r; ++jp)
        for (int ip = 0; ip < ks; ++ip) {
            const int i = row - ip;
            if (i < 0) continue;
            if (col >= jp) s = add(s, mul(RKB(i, col - jp, ip, jp), db[(long)i * ns + col - jp]));
        }
    for (int ip = 1; ip < ks; ++ip) {
        const int ii = row + ip;
        if (ii >= ns) continue;
        for (int jp = 1; jp < ks_r; ++jp)
            if (col >= jp) s = add(s, mul(RKB(row, col - jp, ip, jp), db[(long)ii * ns + col - jp]));
    }
#undef RKB
    double *o = a + b * per + (long)row * ns + col;
    *o = accumulate ? add(*o, s) : s;
    if (symmetric && col < row) {
        double *m = a + b * per + (long)col * ns + row;
        *m = accumulate ? add(*m, s) : s;
    }
}

// ----------------------------------------------------------------- bilinear
// _rkb_bilinear stage 1, gathered: T[m][j][jp] over the reference's scatter
// order (left pairs i = m - ip for ip = ks_l-1..1, then i = m with ip = 0..).
__global__ void bilinear_t_kernel(const double *__restrict__ K, long ld, int ns, const double *__restrict__ wa,
                                  int n_left, int n_right, int ks_l, int ks_r, int ns_out, double *__restrict__ T) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ns_out * n_right * ks_r) return;
    const int jp = (int)(t % ks_r);
    const long r = t / ks_r;
    const int j = (int)(r % n_right), m = (int)(r / n_right);
#define RKB(i, j, ip, jp) K[((long)(ip) * ns + (i)) * ld + (long)(jp) * ns + (j)]
    double s = 0.0;
    if (j + jp < n_right) {
        for (int i = max(0, m - (ks_l - 1)); i < m; ++i) {  // i + ip = m, ip = m - i > 0
            if (i >= n_left || m >= n_left) continue;
            s = add(s, mul(RKB(i, j, m - i, jp), wa[i]));
        }
        if (m < n_left)
            for (int ip = 0; ip < ks_l; ++ip) {
                if (m + ip >= n_left) break;
                s = add(s, mul(RKB(m, j, ip, jp), wa[m + ip]));
            }
    }
#undef RKB
    T[t] = s;
}

// stage 2: M[m][n] from T over the reference's order (right pairs j = n - jp
// for jp = ks_r-1..1, then j = n with jp = 0..)
__global__ void bilinear_m_kernel(const double *__restrict__ T, const double *__restrict__ wb, int n_right, int ks_r,
                                  int ns_out, double *__restrict__ M) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ns_out * ns_out) return;
    const int n = (int)(t % ns_out), m = (int)(t / ns_out);
    const double *Tm = T + (long)m * n_right * ks_r;
    double s = 0.0;
    for (int j = max(0, n - (ks_r - 1)); j < n; ++j) {  // j + jp = n, jp > 0
        if (j >= n_right || n >= n_right) continue;
        s = add(s, mul(Tm[(long)j * ks_r + (n - j)], wb[j]));
    }
    if (n < n_right)
        for (int jp = 0; jp < ks_r; ++jp) {
            if (n + jp >= n_right) break;
            s = add(s, mul(Tm[(long)n * ks_r + jp], wb[n + jp]));
        }
    M[t] = s;
}

// ------------------------------------------------------- Fock-block helpers
// Direct density of one (target, block, k): dd[s*ns + i] = sum_j c_j (doubled
// for j = target) of the symmetric band of comp[j] (convol.py:647-686).
__global__ void direct_density_kernel(const double *__restrict__ comp, long ld, int n_orb,
                                      const double *__restrict__ coef, long coef_stride, const int *__restrict__ target,
                                      int ns, int ks, double *__restrict__ dd, long out_ld, long nbatch) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ns * ks * nbatch) return;
    const long b = t / ((long)ns * ks);
    const int s = (int)((t / ns) % ks), i = (int)(t % ns);
    const double *c = coef + b * coef_stride;
    double v = 0.0;
    if (i + s < ns)
        for (int j = 0; j < n_orb; ++j) {
            double cj = c[j];
            if (cj == 0.0) continue;
            if (j == target[b]) cj = add(cj, cj);
            const double pi = comp[(long)j * ld + i];
            if (s == 0) v = add(v, mul(mul(cj, pi), pi));
            else {
                const double ps = comp[(long)j * ld + i + s];
                v = add(v, mul(cj, add(mul(pi, ps), mul(ps, pi))));
            }
        }
    dd[b * out_ld + (long)s * ns + i] = v;
}

// Exchange density: xx[i][k] = sum_j (c_j comp_ii[j][i]) comp_jj[j][k] (convol.py:689-710)
__global__ void exchange_density_kernel(const double *__restrict__ comp_ii, const double *__restrict__ comp_jj,
                                        long ld, int n_orb, const double *__restrict__ coef, long coef_stride, int ns,
                                        double *__restrict__ xx, long nbatch) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long per = (long)ns * ns;
    if (t >= per * nbatch) return;
    const long b = t / per;
    const int i = (int)((t % per) / ns), kk = (int)(t % ns);
    const double *c = coef + b * coef_stride;
    double v = 0.0;
    for (int j = 0; j < n_orb; ++j) {
        const double cj = c[j];
        if (cj == 0.0) continue;
        v = add(v, mul(mul(cj, comp_ii[(long)j * ld + i]), comp_jj[(long)j * ld + kk]));
    }
    xx[t] = v;
}

// Banded potential to a full symmetric matrix: V[i][i+s] += v[s*ns + i] and
// its mirror (convol.py:815-826).  One thread per (i, s); rows of one batch
// element touch disjoint entries for distinct (i, s).
__global__ void banded_to_full_kernel(const double *__restrict__ v, int ns, int ks, double *__restrict__ V,
                                      long nbatch) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)ns * ks * nbatch) return;
    const long b = t / ((long)ns * ks);
    const int s = (int)((t / ns) % ks), i = (int)(t % ns);
    if (i + s >= ns) return;
    const double val = v[t];
    double *Vb = V + b * (long)ns * ns;
    Vb[(long)i * ns + i + s] = add(Vb[(long)i * ns + i + s], val);
    if (s > 0) Vb[(long)(i + s) * ns + i] = add(Vb[(long)(i + s) * ns + i], val);
}

// Fock blocks: PP = 0.5 (PP + PP^T), QQ likewise, PQ = 0.5 (PQ + QP^T) (or
// QP^T when the PQ exchange was skipped), QP = PQ^T, all divided by the norm
// when it exceeds 1e-15 (dirac_fock.py:1295-1319).  h holds PP, QQ, PQ, QP of
// each batch element (4 ns x ns); out receives the result.
__global__ void fock_finish_kernel(const double *__restrict__ h, const double *__restrict__ norm, int ns,
                                   int skip_pq, double *__restrict__ out, long nbatch) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long per = (long)ns * ns;
    if (t >= per * nbatch) return;
    const long b = t / per;
    const int i = (int)((t % per) / ns), j = (int)(t % ns);
    const double *H = h + b * 4 * per;
    double *O = out + b * 4 * per;
    const double nb = norm[b];
    auto fin = [&](double x) { return nb > 1e-15 ? x / nb : x; };
    const long ij = (long)i * ns + j, ji = (long)j * ns + i;
    O[ij] = fin(0.5 * (H[ij] + H[ji]));
    O[per + ij] = fin(0.5 * (H[per + ij] + H[per + ji]));
    const double pq = skip_pq ? H[3 * per + ji] : 0.5 * (H[2 * per + ij] + H[3 * per + ji]);
    const double qp = skip_pq ? H[3 * per + ij] : 0.5 * (H[2 * per + ji] + H[3 * per + ij]);
    O[2 * per + ij] = fin(pq);
    O[3 * per + ij] = fin(qp);
}

// ------------------------------------------------- Fock blocks of many targets
// All the densities, and then all the exchange contractions, of a DBSR Fock step
// in one launch each: component blocks (PP, QQ, PQ, QP), multipoles and targets
// together.  Launched one (block, multipole) at a time they were 226 launches a step,
// each too small for the chip.
struct FockArgs {
    const double *const *K;  // bank matrices of the nk multipoles (device array of device pointers)
    long ld, q_off;          // their leading dimension, and the Q block's row and column offset
    int nk, nt, n_orb, ns, ks[2];  // spline orders of P, Q
    const double *comp[2];   // coefficient stacks P, Q
    long c_ld;
    const double *ad, *ax;   // angular coefficients [nk][nt][n_orb]
    const int *target;
    double *dd;              // direct densities [Q or P][nk][nt][dd_ld], zero padded
    long dd_ld;
    const double *v;         // their potentials [P or Q source][nk][nt][ld]
    double *xx;              // exchange densities [block][nk][nt][ns][ns]
    double *h;               // blocks [nt][4][ns][ns]
    int skip_pq;
};
__global__ void fock_direct_density_kernel(const __grid_constant__ FockArgs f) {
    const long x = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= f.dd_ld) return;
    const int t = blockIdx.y % f.nt, kc = blockIdx.y / f.nt;  // kc = source component * nk + multipole
    const int src = kc / f.nk, k = kc % f.nk;
    const int s = (int)(x / f.ns), i = (int)(x % f.ns);
    const double *c = f.ad + ((long)k * f.nt + t) * f.n_orb, *comp = f.comp[src];
    double v = 0.0;
    if (s < f.ks[src] && i + s < f.ns)
        for (int j = 0; j < f.n_orb; ++j) {
            double cj = c[j];
            if (cj == 0.0) continue;
            if (j == f.target[t]) cj = add(cj, cj);
            const double pi = comp[(long)j * f.c_ld + i];
            if (s == 0) v = add(v, mul(mul(cj, pi), pi));
            else {
                const double ps = comp[(long)j * f.c_ld + i + s];
                v = add(v, mul(cj, add(mul(pi, ps), mul(ps, pi))));
            }
        }
    f.dd[((long)kc * f.nt + t) * f.dd_ld + x] = v;
}

__global__ void fock_exchange_density_kernel(const __grid_constant__ FockArgs f) {
    const int per = f.ns * f.ns;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= per) return;
    const int t = blockIdx.y % f.nt, bk = blockIdx.y / f.nt;  // bk = block * nk + multipole
    const int blk = bk / f.nk, k = bk % f.nk;
    if (f.skip_pq && blk == 1) return;
    const int i = e / f.ns, j2 = e % f.ns;
    const double *c = f.ax + ((long)k * f.nt + t) * f.n_orb;
    const double *pl = f.comp[blk >> 1] + i, *pr = f.comp[blk & 1] + j2;
    double v = 0.0;
    for (int j = 0; j < f.n_orb; ++j) {
        const double cj = __ldg(c + j);
        if (cj == 0.0) continue;
        v = add(v, mul(mul(cj, __ldg(pl + j * f.c_ld)), __ldg(pr + j * f.c_ld)));
    }
    f.xx[((long)bk * f.nt + t) * per + e] = v;
}

// One thread per (row, column) entry of BT targets, which share each bank element
// read.  The summation order of exchange_kernel is kept for every entry, and the sums
// over blocks and multipoles are those of one block and multipole at a time.
// Bound by the latency of the bank reads from L2.  A whole Fock step of 24 targets and
// 8 multipoles at 120 splines took 6.0 ms in 226 launches, one target a thread (3.5 ms
// of it in 32 exchange launches), and took 2.67 ms with eight targets a thread (2.21 with
// the grouped GEMM too); four targets 3.07, twelve 3.65, four targets of two rows 4.1.
constexpr int FOCK_THREADS = 128;  // columns a block
template <int BT>
__global__ void __launch_bounds__(FOCK_THREADS, 5) fock_exchange_kernel(const __grid_constant__ FockArgs f) {
    const int ns = f.ns, blk = blockIdx.z & 3, t0 = (blockIdx.z >> 2) * BT;
    const int left = blk >> 1, right = blk & 1, row = blockIdx.y, col = blockIdx.x * blockDim.x + threadIdx.x;
    const bool symmetric = left == right;
    if ((f.skip_pq && blk == 1) || col >= ns || (symmetric && col > row)) return;
    const int ks = f.ks[left], ks_r = f.ks[right];
    const long per = (long)ns * ns, ld = f.ld;
    double h[BT];
#pragma unroll
    for (int b = 0; b < BT; ++b) h[b] = 0.0;
    // the banded direct potential of source component src through this block's bra component
    auto direct = [&](int src, int k) {
        const int s = row > col ? row - col : col - row;
        if (s >= ks) return;
        const long at = (left ? f.q_off : 0) + (long)s * ns + (row < col ? row : col);
#pragma unroll
        for (int b = 0; b < BT; ++b)
            h[b] = add(h[b], __ldg(f.v + (((long)src * f.nk + k) * f.nt + min(t0 + b, f.nt - 1)) * ld + at));
    };
    if (blk == 3)
        for (int k = 0; k < f.nk; ++k) direct(0, k);
    for (int k = 0; k < f.nk; ++k) {
        if (symmetric) direct(left, k);
        const double *Kb = f.K[k] + (left ? f.q_off * ld : 0) + (right ? f.q_off : 0) + col;
        const double *d[BT];
        double s[BT];
#pragma unroll
        for (int b = 0; b < BT; ++b) {
            d[b] = f.xx + (((long)blk * f.nk + k) * f.nt + min(t0 + b, f.nt - 1)) * per + col;
            s[b] = 0.0;
        }
        // one step: density entry (i, col + off), bank element of the left pair of i and row
        auto step = [&](int i, int jp, int off) {
            if (col + off < 0 || col + off >= ns) return;
            const int ip = row >= i ? row - i : i - row;
            const double kv = __ldg(Kb + ((long)ip * ns + min(i, row)) * ld + (long)jp * ns + min(off, 0));
#pragma unroll
            for (int b = 0; b < BT; ++b) s[b] = add(s[b], mul(kv, __ldg(d[b] + (long)i * ns + off)));
        };
        const int i_lo = max(row - ks + 1, 0), i_hi = min(row + ks - 1, ns - 1);
        for (int i = row; i >= i_lo; --i)
#pragma unroll 2
            for (int jp = 0; jp < ks_r; ++jp) step(i, jp, jp);
        for (int i = row + 1; i <= i_hi; ++i)
#pragma unroll 2
            for (int jp = 0; jp < ks_r; ++jp) step(i, jp, jp);
        for (int jp = 1; jp < ks_r; ++jp)
#pragma unroll 2
            for (int i = row; i >= i_lo; --i) step(i, jp, -jp);
        for (int i = row + 1; i <= i_hi; ++i)
#pragma unroll 2
            for (int jp = 1; jp < ks_r; ++jp) step(i, jp, -jp);
#pragma unroll
        for (int b = 0; b < BT; ++b) h[b] = add(h[b], s[b]);
    }
    if (blk == 0)
        for (int k = 0; k < f.nk; ++k) direct(1, k);
    const int slot = blk == 0 ? 0 : blk == 1 ? 2 : blk == 2 ? 3 : 1;
#pragma unroll
    for (int b = 0; b < BT; ++b)
        if (t0 + b < f.nt) {
            double *o = f.h + ((long)(t0 + b) * 4 + slot) * per;
            o[(long)row * ns + col] = h[b];
            if (symmetric && col < row) o[(long)col * ns + row] = h[b];
        }
}

}  // namespace cell
}  // namespace rkb

using namespace rkb;

// ----------------------------------------------------------------- host side
namespace {
inline unsigned blocks_for(long n, int threads = 256) { return (unsigned)ceil_div(n, threads); }
}

extern "C" void rkb_gauss_legendre_01(int n, double *x, double *w) {
    if (n == 1) {
        x[0] = 0.5;
        w[0] = 1.0;
        return;
    }
    // Newton's iteration on the Legendre three-term recurrence from the
    // Chebyshev-like guess cos(pi (i + 3/4) / (n + 1/2)), then mapped to [0, 1]
    const double pi = 3.14159265358979323846;
    for (int i = 0; i < n; ++i) {
        double xi = std::cos(pi * (i + 0.75) / (n + 0.5)), p0 = 1.0, p1 = xi, dp = 0.0;
        for (int it = 0; it < 50; ++it) {
            p0 = 1.0;
            p1 = xi;
            for (int j = 2; j <= n; ++j) {
                const double p2 = ((2 * j - 1) * xi * p1 - (j - 1) * p0) / j;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (xi * p1 - p0) / (xi * xi - 1.0);
            const double dx = p1 / dp;
            xi -= dx;
            if (std::fabs(dx) < 1e-15) break;
        }
        x[i] = 0.5 * (xi + 1.0);
        w[i] = 1.0 / ((1.0 - xi * xi) * dp * dp);
    }
}

extern "C" int rkb_cell_moments(const double *d_bsp, const double *d_gr, const double *d_grw, int nv, int ng, int ks,
                                int k, double *d_out, void *stream) {
    RKB_CHECK_ARG(nv >= 1 && ng >= 1 && ng <= RKB_MAX_NG && ks >= 1 && ks <= cell::MAX_KS, "invalid basis sizes");
    RKB_CHECK_ARG(k >= -64 && k <= 64, "multipole power out of range (%d)", k);
    const long n = (long)ks * (ks + 1) / 2 * nv;
    cell::moments_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_bsp, d_gr, d_grw, nv, ng, ks, k, d_out);
    RKB_LAUNCHED("cell::moments_kernel");
    return RKB_OK;
}

static size_t diag_smem(int ng, int n_sub, int ks_l, int ks_r) {
    const int ksm = ks_l > ks_r ? ks_l : ks_r;
    const long kkl = ks_l * (ks_l + 1) / 2, kkr = ks_r * (ks_r + 1) / 2, kkm = ksm * (ksm + 1) / 2;
    return sizeof(double) * ((size_t)ng * n_sub * ksm + (size_t)ng * n_sub + ng + 2 * kkm * ng + 2 * kkl * kkr);
}

extern "C" int rkb_cell_diag(const double *d_bsp_l, const double *d_bsp_r, const double *d_gr, const double *d_grw,
                             const double *d_t_l, const double *d_t_r, int nv, int ng, int ks_l, int ks_r, int same,
                             int k, const double *d_x01, const double *d_w01, int n_sub, double *d_out, void *stream) {
    RKB_CHECK_ARG(nv >= 1 && ng >= 1 && ng <= RKB_MAX_NG, "invalid grid");
    RKB_CHECK_ARG(ks_l >= 1 && ks_l <= cell::MAX_KS && ks_r >= 1 && ks_r <= cell::MAX_KS, "orders must be 1..%d",
                  cell::MAX_KS);
    RKB_CHECK_ARG(n_sub >= 1 && n_sub <= cell::MAX_NSUB, "sub-quadrature order must be 1..%d", cell::MAX_NSUB);
    RKB_CHECK_ARG(k >= 0 && k <= 64, "multipole rank must be in [0, 64] (got %d)", k);
    RKB_CHECK_ARG(!same || ks_l == ks_r, "a same-component cell needs equal orders");
    const size_t smem = diag_smem(ng, n_sub, ks_l, ks_r);
    RKB_CHECK_ARG(smem <= 200 * 1024, "diagonal-cell workspace too large (%zu bytes)", smem);
    RKB_CUDA(set_smem(cell::diag_kernel, (int)smem));
    cell::diag_kernel<<<(unsigned)nv, 256, smem, as_stream(stream)>>>(d_bsp_l, d_bsp_r, d_gr, d_grw, d_t_l, d_t_r, nv,
                                                                       ng, ks_l, ks_r, same, k, n_sub, d_x01, d_w01,
                                                                       d_out);
    RKB_LAUNCHED("cell::diag_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_assemble(const double *d_rising_l, const double *d_falling_l, const double *d_rising_r,
                                 const double *d_falling_r, const double *d_diag, int nv, int ks_l, int ks_r, int ns,
                                 double *d_out, long ld, long row_off, long col_off, void *stream) {
    RKB_CHECK_ARG(nv >= 1 && ns >= 1 && ks_l >= 1 && ks_l <= cell::MAX_KS && ks_r >= 1 && ks_r <= cell::MAX_KS,
                  "invalid bank sizes");
    RKB_CHECK_ARG(row_off >= 0 && col_off >= 0 && ld >= col_off + (long)ks_r * ns, "bank block outside the matrix");
    const long n = (long)ks_l * ns * ks_r * ns;
    cell::assemble_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_rising_l, d_falling_l, d_rising_r,
                                                                        d_falling_r, d_diag, nv, ks_l, ks_r, ns, d_out,
                                                                        ld, row_off, col_off);
    RKB_LAUNCHED("cell::assemble_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_densities(const double *d_c1, const double *d_c2, long ld, const long *d_pairs, long n_pairs,
                                  int n1, int n2, int ns_d, int ns_k, int ks, double *d_out, long out_ld, long col_off,
                                  void *stream) {
    RKB_CHECK_ARG(n1 >= 0 && n2 >= 0 && n1 <= ld && n2 <= ld && ns_d >= 1 && ns_d <= ns_k && ks >= 1,
                  "invalid density sizes");
    RKB_CHECK_ARG(col_off >= 0 && out_ld >= col_off + (long)ks * ns_k, "density block outside the row");
    if (n_pairs == 0) return RKB_OK;
    const long n = n_pairs * ks * ns_k;
    cell::densities_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_c1, d_c2, ld, d_pairs, n_pairs, n1, n2,
                                                                         ns_d, ns_k, ks, d_out, out_ld, col_off);
    RKB_LAUNCHED("cell::densities_kernel");
    return RKB_OK;
}

extern "C" int rkb_gemm_nt_fp64(const double *d_A, long lda, const double *d_B, long ldb, double *d_C, long ldc,
                                long M, long N, long K, int accumulate, void *stream) {
    RKB_CHECK_ARG(M >= 0 && N >= 0 && K >= 0 && K % dgemm::BK == 0, "K (%ld) must be a multiple of %d", K, dgemm::BK);
    RKB_CHECK_ARG(lda >= K && ldb >= K && ldc >= N && lda % 2 == 0 && ldb % 2 == 0,
                  "leading dimensions must cover the matrices (and lda, ldb be even)");
    RKB_CHECK_ARG(((uintptr_t)d_A % 16) == 0 && ((uintptr_t)d_B % 16) == 0, "A and B must be 16-byte aligned");
    if (M == 0 || N == 0) return RKB_OK;
    const long tiles = ceil_div(M, dgemm::Tile64::SIDE) * ceil_div(N, dgemm::Tile64::SIDE);
    RKB_CHECK_ARG(tiles < (1L << 31), "result too large (%ld x %ld)", M, N);
    auto launch = [&](auto tile) {
        using T = decltype(tile);
        RKB_CUDA(set_smem(cell::gemm_nt_kernel<T>, (int)T::SMEM));
        cell::gemm_nt_kernel<T><<<(unsigned)(ceil_div(M, T::SIDE) * ceil_div(N, T::SIDE)), dgemm::THREADS, T::SMEM,
                                  as_stream(stream)>>>(d_A, lda, d_B, ldb, d_C, ldc, M, N, K, accumulate);
        return (int)RKB_OK;
    };
    const int st = dgemm::small_problem(tiles) ? launch(dgemm::Tile32()) : launch(dgemm::Tile64());
    if (st) return st;
    RKB_LAUNCHED("cell::gemm_nt_kernel");
    return RKB_OK;
}

extern "C" int rkb_gemm_nt_fp64_groups(const double *d_A, long lda, const void *const *B, const long *row0, int n_groups,
                                       long ldb, double *d_C, long ldc, long N, long K, void *stream) {
    RKB_CHECK_ARG(n_groups >= 0 && N >= 0 && K >= 0 && K % dgemm::BK == 0, "K (%ld) must be a multiple of %d", K,
                  dgemm::BK);
    RKB_CHECK_ARG(lda >= K && ldb >= K && ldc >= N && lda % 2 == 0 && ldb % 2 == 0,
                  "leading dimensions must cover the matrices (and lda, ldb be even)");
    RKB_CHECK_ARG(((uintptr_t)d_A % 16) == 0, "A must be 16-byte aligned");
    long rows = 0;
    for (int q = 0; q < n_groups; ++q) {
        RKB_CHECK_ARG(row0[q + 1] >= row0[q] && ((uintptr_t)B[q] % 16) == 0,
                      "row ranges must ascend and every B be 16-byte aligned");
        rows += ceil_div(row0[q + 1] - row0[q], dgemm::Tile64::SIDE);
    }
    if (rows == 0 || N == 0) return RKB_OK;
    RKB_CHECK_ARG(rows * ceil_div(N, dgemm::Tile64::SIDE) < (1L << 29), "result too large");
    auto launch = [&](auto tile) {
        using T = decltype(tile);
        RKB_CUDA(set_smem(cell::gemm_nt_groups_kernel<T>, (int)T::SMEM));
        for (int q0 = 0; q0 < n_groups; q0 += cell::MAX_GROUPS) {
            cell::GroupArgs g = {};
            g.n = n_groups - q0 < cell::MAX_GROUPS ? n_groups - q0 : cell::MAX_GROUPS;
            for (int q = 0; q < g.n; ++q) {
                g.B[q] = static_cast<const double *>(B[q0 + q]);
                g.row0[q] = row0[q0 + q];
                g.tile0[q + 1] = g.tile0[q] + ceil_div(row0[q0 + q + 1] - row0[q0 + q], T::SIDE) * ceil_div(N, T::SIDE);
            }
            g.row0[g.n] = row0[q0 + g.n];
            if (g.tile0[g.n] == 0) continue;
            cell::gemm_nt_groups_kernel<T><<<(unsigned)g.tile0[g.n], dgemm::THREADS, T::SMEM, as_stream(stream)>>>(
                d_A, lda, g, ldb, d_C, ldc, N, K);
            RKB_LAUNCHED("cell::gemm_nt_groups_kernel");
        }
        return (int)RKB_OK;
    };
    return dgemm::small_problem(rows * ceil_div(N, dgemm::Tile64::SIDE)) ? launch(dgemm::Tile32())
                                                                        : launch(dgemm::Tile64());
}

extern "C" int rkb_cell_dots(const double *d_L, long l_ld, const double *d_W, long w_ld, long n, const long *d_il,
                             const long *d_iw, long n_ent, double *d_out, void *stream) {
    RKB_CHECK_ARG(n >= 0 && l_ld >= n && w_ld >= n, "invalid sizes");
    if (n_ent == 0) return RKB_OK;
    cell::dots_kernel<<<(unsigned)ceil_div(n_ent, 8), 256, 0, as_stream(stream)>>>(d_L, l_ld, d_W, w_ld, n, d_il,
                                                                                  d_iw, n_ent, d_out);
    RKB_LAUNCHED("cell::dots_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_exchange(const double *d_K, long ld, const long *d_kofs, const double *d_dens, long nbatch,
                                 int ns, int ks_l, int ks_r, int symmetric, int accumulate, double *d_out,
                                 void *stream) {
    RKB_CHECK_ARG(ns >= 1 && ks_l >= 1 && ks_r >= 1 && ld >= (long)ks_r * ns, "invalid sizes");
    RKB_CHECK_ARG(!symmetric || ks_l == ks_r, "a symmetric exchange needs equal orders");
    if (nbatch == 0) return RKB_OK;
    const long n = (long)ns * ns * nbatch;
    cell::exchange_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_K, ld, d_kofs, d_dens, ns, ks_l, ks_r,
                                                                        symmetric, accumulate, d_out, nbatch);
    RKB_LAUNCHED("cell::exchange_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_bilinear(const double *d_K, long ld, int ns, const double *d_wa, const double *d_wb,
                                 int n_left, int n_right, int ks_l, int ks_r, int ns_out, double *d_T, double *d_M,
                                 void *stream) {
    RKB_CHECK_ARG(ns >= 1 && n_left >= 0 && n_left <= ns && n_right >= 0 && n_right <= ns && ns_out >= n_left &&
                      ns_out >= n_right && ld >= (long)ks_r * ns,
                  "invalid bilinear sizes");
    const long nt = (long)ns_out * n_right * ks_r, nm = (long)ns_out * ns_out;
    if (nt > 0) {
        cell::bilinear_t_kernel<<<blocks_for(nt), 256, 0, as_stream(stream)>>>(d_K, ld, ns, d_wa, n_left, n_right,
                                                                               ks_l, ks_r, ns_out, d_T);
        RKB_LAUNCHED("cell::bilinear_t_kernel");
    }
    if (nm > 0) {
        cell::bilinear_m_kernel<<<blocks_for(nm), 256, 0, as_stream(stream)>>>(d_T, d_wb, n_right, ks_r, ns_out, d_M);
        RKB_LAUNCHED("cell::bilinear_m_kernel");
    }
    return RKB_OK;
}

extern "C" int rkb_cell_direct_density(const double *d_comp, long ld, int n_orb, const double *d_coef,
                                       long coef_stride, const int *d_target, long nbatch, int ns, int ks,
                                       double *d_out, long out_ld, void *stream) {
    RKB_CHECK_ARG(ns >= 1 && ks >= 1 && ld >= ns && n_orb >= 0 && out_ld >= (long)ks * ns, "invalid sizes");
    if (nbatch == 0) return RKB_OK;
    const long n = (long)ns * ks * nbatch;
    cell::direct_density_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_comp, ld, n_orb, d_coef, coef_stride,
                                                                              d_target, ns, ks, d_out, out_ld, nbatch);
    RKB_LAUNCHED("cell::direct_density_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_exchange_density(const double *d_comp_ii, const double *d_comp_jj, long ld, int n_orb,
                                         const double *d_coef, long coef_stride, long nbatch, int ns, double *d_out,
                                         void *stream) {
    RKB_CHECK_ARG(ns >= 1 && ld >= ns && n_orb >= 0, "invalid sizes");
    if (nbatch == 0) return RKB_OK;
    const long n = (long)ns * ns * nbatch;
    cell::exchange_density_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_comp_ii, d_comp_jj, ld, n_orb,
                                                                                d_coef, coef_stride, ns, d_out,
                                                                                nbatch);
    RKB_LAUNCHED("cell::exchange_density_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_banded_to_full(const double *d_v, int ns, int ks, long nbatch, double *d_V, void *stream) {
    RKB_CHECK_ARG(ns >= 1 && ks >= 1, "invalid sizes");
    if (nbatch == 0) return RKB_OK;
    const long n = (long)ns * ks * nbatch;
    cell::banded_to_full_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_v, ns, ks, d_V, nbatch);
    RKB_LAUNCHED("cell::banded_to_full_kernel");
    return RKB_OK;
}

extern "C" int rkb_cell_fock_finish(const double *d_h, const double *d_norm, int ns, int skip_pq, long nbatch,
                                    double *d_out, void *stream) {
    RKB_CHECK_ARG(ns >= 1 && d_h != d_out, "invalid sizes (the output must not alias the input)");
    if (nbatch == 0) return RKB_OK;
    const long n = (long)ns * ns * nbatch;
    cell::fock_finish_kernel<<<blocks_for(n), 256, 0, as_stream(stream)>>>(d_h, d_norm, ns, skip_pq, d_out, nbatch);
    RKB_LAUNCHED("cell::fock_finish_kernel");
    return RKB_OK;
}

extern "C" int rkb_fock_blocks(const void *const *K, const void *d_K, long ld, long q_off, int nk, int ns, int ks_p,
                               int ks_q, const double *d_P, const double *d_Q, long c_ld, int n_orb,
                               const double *d_ad, const double *d_ax, const int *d_target, int nt,
                               const double *d_norm, int skip_pq, double *d_dd, long dd_ld, double *d_v, double *d_xx,
                               double *d_h, double *d_out, void *stream) {
    RKB_CHECK_ARG(ns >= 1 && nk >= 0 && nt >= 0 && n_orb >= 0 && ks_p >= 1 && ks_q >= 1, "invalid sizes");
    RKB_CHECK_ARG(q_off >= (long)ks_p * ns && ld >= q_off + (long)ks_q * ns && c_ld >= ns,
                  "leading dimensions must cover the blocks");
    RKB_CHECK_ARG(dd_ld % dgemm::BK == 0 && q_off % dgemm::BK == 0 && (ld - q_off) % dgemm::BK == 0 &&
                      dd_ld >= q_off && dd_ld >= ld - q_off,
                  "block widths must be multiples of %d, and dd_ld cover them", dgemm::BK);
    RKB_CHECK_ARG((long)4 * nk * nt <= 65535 && ns <= 65535, "too many targets and multipoles (%d x %d)", nt,
                  nk);
    RKB_CHECK_ARG(d_h != d_out, "the output must not alias the blocks");
    if (nt == 0) return RKB_OK;
    cudaStream_t st = as_stream(stream);
    const long per = (long)ns * ns;
    RKB_CUDA(cudaMemsetAsync(d_h, 0, sizeof(double) * 4 * per * nt, st));
    if (nk > 0) {
        cell::FockArgs f = {};
        f.K = static_cast<const double *const *>(d_K);
        f.ld = ld; f.q_off = q_off; f.nk = nk; f.nt = nt; f.n_orb = n_orb; f.ns = ns; f.ks[0] = ks_p; f.ks[1] = ks_q;
        f.comp[0] = d_P; f.comp[1] = d_Q; f.c_ld = c_ld; f.ad = d_ad; f.ax = d_ax; f.target = d_target;
        f.dd = d_dd; f.dd_ld = dd_ld; f.v = d_v; f.xx = d_xx; f.h = d_h; f.skip_pq = skip_pq;
        cell::fock_direct_density_kernel<<<dim3(blocks_for(dd_ld), 2u * nk * nt), 256, 0, st>>>(f);
        RKB_LAUNCHED("cell::fock_direct_density_kernel");
        for (int src = 0; src < 2; ++src)
            for (int k0 = 0; k0 < nk; k0 += cell::MAX_GROUPS) {
                const int m = nk - k0 < cell::MAX_GROUPS ? nk - k0 : cell::MAX_GROUPS;
                const void *Bk[cell::MAX_GROUPS];
                long rows[cell::MAX_GROUPS + 1];
                for (int k = 0; k <= m; ++k) rows[k] = ((long)src * nk + k0 + k) * nt;
                for (int k = 0; k < m; ++k) Bk[k] = static_cast<const double *>(K[k0 + k]) + (src ? q_off : 0);
                const int rc = rkb_gemm_nt_fp64_groups(d_dd, dd_ld, Bk, rows, m, ld, d_v, ld, ld,
                                                       src ? ld - q_off : q_off, stream);
                if (rc != RKB_OK) return rc;
            }
        cell::fock_exchange_density_kernel<<<dim3(blocks_for(per), 4u * nk * nt), 256, 0, st>>>(f);
        RKB_LAUNCHED("cell::fock_exchange_density_kernel");
        constexpr int BT = 8;
        cell::fock_exchange_kernel<BT><<<dim3((unsigned)ceil_div(ns, cell::FOCK_THREADS), (unsigned)ns,
                                              4u * (unsigned)ceil_div(nt, BT)), cell::FOCK_THREADS, 0, st>>>(f);
        RKB_LAUNCHED("cell::fock_exchange_kernel");
    }
    cell::fock_finish_kernel<<<blocks_for(per * nt), 256, 0, st>>>(d_h, d_norm, ns, skip_pq, d_out, nt);
    RKB_LAUNCHED("cell::fock_finish_kernel");
    return RKB_OK;
}
