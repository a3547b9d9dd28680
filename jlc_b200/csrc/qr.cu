// Blocked Householder QR kept on the device: the kernels around the GEMM
// route.  Follows the reference's blocked factorisation on the column-major
// matrix (HouseholderQR.java:133-210, 215-343): panels of 64 columns are
// factored column by column (max-normalised Householder vectors, each applied
// to the panel's later columns), then the trailing columns are updated with
// the compact-WY form Q^T C = C - (V T^T) (V^T C) as two GEMMs (api.cu).
//
//   qr_panel_rg_kernel: the panel on one thread-block cluster (1..16 CTAs),
//                      the rows held in registers; panels of up to 4096 rows;
//   qr_panel_cl_kernel: the same with the rows in shared memory and one
//                      cluster barrier per column; panels of up to 6400 rows;
//   qr_panel_sm_kernel / qr_panel_mp_kernel: taller panels on a cooperative
//                      grid of up to one CTA per SM, slabs in shared memory
//                      or (taller still) in place, one grid barrier per column;
//                      all merge partials in a fixed order, so the
//                      factorisation is deterministic;
//   qr_vt_kernel:      V = the panel's reflectors with unit diagonal and zeros
//                      above it (packV, HouseholderQR.java:445-471) and the T
//                      of their compact-WY form (buildT, :300-325), one cluster
//                      per panel, any number of panels per launch;
//   qr_vt_product_kernel: V T or V T^T, so that a block reflector is applied in
//                      two GEMMs;
//   qr_pack_v_kernel, qr_gram_partial_kernel / qr_gram_sum_kernel,
//   qr_build_t_kernel: V and T of panels above 4096 rows, V^T V over row slabs
//                      on the whole grid.
#include <cfloat>
#include <cmath>

#include <cooperative_groups.h>
#include <math_constants.h>

#include "jlc_device.cuh"
#include "jlc_dmma.cuh"
#include "jlc_internal.h"
#include "jlc_slab.cuh"

namespace jlc {
namespace qr {

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ------------------------------------------------------------ multi-CTA panel
// The panel factorisation (computeHouseholder / applyHouseholderToColumn,
// HouseholderQR.java:219-384) with the panel's rows split over the CTAs of one
// cooperative launch (CTA c owns rows [k0 + c R, k0 + (c+1) R)).  Per column
// k, one pass per CTA over its rows gives the column's local max, its scaled
// sum of squares (scale, ssq) and its dots with the panel's later columns
// (with the column still unscaled); one grid barrier; every CTA combines the
// CTAs' partials in CTA order (the same result everywhere, and the same bits
// on every run), forms beta, tau and 1/(x0 - beta) as the reference does
// (sigma = (scale/max)^2 ssq, dot_j = (a_kj + sum_i x_i a_ij / (x0 - beta))
// tau), then scales and updates its own rows.  Row k's entries reach the
// other CTAs through a row record written by its owner before the barrier;
// partial and row records alternate between two buffers by column parity,
// so one barrier per column is enough.
constexpr int MP_THREADS = 256, MP_WARPS = MP_THREADS / 32;
constexpr int MP_PART = 72;  // per CTA and column: max, scale, ssq, dots with up to 63 later columns


// (scale, ssq) pairs: sum of squares = scale^2 * ssq, combined without overflow
__device__ __forceinline__ void ssq_add(double& scale, double& ssq, double x) {
    const double a = fabs(x);
    if (a == 0.0) return;
    if (a > scale) {
        const double r = scale / a;
        ssq = 1.0 + ssq * r * r;
        scale = a;
    } else {
        const double r = a / scale;
        ssq += r * r;
    }
}
__device__ __forceinline__ void ssq_merge(double& scale, double& ssq, double s2, double q2) {
    if (s2 == 0.0) return;
    if (s2 > scale) {
        const double r = scale / s2;
        ssq = q2 + ssq * r * r;
        scale = s2;
    } else {
        const double r = s2 / scale;
        ssq += q2 * r * r;
    }
}

// Power-of-two scaling shared by the panels: a column's values are scaled by
// 2^-e, e the exponent of a maximum, before squares and dots are formed, so
// nothing overflows or underflows whatever the input's range; sums carried in
// units of 2^e (dots) or 4^e (squares) are rescaled exactly.
constexpr double SP_EMPTY_EXP = -4096.0;  // exponent of an empty partial

// exponent e with 2^e <= x < 2^(e+1) for a positive normal x, clamped to [-1000, 1000]
__device__ __forceinline__ int sp_exp(double x) {
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return x > 0.0 && ex != 0x7ff ? min(1000, max(-1000, ex - 1023)) : 0;
}
__device__ __forceinline__ double sp_pow2(int e) {  // 2^e, -1022 <= e <= 1023
    return __longlong_as_double((long long)(e + 1023) << 52);
}
// s * 2^d for d <= 0 (flushed to zero below d = -2044, where the term is negligible)
__device__ __forceinline__ double sp_scale(double s, int d) {
    if (d >= -1022) return s * sp_pow2(d);
    if (d >= -2044) return (s * sp_pow2(-1022)) * sp_pow2(d + 1022);
    return 0.0;
}
// (e, s) += (e2, s2), both sums of squares in units of 4^e
__device__ __forceinline__ void sp_merge(double& e, double& s, double e2, double s2) {
    const double E = fmax(e, e2);
    s = sp_scale(s, 2 * (int)(e - E)) + sp_scale(s2, 2 * (int)(e2 - E));
    e = E;
}

__global__ void __launch_bounds__(MP_THREADS) qr_panel_mp_kernel(double* A, long long lda, int m, int k0, int kb,
                                                                 double* tau, double* part, double* rowrec,
                                                                 unsigned* counter, int* status) {
    __shared__ double fin[64];  // fin[0] = tau, fin[t] = dot_t for the later columns
    __shared__ double fin_v0inv, fin_v0s, fin_beta;
    __shared__ int fin_e;
    __shared__ int fin_mode;  // 0: no reflector, 1: reflector, 2: sign flip (tau = 2)
    __shared__ int s_ok;
    const int P = gridDim.x, cta = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = (m - k0 + P - 1) / P;
    const int r0 = k0 + cta * R, r1 = min(m, r0 + R);
    for (int kk = 0; kk < kb; ++kk) {
        const int k = k0 + kk;
        const int later = kb - kk - 1;  // columns k+1 .. k0+kb-1
        const double* colk = A + (long long)k * lda;
        double* pk = part + ((size_t)(kk & 1) * P + cta) * MP_PART;
        double* rk = rowrec + (size_t)(kk & 1) * 64;
        // Phase A: this CTA's rows -- task 0 the column's max and (scale, ssq)
        // over rows > k, task t >= 1 the dot of column k with column k + t
        const int lo = max(r0, k), lo1 = max(r0, k + 1);
        // the dots use x 2^-e, e the exponent of this CTA's max of column k
        // (every warp finds the same max)
        double cmx = 0.0;
        for (int i = lo + lane; i < r1; i += 32) cmx = fmax(cmx, fabs(colk[i]));
        cmx = warp_max(cmx);
        const double csc = sp_pow2(-sp_exp(cmx));
        for (int t = warp; t <= later; t += MP_WARPS) {
            if (t == 0) {
                double mx = 0.0, sc = 0.0, sq = 0.0;
                for (int i = lo + lane; i < r1; i += 32) {
                    const double x = colk[i];
                    mx = fmax(mx, fabs(x));
                    if (i > k) ssq_add(sc, sq, x);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                    const double s2 = __shfl_xor_sync(0xffffffffu, sc, o);
                    const double q2 = __shfl_xor_sync(0xffffffffu, sq, o);
                    // merge in a fixed orientation so both lanes of a pair hold the same result
                    double a_s = (lane & o) ? s2 : sc, a_q = (lane & o) ? q2 : sq;
                    const double b_s = (lane & o) ? sc : s2, b_q = (lane & o) ? sq : q2;
                    ssq_merge(a_s, a_q, b_s, b_q);
                    sc = a_s;
                    sq = a_q;
                }
                if (lane == 0) {
                    pk[0] = mx;
                    pk[1] = sc;
                    pk[2] = sq;
                }
            } else {
                const double* cj = A + (long long)(k + t) * lda;
                double d = 0.0;
                for (int i = lo1 + lane; i < r1; i += 32) d = fma(colk[i] * csc, cj[i], d);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                if (lane == 0) pk[2 + t] = d;
            }
        }
        // row k (its owner): x0 and the later columns' entries on row k
        if (k >= r0 && k < r1)
            for (int t = tid; t <= later; t += MP_THREADS) rk[t] = A[(long long)(k + t) * lda + k];
        if (!grid_barrier(counter, (unsigned)(kk + 1) * (unsigned)P, status, &s_ok)) return;
        // Phase B: combine the CTAs' partials in CTA order
        const double* pb = part + (size_t)(kk & 1) * P * MP_PART;
        if (tid == 0) {
            fin_mode = 0;
            if (m - k > 1) {
                double mx = 0.0, sc = 0.0, sq = 0.0;
                for (int q = 0; q < P; ++q) {
                    mx = fmax(mx, pb[q * MP_PART]);
                    ssq_merge(sc, sq, pb[q * MP_PART + 1], pb[q * MP_PART + 2]);
                }
                if (mx >= DBL_MIN) {
                    const double inv = 1.0 / mx;  // as the reference: x * (1/max)
                    const double x0 = rk[0] * inv;
                    const double r = sc * inv;
                    const double xnorm = sqrt(r * r * sq);
                    if (xnorm == 0.0) {
                        if (x0 < 0.0) fin_mode = 2;
                    } else {
                        const double nb = -copysign(hypot(x0, xnorm), x0);
                        fin_mode = 1;
                        fin_beta = nb * mx;
                        fin_v0inv = 1.0 / ((x0 - nb) * mx);
                        fin_e = sp_exp(mx);
                        fin_v0s = (inv * sp_pow2(fin_e)) / (x0 - nb);  // 2^E / ((x0 - beta) max), O(1)
                        fin[0] = (nb - x0) / nb;  // tau
                    }
                }
            }
        }
        __syncthreads();
        const int mode = fin_mode;
        const double tk = mode == 1 ? fin[0] : (mode == 2 ? 2.0 : 0.0);
        if (mode == 1) {
            const int E = fin_e;
            for (int t = 1 + tid; t <= later; t += MP_THREADS) {
                double d = 0.0;  // CTA q's dot is in units of 2^e_q, brought to 2^E
                for (int q = 0; q < P; ++q) {
                    const double mq = pb[q * MP_PART];
                    if (mq > 0.0) d += sp_scale(pb[q * MP_PART + 2 + t], sp_exp(mq) - E);
                }
                fin[t] = (rk[t] + d * fin_v0s) * tk;
            }
        } else if (mode == 2) {
            for (int t = 1 + tid; t <= later; t += MP_THREADS) fin[t] = rk[t] * 2.0;  // the tail is zero
        }
        if (cta == 0 && tid == 0) tau[k] = tk;
        __syncthreads();
        if (mode != 0) {
            // Phase C: reflector tail on this CTA's rows, then the later columns
            const int nrows = r1 - lo1;
            if (mode == 1) {
                double* ck = A + (long long)k * lda;
                for (int i = lo1 + tid; i < r1; i += MP_THREADS) ck[i] *= fin_v0inv;
            }
            if (k >= r0 && k < r1 && tid == 0) {
                double* ck = A + (long long)k * lda;
                ck[k] = mode == 1 ? fin_beta : -ck[k];
            }
            __syncthreads();
            if (nrows > 0) {
                for (int e = tid; e < nrows * later; e += MP_THREADS) {
                    const int i = lo1 + e % nrows, t = 1 + e / nrows;
                    A[(long long)(k + t) * lda + i] -= fin[t] * colk[i];
                }
            }
            if (k >= r0 && k < r1)
                for (int t = 1 + tid; t <= later; t += MP_THREADS) A[(long long)(k + t) * lda + k] -= fin[t];
        }
        __syncthreads();
    }
}

// The multi-CTA panel with each CTA's rows held in shared memory for the
// whole panel (slab = kb columns x R rows, column-major, loaded once and
// written back once), so the per-column passes touch no global memory but
// the partials.  The column's sum of squares is kept as (e, s) with
// sum = s * 4^e, e a power-of-two exponent taken from a maximum (clamped to
// +-1000 so that 2^-e is a normal number): every rescaling is exact, and the
// merge needs no division.  The partials are laid out by quantity
// (part[q][cta]); warp lanes merge them in a fixed order (lane l takes CTAs
// l, l+32, ..., then a butterfly), so every CTA derives the same bits.
constexpr int SP_MAX_SLAB_BYTES = 200 * 1024;
constexpr int SP_MAX_CTAS = 160;                    // partial loads: up to 5 per lane
constexpr int SP_TASKS = 64 / MP_WARPS;             // later columns per warp

__global__ void __launch_bounds__(MP_THREADS) qr_panel_sm_kernel(double* A, long long lda, int m, int k0, int kb,
                                                                 double* tau, double* part, double* rowrec,
                                                                 unsigned* counter, int* status) {
    extern __shared__ double slab[];  // slab[c * R + (i - r0)] = A[i, k0 + c]
    __shared__ double fin[64];
    __shared__ double fin_v0inv, fin_v0s, fin_beta, fin_tau;
    __shared__ int fin_mode;
    __shared__ int s_ok;
    const int P = gridDim.x, cta = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = (m - k0 + P - 1) / P;
    const int r0 = k0 + cta * R, r1 = min(m, r0 + R);
    const int rows = max(0, r1 - r0);
    for (int e = tid; e < rows * kb; e += MP_THREADS) {
        const int c = e / rows, i = e - c * rows;
        slab[c * R + i] = A[(long long)(k0 + c) * lda + r0 + i];
    }
    __syncthreads();
    for (int kk = 0; kk < kb; ++kk) {
        const int k = k0 + kk;
        const int later = kb - kk - 1;
        double* ck = slab + kk * R;  // ck[i - r0] = A[i, k] for own rows i
        double* pk = part + (size_t)(kk & 1) * MP_PART * P + cta;
        double* rk = rowrec + (size_t)(kk & 1) * 64;
        const int lo = max(r0, k), lo1 = max(r0, k + 1);
        // Phase A: every warp the max of column k over own rows >= k and its
        // exponent e; warp w the dots of x 2^-e with the later columns
        // t = 1 + w + 8j (all j together); the last warp also the sum of
        // squares over rows > k
        {
            double mx = 0.0;
            for (int i = lo + lane; i < r1; i += 32) mx = fmax(mx, fabs(ck[i - r0]));
            mx = warp_max(mx);
            const int e = sp_exp(mx);
            const double sc = sp_pow2(-e);
            double d[SP_TASKS];
#pragma unroll
            for (int j = 0; j < SP_TASKS; ++j) d[j] = 0.0;
            for (int i = lo1 + lane; i < r1; i += 32) {
                const double x = ck[i - r0] * sc;
#pragma unroll
                for (int j = 0; j < SP_TASKS; ++j) {
                    const int t = 1 + warp + j * MP_WARPS;
                    if (t <= later) d[j] = fma(x, ck[t * R + (i - r0)], d[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < SP_TASKS; ++j) {
                const int t = 1 + warp + j * MP_WARPS;
                if (t <= later) {  // warp-uniform
                    const double v = warp_sum(d[j]);
                    if (lane == 0) pk[(2 + t) * P] = v;
                }
            }
            if (warp == MP_WARPS - 1) {
                double sq = 0.0;
                for (int i = lo1 + lane; i < r1; i += 32) {
                    const double y = ck[i - r0] * sc;
                    sq = fma(y, y, sq);
                }
                sq = warp_sum(sq);
                if (lane == 0) {
                    pk[0] = mx;
                    pk[P] = mx > 0.0 ? (double)e : SP_EMPTY_EXP;
                    pk[2 * P] = sq;
                }
            }
        }
        if (k >= r0 && k < r1)
            for (int t = tid; t <= later; t += MP_THREADS) rk[t] = ck[t * R + (k - r0)];
        if (!grid_barrier(counter, (unsigned)(kk + 1) * (unsigned)P, status, &s_ok)) return;
        // Phase B: merge the CTAs' partials (every CTA the same way).  All
        // loads are issued before any result is needed.
        const double* pb = part + (size_t)(kk & 1) * MP_PART * P;
        double dsum[SP_TASKS], rkv[SP_TASKS];
#pragma unroll
        for (int j = 0; j < SP_TASKS; ++j) {
            const int t = 1 + warp + j * MP_WARPS;
            dsum[j] = 0.0;
            rkv[j] = t <= later ? rk[t] : 0.0;
        }
        const double x0raw = rk[0];
        // CTA q's dots are in units of 2^e_q: each is brought to 2^E, E = max e_q
        double eqv[SP_MAX_CTAS / 32];
        double emax = SP_EMPTY_EXP;
#pragma unroll
        for (int c = 0; c < SP_MAX_CTAS / 32; ++c) {
            const int q = lane + 32 * c;
            eqv[c] = q < P ? pb[P + q] : SP_EMPTY_EXP;
            emax = fmax(emax, eqv[c]);
        }
        emax = warp_max(emax);
#pragma unroll
        for (int c = 0; c < SP_MAX_CTAS / 32; ++c) {
            const int q = lane + 32 * c;
            if (32 * c < P) {  // warp-uniform
#pragma unroll
                for (int j = 0; j < SP_TASKS; ++j) {
                    const int t = 1 + warp + j * MP_WARPS;
                    if (t <= later && q < P) dsum[j] += sp_scale(pb[(2 + t) * P + q], (int)(eqv[c] - emax));
                }
            }
        }
        if (warp == 0) {
            double mx = 0.0, e = SP_EMPTY_EXP, sq = 0.0;
#pragma unroll
            for (int c = 0; c < SP_MAX_CTAS / 32; ++c) {
                const int q = lane + 32 * c;
                if (q < P) {
                    mx = fmax(mx, pb[q]);
                    sp_merge(e, sq, pb[P + q], pb[2 * P + q]);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {  // the merge is symmetric: both lanes get the same bits
                mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const double e2 = __shfl_xor_sync(0xffffffffu, e, o);
                const double s2 = __shfl_xor_sync(0xffffffffu, sq, o);
                sp_merge(e, sq, e2, s2);
            }
            if (lane == 0) {
                int mode = 0;
                if (m - k > 1 && mx >= DBL_MIN) {
                    const double inv = 1.0 / mx;  // as the reference: x * (1/max)
                    const double x0 = x0raw * inv;
                    // sqrt(sum over rows > k of (x/max)^2) = sqrt(sq) 2^e / max, 2^e <= max
                    const double xnorm = sq > 0.0 ? sqrt(sq) * (inv * sp_pow2((int)e)) : 0.0;
                    if (xnorm == 0.0) {
                        if (x0 < 0.0) mode = 2;
                    } else {
                        const double nb = -copysign(hypot(x0, xnorm), x0);
                        mode = 1;
                        fin_beta = nb * mx;
                        fin_v0inv = 1.0 / ((x0 - nb) * mx);
                        fin_v0s = (inv * sp_pow2((int)e)) / (x0 - nb);  // 2^E / ((x0 - beta) max), O(1)
                        fin_tau = (nb - x0) / nb;
                    }
                }
                fin_mode = mode;
                if (cta == 0) tau[k] = mode == 1 ? fin_tau : (mode == 2 ? 2.0 : 0.0);
            }
        }
        __syncthreads();
        const int mode = fin_mode;
        if (mode == 1) {
            const double v0s = fin_v0s, tk = fin_tau;
#pragma unroll
            for (int j = 0; j < SP_TASKS; ++j) {
                const int t = 1 + warp + j * MP_WARPS;
                if (t <= later) {  // warp-uniform
                    const double d = warp_sum(dsum[j]);
                    if (lane == 0) fin[t] = (rkv[j] + d * v0s) * tk;
                }
            }
        } else if (mode == 2) {
            for (int t = 1 + tid; t <= later; t += MP_THREADS) fin[t] = rk[t] * 2.0;  // the tail is zero
        }
        __syncthreads();
        if (mode != 0) {
            // Phase C: reflector tail on own rows, then the later columns
            if (mode == 1) {
                const double v0inv = fin_v0inv;
                for (int i = lo1 + tid; i < r1; i += MP_THREADS) ck[i - r0] *= v0inv;
            }
            if (k >= r0 && k < r1 && tid == 0) ck[k - r0] = mode == 1 ? fin_beta : -ck[k - r0];
            __syncthreads();
            for (int t = 1 + warp; t <= later; t += MP_WARPS) {
                double* cj = ck + t * R;
                const double f = fin[t];
                for (int i = lo1 + lane; i < r1; i += 32) cj[i - r0] -= f * ck[i - r0];
                if (lane == 0 && k >= r0 && k < r1) cj[k - r0] -= f;
            }
        }
        __syncthreads();
    }
    for (int e = tid; e < rows * kb; e += MP_THREADS) {
        const int c = e / rows, i = e - c * rows;
        A[(long long)(k0 + c) * lda + r0 + i] = slab[c * R + i];
    }
}

// The panel on one thread-block cluster (1..16 CTAs, one slab of rows each in
// shared memory).  Each CTA stores its partials (and the CTA holding row k
// the row record) straight into every CTA's shared memory, lane r to CTA r;
// the stores complete under the cluster barrier's release, so after it every
// CTA merges from its own shared memory.  The barrier is the hardware cluster
// barrier (release/acquire), so nothing spins on memory.  Partials and row
// records alternate between two buffers by column parity: a CTA writes
// column k+1's while a slower one may still read column k's, and overwrites
// column k's only after the next barrier.
namespace cg = cooperative_groups;
constexpr int CL_THREADS = 512, CL_WARPS = CL_THREADS / 32;
constexpr int CL_TASKS = 64 / CL_WARPS;  // later columns per warp
constexpr int CL_MAX = 16;
constexpr int CL_MAX_SLAB_BYTES = 200 * 1024;

__global__ void __launch_bounds__(CL_THREADS, 1) qr_panel_cl_kernel(double* A, long long lda, int m, int k0, int kb,
                                                                 double* tau) {
    extern __shared__ double slab[];          // slab[c * R + (i - r0)] = A[i, k0 + c]
    __shared__ double part[2][CL_MAX][MP_PART];  // from CTA q: 0 max, 1 exponent, 2 sum of squares, 2 + t dot
    __shared__ double rrec[2][64];            // row k of columns k .. k0 + kb - 1
    __shared__ double fin[64];
    __shared__ double fin_v0inv, fin_v0s, fin_beta, fin_tau;
    __shared__ int fin_mode;
    cg::cluster_group cluster = cg::this_cluster();
    const int P = (int)cluster.num_blocks(), cta = (int)cluster.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = (m - k0 + P - 1) / P;
    const int r0 = k0 + cta * R, r1 = min(m, r0 + R);
    const int rows = max(0, r1 - r0);
    for (int e = tid; e < rows * kb; e += CL_THREADS) {
        const int c = e / rows, i = e - c * rows;
        slab[c * R + i] = A[(long long)(k0 + c) * lda + r0 + i];
    }
    __syncthreads();
    for (int kk = 0; kk < kb; ++kk) {
        const int k = k0 + kk;
        const int later = kb - kk - 1;
        const int owner = kk / R;  // the CTA holding row k
        double* ck = slab + kk * R;
        // this CTA's partials in CTA `lane`'s shared memory (lanes >= P unused)
        double* pk = cluster.map_shared_rank(&part[kk & 1][cta][0], lane < P ? lane : 0);
        const int lo = max(r0, k), lo1 = max(r0, k + 1);
        // Phase A (own rows): every warp the max of column k over rows >= k
        // and its exponent e (the same in every warp); warp w the dots of
        // x 2^-e with columns t = 1 + w + 16j; the last warp also the (e, s)
        // sum of squares.  Scaling x by 2^-e keeps the dots finite and exact
        // to rounding for any input range, as the reference's dots with the
        // normalised reflector are.
        {
            double mx = 0.0;
            for (int i = lo + lane; i < r1; i += 32) mx = fmax(mx, fabs(ck[i - r0]));
            mx = warp_max(mx);
            const int e = sp_exp(mx);
            const double sc = sp_pow2(-e);
            double d[CL_TASKS];
#pragma unroll
            for (int j = 0; j < CL_TASKS; ++j) d[j] = 0.0;
            for (int i = lo1 + lane; i < r1; i += 32) {
                const double x = ck[i - r0] * sc;
#pragma unroll
                for (int j = 0; j < CL_TASKS; ++j) {
                    const int t = 1 + warp + j * CL_WARPS;
                    if (t <= later) d[j] = fma(x, ck[t * R + (i - r0)], d[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < CL_TASKS; ++j) {
                const int t = 1 + warp + j * CL_WARPS;
                if (t <= later) {  // warp-uniform
                    const double v = warp_sum(d[j]);  // every lane holds the sum
                    if (lane < P) pk[2 + t] = v;
                }
            }
            if (warp == CL_WARPS - 1) {
                double sq = 0.0;
                for (int i = lo1 + lane; i < r1; i += 32) {
                    const double y = ck[i - r0] * sc;
                    sq = fma(y, y, sq);
                }
                sq = warp_sum(sq);
                if (lane < P) {
                    pk[0] = mx;
                    pk[1] = mx > 0.0 ? (double)e : SP_EMPTY_EXP;
                    pk[2] = sq;
                }
            }
            if (cta == owner)
                for (int e = tid; e < (later + 1) * P; e += CL_THREADS) {
                    const int t = e / P, r = e - t * P;
                    *cluster.map_shared_rank(&rrec[kk & 1][t], r) = ck[t * R + (k - r0)];
                }
        }
        cluster.sync();
        // Phase B: every CTA merges the partials of CTAs 0 .. P-1 in the same order
        const double* orow = rrec[kk & 1];
        double dsum[CL_TASKS], rkv[CL_TASKS];
        const double* rp = part[kk & 1][lane < P ? lane : 0];
        const double eq = lane < P ? rp[1] : SP_EMPTY_EXP;
#pragma unroll
        for (int j = 0; j < CL_TASKS; ++j) {
            const int t = 1 + warp + j * CL_WARPS;
            rkv[j] = t <= later ? orow[t] : 0.0;
            dsum[j] = t <= later && lane < P ? rp[2 + t] : 0.0;
        }
        {
            // CTA q's dots are in units of 2^e_q: bring them to 2^E, E = max e_q
            const double emax = warp_max(eq);
#pragma unroll
            for (int j = 0; j < CL_TASKS; ++j) dsum[j] = sp_scale(dsum[j], (int)(eq - emax));
        }
        if (warp == 0) {
            const double x0raw = orow[0];
            double mx = 0.0, e = SP_EMPTY_EXP, sq = 0.0;
            if (lane < P) {
                mx = rp[0];
                e = rp[1];
                sq = rp[2];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {  // symmetric merge: every lane gets the same bits
                mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const double e2 = __shfl_xor_sync(0xffffffffu, e, o);
                const double s2 = __shfl_xor_sync(0xffffffffu, sq, o);
                sp_merge(e, sq, e2, s2);
            }
            if (lane == 0) {
                int mode = 0;
                if (m - k > 1 && mx >= DBL_MIN) {
                    const double inv = 1.0 / mx;  // as the reference: x * (1/max)
                    const double x0 = x0raw * inv;
                    const double xnorm = sq > 0.0 ? sqrt(sq) * (inv * sp_pow2((int)e)) : 0.0;
                    if (xnorm == 0.0) {
                        if (x0 < 0.0) mode = 2;
                    } else {
                        const double nb = -copysign(hypot(x0, xnorm), x0);
                        mode = 1;
                        fin_beta = nb * mx;
                        fin_v0inv = 1.0 / ((x0 - nb) * mx);
                        fin_v0s = (inv * sp_pow2((int)e)) / (x0 - nb);  // 2^E / ((x0 - beta) max), O(1)
                        fin_tau = (nb - x0) / nb;
                    }
                }
                fin_mode = mode;
                if (cta == 0) tau[k] = mode == 1 ? fin_tau : (mode == 2 ? 2.0 : 0.0);
            }
        }
        __syncthreads();
        const int mode = fin_mode;
        if (mode == 1) {
            const double v0s = fin_v0s, tk = fin_tau;
#pragma unroll
            for (int j = 0; j < CL_TASKS; ++j) {
                const int t = 1 + warp + j * CL_WARPS;
                if (t <= later) {  // warp-uniform
                    const double d = warp_sum(dsum[j]);
                    if (lane == 0) fin[t] = (rkv[j] + d * v0s) * tk;
                }
            }
        } else if (mode == 2) {
#pragma unroll
            for (int j = 0; j < CL_TASKS; ++j) {
                const int t = 1 + warp + j * CL_WARPS;
                if (t <= later && lane == 0) fin[t] = rkv[j] * 2.0;  // the tail is zero
            }
        }
        __syncthreads();
        if (mode != 0) {
            // Phase C: reflector tail on own rows, then the later columns
            if (mode == 1) {
                const double v0inv = fin_v0inv;
                for (int i = lo1 + tid; i < r1; i += CL_THREADS) ck[i - r0] *= v0inv;
            }
            if (k >= r0 && k < r1 && tid == 0) ck[k - r0] = mode == 1 ? fin_beta : -ck[k - r0];
            __syncthreads();
            for (int t = 1 + warp; t <= later; t += CL_WARPS) {
                double* cj = ck + t * R;
                const double f = fin[t];
                for (int i = lo1 + lane; i < r1; i += 32) cj[i - r0] -= f * ck[i - r0];
                if (lane == 0 && k >= r0 && k < r1) cj[k - r0] -= f;
            }
        }
        __syncthreads();
    }
    cluster.sync();  // no CTA leaves while another may still read its shared memory
    for (int e = tid; e < rows * kb; e += CL_THREADS) {
        const int c = e / rows, i = e - c * rows;
        A[(long long)(k0 + c) * lda + r0 + i] = slab[c * R + i];
    }
}

// The panel on one cluster with the rows held in registers: lane l of warp w
// holds rows l, l + 32, ... (NR of them) of columns w, w + 16, w + 32, w + 48
// for the whole panel.  Per column:
//   * the warp that holds the pivot column scales its entries below the pivot
//     by 2^-e (e the exponent of the CTA's maximum) into shared memory; one CTA
//     barrier, the only one of the step;
//   * every warp forms the dots of its columns with it and sends them to all
//     CTAs of the cluster (16 destinations x 4 values, one 16-byte st.async per
//     lane); the last warp also sends the sum of squares and e, and the CTA
//     that holds row k its entries of the row;
//   * the stores signal the destination's mbarrier, which expects a fixed
//     number of bytes per column; every warp waits for it, merges the CTAs'
//     values for its own columns and forms the reflector (the same bits in
//     every warp and CTA), and updates its registers.
// What is received alternates between two buffers by column parity: a CTA sends
// column k + 2 only after it has every CTA's column k + 1, which each sends
// after merging column k.
//
// A column is a chain of latencies: the exchange (about 900 cycles from the
// first send to the last arrival at 16 CTAs), the merge and the reflector
// (FP64 sums over lanes, a square root, a division: 1 100), the update and the
// next pivot column (800), the dots (300); no pass touches shared memory but
// for the pivot column.  The shared-memory cluster kernel walks its slab three
// times per column between five CTA barriers and a cluster barrier, in 53 KB of
// code.  us per column on B200: 2304 rows 5.7 -> 2.3, 1024 rows 5.1 -> 2.0.
constexpr int RG_THREADS = 512, RG_WARPS = RG_THREADS / 32;
constexpr int RG_MAX = 16;              // CTAs of the cluster
constexpr int RG_COLS = 64 / RG_WARPS;  // columns per warp
constexpr int RG_PART = 66;             // doubles from one CTA: 64 dots (4 w + j: column w + 16 j), sum of squares, exponent
constexpr int RG_MAX_NR = 8;
constexpr int kRgEmpty = -4096;   // exponent sent for a zero column
constexpr int kRgDenormal = -1001;  // and for one of denormals alone: below every normal one's (-1000 and up)

__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// 16 bytes to a CTA of the cluster, counted by the mbarrier `bar` there
__device__ __forceinline__ void send2(uint32_t dst, double x, double y, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(x), "d"(y), "r"(bar)
                 : "memory");
}
// Bounded wait for what the CTAs of the cluster send (false: the wait limit has passed or an error is recorded)
__device__ __forceinline__ bool wait_sent(uint64_t* bar, uint32_t parity, int* status) {
    const uint32_t b = smem_u32(bar);
    uint64_t t0 = 0;
    unsigned it = 0;
#pragma unroll 1
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(b), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((++it & 255u) == 0u && (t0 = slot_check(t0, status)) == 0) return false;
    }
}

struct RgReflector {
    double tau, beta, v0s;  // v0s = 2^E / (x0 - beta)
    int mode;               // 0: no reflector, 1: reflector, 2: sign flip (tau = 2), 3: of an infinite norm (NaN)
};
// computeHouseholder's recipe from x0, the tail's sum of squares S 4^E (positive
// and finite) and E, by a whole warp: the half-warps take one of the two quotients each
__device__ __forceinline__ RgReflector rg_reflector(double x0, double S, int E) {
    const double xn = x0 * sp_pow2(-E);
    const double nb = -copysign(sqrt(fma(xn, xn, S)), xn);
    const bool lower = (threadIdx.x & 16) == 0;
    const double q = (lower ? nb - xn : 1.0) / (lower ? nb : xn - nb);
    return {__shfl_sync(0xffffffffu, q, 0), nb * sp_pow2(E), __shfl_sync(0xffffffffu, q, 16), 1};
}
// how many of the 32 column pairs (columns w + 32 i, w + 32 i + 16) still hold a column >= kk
__device__ __forceinline__ int rg_live_pairs(int kk) { return 32 - min(16, max(0, kk - 16)) - min(16, max(0, kk - 48)); }

template <int NR>
__global__ void __launch_bounds__(RG_THREADS, 1) qr_panel_rg_kernel(double* A, long long lda, int m, int k0, int kb,
                                                                    double* tau, int* status, int withhold) {
    __shared__ __align__(16) double part[2][RG_MAX][RG_PART];
    __shared__ __align__(16) double rrec[2][64];  // row k, by the dots' index
    __shared__ double s_x[2][NR * 32];            // the pivot column below the pivot, times 2^-e, by column parity
    __shared__ int s_e[2];                        // its e
    __shared__ __align__(16) double s_row[64];
    __shared__ __align__(8) uint64_t bar[2];
    cg::cluster_group cluster = cg::this_cluster();
    const int P = (int)cluster.num_blocks(), cta = (int)cluster.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = (m - k0 + P - 1) / P;
    const int r0 = k0 + cta * R, rows = max(0, min(m - r0, R));
    // what column kk's mbarrier phase expects: the live pairs' dots and one pair of scalars from
    // every CTA, and the row's live pairs
    auto bytes = [&](int kk) { return (uint32_t)((P + 1) * rg_live_pairs(kk) + P) * 16u; };
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
        mbar_arrive_expect_tx(&bar[0], bytes(0));
        mbar_arrive_expect_tx(&bar[1], bytes(1));
    }
    grid_dep_wait();
    grid_dep_launch();
    double a[RG_COLS][NR], x[NR];
#pragma unroll
    for (int j = 0; j < RG_COLS; ++j)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int c = warp + RG_WARPS * j, i = lane + 32 * r;
            a[j][r] = c < kb && i < rows ? A[(long long)(k0 + c) * lda + r0 + i] : 0.0;
        }
    cluster.sync();  // every CTA's mbarriers are ready
    bool fail = false;
    // sends: lane 2 d + h the warp's column pair h to CTA d
    const int dest = lane >> 1, half = lane & 1;
    const uint32_t to_part = cluster_addr(&part[0][cta][warp * 4 + 2 * half], dest < P ? dest : 0);
    const uint32_t to_rrec = cluster_addr(&rrec[0][warp * 4 + 2 * half], dest < P ? dest : 0);
    const uint32_t to_bar = cluster_addr(&bar[0], dest < P ? dest : 0);
    // A column of this warp (y), below its pivot row k and scaled by 2^-e, into the buffer of its
    // parity.  Two buffers, because nothing else keeps a warp from writing column k + 1 while another
    // still reads column k: a warp past its last column sends nothing, so no one waits for it until
    // the next step's CTA barrier, after which column k's buffer is written again.
    auto put_pivot = [&](double (&y)[NR], int k, int par) {
        unsigned hi = 0;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            if (r0 + lane + 32 * r < k) y[r] = 0.0;
            hi = max(hi, (unsigned)__double2hiint(y[r]) & 0x7fffffffu);
        }
        hi = __reduce_max_sync(0xffffffffu, hi) >> 20;  // the maximum's biased exponent
        int e = hi == 0x7ff ? 0 : min(1000, max(-1000, (int)hi - 1023));
        if (hi == 0) {
            bool any = false;
#pragma unroll
            for (int r = 0; r < NR; ++r) any |= y[r] != 0.0;
            e = __any_sync(0xffffffffu, any) ? kRgDenormal : kRgEmpty;
        }
        const double sc = sp_pow2(-max(e, kRgDenormal));
#pragma unroll
        for (int r = 0; r < NR; ++r) s_x[par][lane + 32 * r] = r0 + lane + 32 * r > k ? y[r] * sc : 0.0;
        if (lane == 0) s_e[par] = e;
    };
    if (warp == 0) {
        double y[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) y[r] = a[0][r];
        put_pivot(y, k0, 0);
    }
#pragma unroll 1
    for (int kk = 0; kk < kb; ++kk) {
        const int k = k0 + kk, par = kk & 1;
        const bool live = dest < P && warp + RG_WARPS * (2 * half + 1) >= kk;
        // ---- row k's entries of this warp's columns, from the lane that holds them
        if (k >= r0 && k < r0 + rows) {
#pragma unroll
            for (int r = 0; r < NR; ++r)
                if (r0 + lane + 32 * r == k) {
#pragma unroll
                    for (int j = 0; j < RG_COLS; ++j) s_row[warp * 4 + j] = a[j][r];
                }
            __syncwarp();
            const double2 v = *reinterpret_cast<const double2*>(&s_row[warp * 4 + 2 * half]);
            if (live) send2(to_rrec + par * 512u, v.x, v.y, to_bar + par * 8u);
        }
        if (__syncthreads_or(fail)) break;  // the pivot column is in shared memory
        // ---- this CTA's dots with it
        const int e_own = s_e[par];
        double d[RG_COLS];
#pragma unroll
        for (int j = 0; j < RG_COLS; ++j) d[j] = 0.0;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            x[r] = s_x[par][lane + 32 * r];
#pragma unroll
            for (int j = 0; j < RG_COLS; ++j) d[j] = fma(x[r], a[j][r], d[j]);
        }
        {
            // the four sums over the lanes: lanes with bit 0 = half keep columns 2 half, 2 half + 1
            double k0v = half ? d[2] : d[0], k1v = half ? d[3] : d[1];
            k0v += shfl_xor(half ? d[0] : d[2], 1);
            k1v += shfl_xor(half ? d[1] : d[3], 1);
            const bool second = lane & 2;
            double v = (second ? k1v : k0v) + shfl_xor(second ? k0v : k1v, 2);
            v += shfl_xor(v, 4);
            v += shfl_xor(v, 8);
            v += shfl_xor(v, 16);
            const double o = shfl_xor(v, 2);
            if (live)
                send2(to_part + par * (uint32_t)sizeof(part[0]), second ? o : v, second ? v : o, to_bar + par * 8u);
        }
        if (warp == RG_WARPS - 1) {
            double q = 0.0;
#pragma unroll
            for (int r = 0; r < NR; ++r) q = fma(x[r], x[r], q);
            q = warp_sum(q);
            // (withhold, a test hook: CTA 0 leaves the first column's scalars out, so the waits run out)
            if (lane < P && !(withhold && cta == 0 && kk == 0))
                send2(cluster_addr(&part[par][cta][64], lane), q, (double)e_own, cluster_addr(&bar[par], lane));
        }
        // ---- merge: lane q (and q + 16) takes CTA q's dots of columns 0, 1 (2, 3) of this warp
        if (__any_sync(0xffffffffu, !wait_sent(&bar[par], (kk >> 1) & 1, status))) {
            // Given up: the CTA leaves at the next barrier.  Nothing else of the step, least of all the arming
            // below: this phase is still open, and a second arrival in it takes its count below zero, which
            // ends the kernel with an error.
            fail = true;
            continue;
        }
        const int q = lane & 15, h = lane >> 4;
        const double* pq = part[par][q < P ? q : 0];
        const double2 se = *reinterpret_cast<const double2*>(pq + 64);
        const double2 dd = *reinterpret_cast<const double2*>(pq + warp * 4 + 2 * h);
        const double2 rr = *reinterpret_cast<const double2*>(&rrec[par][warp * 4 + 2 * h]);
        const double x0 = rrec[par][(kk & (RG_WARPS - 1)) * 4 + kk / RG_WARPS];
        const int eq = q < P ? (int)se.y : kRgEmpty;
        const int E = __reduce_max_sync(0xffffffffu, eq);
        const double f = eq - E >= -1022 && q < P ? sp_pow2(eq - E) : 0.0;
        double S = (se.x * f) * f;
        const bool second = lane & 8;
        double dot = (second ? dd.y : dd.x) * f + shfl_xor((second ? dd.x : dd.y) * f, 8);
        S += shfl_xor(S, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            S += shfl_xor(S, o);
            dot += shfl_xor(dot, o);
        }
        // ---- the reflector.  A zero tail leaves a sign flip or none, a NaN in it likewise; x is then
        // made finite, as the update multiplies it by 0 where it must change nothing
        RgReflector hh{0.0, x0, 0.0, 0};
        if (m - k > 1 && E > kRgDenormal) {  // (a maximum below the normal range: no reflector)
            if (S > 0.0 && S <= DBL_MAX) {
                hh = rg_reflector(x0, S, E);
            } else {
                if (S > 0.0) hh = {CUDART_NAN, CUDART_NAN, 0.0, 3};
                else if (x0 < 0.0) hh = {2.0, -x0, 0.0, 2};
                dot = 0.0;
#pragma unroll
                for (int r = 0; r < NR; ++r) x[r] = 0.0;
            }
        }
        if (cta == 0 && tid == 0) tau[k] = hh.tau;
        // armed for column kk + 2
        if (tid == 0) mbar_arrive_expect_tx(&bar[par], bytes(kk + 2));
        // ---- update: f_t = tau (a_kt + dot v0s), columns right of the pivot (f = 0 elsewhere), rows from k
        // on (v = 0 above, but a NaN f would take those with it; with both guards the factorisation of
        // 2304 x 2048 takes 5.93 ms, 5.85 without)
        const double ft = hh.tau * fma(dot, hh.v0s, second ? rr.y : rr.x);
        const double sv = hh.mode == 1 && e_own - E >= -1022 ? sp_pow2(e_own - E) * hh.v0s : 0.0;
        double fj[RG_COLS];
#pragma unroll
        for (int j = 0; j < RG_COLS; ++j) {
            const double v = __shfl_sync(0xffffffffu, ft, (j >> 1) * 16 + (j & 1) * 8);
            fj[j] = warp + RG_WARPS * j > kk && hh.mode != 0 ? v : 0.0;
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) x[r] = r0 + lane + 32 * r == k ? 1.0 : x[r] * sv;  // v (0 above row k)
        if (kk + 1 < kb && warp == ((kk + 1) & (RG_WARPS - 1))) {
            // the next pivot column ahead of the rest: the other warps wait for it
            const int jn = (kk + 1) / RG_WARPS;
            const double f = jn == 0 ? fj[0] : jn == 1 ? fj[1] : jn == 2 ? fj[2] : fj[3];
            double y[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r)
                y[r] = fma(-f, x[r], jn == 0 ? a[0][r] : jn == 1 ? a[1][r] : jn == 2 ? a[2][r] : a[3][r]);
            put_pivot(y, k + 1, par ^ 1);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r)
            if (r0 + lane + 32 * r >= k) {
#pragma unroll
                for (int j = 0; j < RG_COLS; ++j) a[j][r] = fma(-fj[j], x[r], a[j][r]);
            }
#pragma unroll
        for (int j = 0; j < RG_COLS; ++j) {
            if (warp + RG_WARPS * j == kk) {  // the pivot column itself: its tail, and beta on row k
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int g = r0 + lane + 32 * r;
                    if (g == k) a[j][r] = hh.beta;
                    else if (g > k && (hh.mode & 1)) a[j][r] = hh.mode == 1 ? x[r] : hh.beta;
                }
            }
        }
    }
    // No CTA leaves while another may still send to it.  What a CTA waited for has arrived; one that gave
    // up lets its own sends land first (they take a microsecond).
    if (__syncthreads_or(fail)) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 100000) {
        }
    }
    cluster.sync();
#pragma unroll
    for (int j = 0; j < RG_COLS; ++j)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const int c = warp + RG_WARPS * j, i = lane + 32 * r;
            if (c < kb && i < rows) A[(long long)(k0 + c) * lda + r0 + i] = a[j][r];
        }
}

// V (ldv x 64, column-major): column i < kb holds reflector k0+i (zeros above
// row k0+i+shift, one on it, A's tail below); columns kb .. 63 are zero.  A step
// without a reflector (tau = 0) may have left anything below the diagonal, a NaN
// for instance, which V^T V would spread over T: its tail is zero in V.
__global__ void qr_pack_v_kernel(const double* A, long long lda, int m, int k0, int kb, int shift, const double* tau,
                                 double* V, long long ldv) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ldv * 64) return;
    const int i = (int)(e / ldv);
    const int row = (int)(e % ldv);
    double v = 0.0;
    if (i < kb && row < m) {
        const int k = k0 + i + shift;
        v = row < k ? 0.0 : (row == k ? 1.0 : tau[i] != 0.0 ? A[(long long)(k0 + i) * lda + row] : 0.0);
    }
    V[e] = v;
}

// G = V^T V (64 x 64, row-major) over rows [r0, r1) of the packed V
// (column-major, ld ldv), in two launches: every CTA sums its slab of rows,
// 32 rows at a time staged in shared memory, into a 64 x 64 partial (each
// thread a 4 x 4 block of it, the rows in order); a second launch adds the
// partials in slab order.  The result does not depend on timing.
constexpr int GR_THREADS = 256, GR_CHUNK = 32;

__global__ void __launch_bounds__(GR_THREADS) qr_gram_partial_kernel(const double* V, long long ldv, int r0, int r1,
                                                                     int slab, double* part) {
    __shared__ double sv[GR_CHUNK][64 + 1];
    const int tid = threadIdx.x;
    const int bi = (tid >> 4) * 4, bj = (tid & 15) * 4;  // this thread's 4 x 4 block of G
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    const int s0 = r0 + blockIdx.x * slab;
    const int s1 = s0 + slab < r1 ? s0 + slab : r1;
    for (int c0 = s0; c0 < s1; c0 += GR_CHUNK) {
        const int n = s1 - c0 < GR_CHUNK ? s1 - c0 : GR_CHUNK;
        __syncthreads();  // the previous chunk has been read
        for (int e = tid; e < GR_CHUNK * 64; e += GR_THREADS) {
            const int r = e % GR_CHUNK, c = e / GR_CHUNK;  // consecutive threads, consecutive rows
            sv[r][c] = r < n ? V[(long long)c * ldv + c0 + r] : 0.0;
        }
        __syncthreads();
        for (int r = 0; r < n; ++r) {
            double x[4], y[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                x[a] = sv[r][bi + a];
                y[a] = sv[r][bj + a];
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma(x[a], y[b], acc[a][b]);
        }
    }
    double* out = part + (size_t)blockIdx.x * 64 * 64;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) out[(bi + a) * 64 + bj + b] = acc[a][b];
}

__global__ void qr_gram_sum_kernel(const double* part, int parts, double* G) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 64 * 64) return;
    double s = part[e];
    for (int q = 1; q < parts; ++q) s += part[(size_t)q * 64 * 64 + e];
    G[e] = s;
}

// T (64 x 64, row-major, upper triangular) of H_0 H_1 ... H_63 = I - V T V^T from
// G = V^T V and tau, in one CTA of 256 threads.  The reference builds it column
// by column (buildT); that recurrence solves T (D^-1 + U) = I with D = diag(tau)
// and U the part of G above its diagonal, so T = (I + D U)^-1 D, which also
// holds where tau is 0.  The unit triangular inverse comes from the four 16 x 16
// diagonal blocks at once, a thread per column with the column in registers (no
// barrier in the substitution), and two joins X_ab = -X_aa (N_ab X_bb), 16 and
// then 32 wide.  On entry t holds G above its diagonal; x is scratch.
constexpr int BT_THREADS = 256, BT_LD = 65;

__device__ void build_t(double (*t)[BT_LD], double (*x)[33], const double* tau, int kb, double* T) {
    const int tid = threadIdx.x;
    __shared__ double s_tau[64];
    if (tid < 64) s_tau[tid] = tid < kb ? tau[tid] : 0.0;
    __syncthreads();
    for (int e = tid; e < 64 * 64; e += BT_THREADS) {
        const int r = e >> 6, c = e & 63;
        t[r][c] = r < c ? s_tau[r] * t[r][c] : (r == c ? 1.0 : 0.0);
    }
    __syncthreads();
    double y[16];
    const int o = (tid >> 4) * 16, j = tid & 15;
    if (tid < 64) {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = i == j ? 1.0 : 0.0;
#pragma unroll
        for (int c = 15; c > 0; --c)
#pragma unroll
            for (int i = 0; i < c; ++i) y[i] = fma(-t[o + i][o + c], y[c], y[i]);
    }
    __syncthreads();
    if (tid < 64) {
#pragma unroll
        for (int i = 0; i < 16; ++i) t[o + i][o + j] = y[i];
    }
    __syncthreads();
    {
        // blocks (0, 1) and (2, 3): two entries per thread of each 16 x 16 product
        const int p = tid >> 7, a0 = 32 * p, b0 = a0 + 16, r = (tid >> 3) & 15, c = tid & 7;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            s0 = fma(t[a0 + r][b0 + q], t[b0 + q][b0 + c], s0);
            s1 = fma(t[a0 + r][b0 + q], t[b0 + q][b0 + c + 8], s1);
        }
        x[16 * p + r][c] = s0;
        x[16 * p + r][c + 8] = s1;
        __syncthreads();
        s0 = s1 = 0.0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            s0 = fma(t[a0 + r][a0 + q], x[16 * p + q][c], s0);
            s1 = fma(t[a0 + r][a0 + q], x[16 * p + q][c + 8], s1);
        }
        t[a0 + r][b0 + c] = -s0;
        t[a0 + r][b0 + c + 8] = -s1;
        __syncthreads();
    }
    {
        const int r = tid >> 3, c = tid & 7;
        double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
        for (int q = 0; q < 32; ++q) {
            const double v = t[r][32 + q];
#pragma unroll
            for (int i = 0; i < 4; ++i) s4[i] = fma(v, t[32 + q][32 + c + 8 * i], s4[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[r][c + 8 * i] = s4[i];
            s4[i] = 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int q = 0; q < 32; ++q) {
            const double v = t[r][q];
#pragma unroll
            for (int i = 0; i < 4; ++i) s4[i] = fma(v, x[q][c + 8 * i], s4[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) t[r][32 + c + 8 * i] = -s4[i];
        __syncthreads();
    }
    for (int e = tid; e < 64 * 64; e += BT_THREADS) T[e] = t[e >> 6][e & 63] * s_tau[e & 63];
}

__global__ void __launch_bounds__(BT_THREADS) qr_build_t_kernel(const double* G, const double* tau, int kb,
                                                                double* T) {
    extern __shared__ double dyn[];
    double(*t)[BT_LD] = reinterpret_cast<double(*)[BT_LD]>(dyn);
    double(*x)[33] = reinterpret_cast<double(*)[33]>(dyn + 64 * BT_LD);
    for (int e = threadIdx.x; e < 64 * 64; e += BT_THREADS) t[e >> 6][e & 63] = G[e];
    __syncthreads();
    build_t(t, x, tau, kb, T);
}
constexpr int BT_SMEM = (64 * BT_LD + 32 * 33) * 8;

// V and T of one panel per cluster, panels p0, p0 + 1, ... in one launch: the
// cluster's CTAs pack their rows of V, 32 at a time, and sum V^T V over them on
// the DMMA path (the 20 of its 16 x 8 blocks that reach above the diagonal);
// each CTA then adds its share of the CTAs' partial sums in rank order, through
// distributed shared memory, and rank 0 forms T.  Latency-bound: 14 us for one
// panel of 2304 rows (four launches before, 30 us: packing 2, partial sums 7,
// their total 4, T 17.5), 24 us for the 16 panels of n = 1024 together (480 us
// one by one).
constexpr int VT_THREADS = 256, VT_CHUNK = 32, VT_LD = 68;  // VT_LD: fragment loads hit distinct banks
constexpr int VT_SMEM = (64 * 64 + 64 * BT_LD + VT_CHUNK * VT_LD) * 8;
constexpr int VT_MAX_ROWS = 4096;

__global__ void __launch_bounds__(VT_THREADS) qr_vt_kernel(const double* A, long long lda, int m, int kmax, int p0,
                                                           int shift, const double* tau, double* V, long long ldv,
                                                           double* T) {
    extern __shared__ double dyn[];
    grid_dep_wait();
    grid_dep_launch();
    double* part = dyn;                                                           // 64 x 64
    double(*t)[BT_LD] = reinterpret_cast<double(*)[BT_LD]>(dyn + 64 * 64);
    double(*sv)[VT_LD] = reinterpret_cast<double(*)[VT_LD]>(dyn + 64 * 64 + 64 * BT_LD);  // [row][column]
    cg::cluster_group cluster = cg::this_cluster();
    const int P = (int)cluster.num_blocks(), cta = (int)cluster.block_rank();
    const int pi = blockIdx.x / P, k0 = (p0 + pi) * 64, kb = min(64, kmax - k0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const int R = ((m - k0 + P - 1) / P + VT_CHUNK - 1) / VT_CHUNK * VT_CHUNK;
    const int r0 = k0 + cta * R, r1 = min(m, r0 + R);
    double* Vp = V + (size_t)pi * ldv * 64;
    constexpr int CW = 64 / (VT_THREADS / 32);  // columns per warp
    // this warp's columns with a reflector (the tails of the others are zero, as in qr_pack_v_kernel)
    const int cl = warp * CW + (lane & (CW - 1));
    const unsigned has = __ballot_sync(0xffffffffu, cl < kb && tau[min(k0 + cl, kmax - 1)] != 0.0);
    double v[CW];
    auto fetch = [&](int c0) {
        const int row = c0 + lane;
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            const int c = warp * CW + i, k = k0 + c + shift;
            v[i] = c < kb && row > k && row < r1 ? A[(long long)(k0 + c) * lda + row] : (c < kb && row == k ? 1.0 : 0.0);
        }
    };
    // this warp's 16 x 8 blocks: 0 .. 19 in rows of 8, 6, 4, 2
    int bi[3], bj[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int b = warp + 8 * q;
        bi[q] = b < 8 ? 0 : b < 14 ? 1 : b < 18 ? 2 : 3;
        bj[q] = b < 8 ? b : b < 14 ? b - 6 : b < 18 ? b - 10 : b - 12;
    }
    double acc[3][4] = {};
    if (r0 < r1) fetch(r0);
    for (int c0 = r0; c0 < r1; c0 += VT_CHUNK) {
#pragma unroll
        for (int i = 0; i < CW; ++i) {
            const double x = (has >> i & 1) || c0 + lane == k0 + warp * CW + i + shift ? v[i] : 0.0;
            sv[lane][warp * CW + i] = x;
            if (c0 + lane < r1) Vp[(size_t)(warp * CW + i) * ldv + c0 + lane] = x;
        }
        __syncthreads();
        if (c0 + VT_CHUNK < r1) fetch(c0 + VT_CHUNK);
#pragma unroll
        for (int ks = 0; ks < VT_CHUNK; ks += 8)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if (q == 2 && warp >= 4) continue;
                double fa[4], fb[2];
#pragma unroll
                for (int i = 0; i < 4; ++i) fa[i] = sv[ks + tq + 4 * (i >> 1)][16 * bi[q] + g + 8 * (i & 1)];
#pragma unroll
                for (int i = 0; i < 2; ++i) fb[i] = sv[ks + tq + 4 * i][8 * bj[q] + g];
                dmma::mma_f64<8>(acc[q], fa, fb);
            }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        if (q == 2 && warp >= 4) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) part[(16 * bi[q] + g + 8 * (i >> 1)) * 64 + 8 * bj[q] + 2 * tq + (i & 1)] = acc[q][i];
    }
    cluster.sync();
    // entries above the diagonal only: the blocks below it were not formed
    for (int e = cta * VT_THREADS + tid; e < 64 * 64; e += P * VT_THREADS) {
        if ((e >> 6) >= (e & 63)) continue;
        double s[RG_MAX];
#pragma unroll
        for (int q = 0; q < RG_MAX; ++q) s[q] = q < P ? *cluster.map_shared_rank(&part[e], q) : 0.0;
        double sum = s[0];
#pragma unroll
        for (int q = 1; q < RG_MAX; ++q) sum += s[q];
        *cluster.map_shared_rank(&t[e >> 6][e & 63], 0) = sum;
    }
    cluster.sync();
    if (cta == 0) build_t(t, reinterpret_cast<double(*)[33]>(&sv[0][0]), tau + k0, kb, T + (size_t)pi * 64 * 64);
}

// VT = V op(T) (op: T, or T^T), panels p0, p0 + 1, ...: 64 rows of one panel per CTA
constexpr int VP_SMEM = 2 * 64 * VT_LD * 8;
__global__ void __launch_bounds__(VT_THREADS) qr_vt_product_kernel(const double* V, long long ldv, int m, int p0,
                                                                   const double* T, int trans, double* VT) {
    extern __shared__ double dyn[];
    grid_dep_wait();
    grid_dep_launch();
    double(*sv)[VT_LD] = reinterpret_cast<double(*)[VT_LD]>(dyn);                // [column][row]
    double(*st)[VT_LD] = reinterpret_cast<double(*)[VT_LD]>(dyn + 64 * VT_LD);   // T: [row][column]
    const int pi = blockIdx.y, k0 = (p0 + pi) * 64, r0 = k0 + 64 * blockIdx.x;
    if (r0 >= m) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const double* Vp = V + (size_t)pi * ldv * 64;
    const double* Tp = T + (size_t)pi * 64 * 64;
    for (int e = tid; e < 64 * 64; e += VT_THREADS) {
        const int r = e & 63, c = e >> 6;
        sv[c][r] = r0 + r < m ? Vp[(size_t)c * ldv + r0 + r] : 0.0;
        st[e >> 6][e & 63] = Tp[e];
    }
    __syncthreads();
    const int wr = (warp >> 2) * 32, wc = (warp & 3) * 16;
    double acc[2][2][4] = {};
#pragma unroll
    for (int ks = 0; ks < 64; ks += 8) {
        double fa[2][4], fb[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int i = 0; i < 4; ++i) fa[a][i] = sv[ks + tq + 4 * (i >> 1)][wr + 16 * a + g + 8 * (i & 1)];
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                fb[b][i] = trans ? st[wc + 8 * b + g][ks + tq + 4 * i] : st[ks + tq + 4 * i][wc + 8 * b + g];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) dmma::mma_f64<8>(acc[a][b], fa[a], fb[b]);
    }
    double* out = VT + (size_t)pi * ldv * 64;
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = r0 + wr + 16 * a + g + 8 * (i >> 1), col = wc + 8 * b + 2 * tq + (i & 1);
                if (row < m) out[(size_t)col * ldv + row] = acc[a][b][i];
            }
}

// ones on the diagonal of a column-major matrix
__global__ void set_diag_kernel(double* q, long long ldq, long long d) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < d) q[i * ldq + i] = 1.0;
}

}  // namespace qr

// Multi-CTA panel: P CTAs in one cooperative launch (all resident at once);
// scratch holds 2 x P x MP_PART partials, 2 x 64 row entries and the barrier
// counter (zeroed here before the launch).
size_t qr_panel_mp_scratch_bytes(int P) {
    return ((size_t)2 * P * qr::MP_PART + 128) * sizeof(double) + 256;
}

// Largest cluster of the cluster panel kernel that can be resident with a
// full slab on this device (16, else 8), or 1 when none can.
int qr_panel_cluster_max() {
    const void* kern = (const void*)qr::qr_panel_cl_kernel;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, qr::CL_MAX_SLAB_BYTES) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    for (int c = qr::CL_MAX; c >= 8; c /= 2) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(qr::CL_THREADS);
        cfg.dynamicSmemBytes = qr::CL_MAX_SLAB_BYTES;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = c;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) return c;
        cudaGetLastError();
    }
    return 1;
}

namespace qr {
// one CTA per 64 rows, up to the largest cluster (measured against 128 rows per
// CTA: 13.8 vs 14.2 ms at 2048^2, 32.6 vs 33.0 at 4096^2)
static int panel_ctas(int m, int k0, int cluster_max) { return max(1, min((m - k0) / 64, min(cluster_max, CL_MAX))); }
}  // namespace qr

bool qr_panel_waits(int m, int k0, int cluster_max) {
    const int cl = qr::panel_ctas(m, k0, cluster_max);
    return (m - k0 + cl - 1) / cl <= 32 * qr::RG_MAX_NR;
}

// Factors columns k0 .. k0+kb-1 of the column-major m x n matrix A (rows from
// the diagonal down), writing tau[k0 ..]; A's entries below the diagonal of
// those columns become the reflectors' tails (v0 = 1 implied), the diagonal
// the new R entries (computeHouseholder / applyHouseholderToColumn,
// HouseholderQR.java:219-384).  One cluster of CTAs with >= 64 rows each (a
// single CTA below 128 rows) when their rows fit in registers or shared memory,
// else a cooperative grid of P CTAs.
int launch_qr_panel(double* a, long long lda, int m, int k0, int kb, double* tau, int P, int cluster_max,
                    void* scratch, int* status, bool withhold, cudaStream_t st) {
    const int cl = qr::panel_ctas(m, k0, cluster_max), rows = (m - k0 + cl - 1) / cl;
    // rows in registers while every CTA has at most 256 (3.0 us per column at 4000 rows, against 6.8
    // with the slab in shared memory and 9.4 on the grid)
    if (qr_panel_waits(m, k0, cluster_max)) {
        using namespace qr;
        static void (*const kerns[RG_MAX_NR + 1])(double*, long long, int, int, int, double*, int*, int) = {
            nullptr,
            qr_panel_rg_kernel<1>, qr_panel_rg_kernel<2>, qr_panel_rg_kernel<3>, qr_panel_rg_kernel<4>,
            qr_panel_rg_kernel<5>, qr_panel_rg_kernel<6>, qr_panel_rg_kernel<7>, qr_panel_rg_kernel<8>};
        auto kern = kerns[(rows + 31) / 32];
        if (cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return JLC_E_LAUNCH;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        cfg.gridDim = dim3(cl);
        cfg.blockDim = dim3(qr::RG_THREADS);
        cfg.stream = st;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1] = chained_launch();
        cfg.attrs = at;
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, kern, a, lda, m, k0, kb, tau, status, withhold ? 1 : 0) == cudaSuccess
                   ? JLC_OK
                   : JLC_E_LAUNCH;
    }
    if ((size_t)((m - k0 + cl - 1) / cl) * kb * sizeof(double) <= (size_t)qr::CL_MAX_SLAB_BYTES) {
        const void* kern = (const void*)qr::qr_panel_cl_kernel;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, qr::CL_MAX_SLAB_BYTES) !=
                cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return JLC_E_LAUNCH;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        cfg.gridDim = dim3(cl);
        cfg.blockDim = dim3(qr::CL_THREADS);
        cfg.dynamicSmemBytes = (size_t)((m - k0 + cl - 1) / cl) * kb * sizeof(double);
        cfg.stream = st;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, qr::qr_panel_cl_kernel, a, lda, m, k0, kb, tau) == cudaSuccess
                   ? JLC_OK
                   : JLC_E_LAUNCH;
    }
    double* part = static_cast<double*>(scratch);
    double* rowrec = part + (size_t)2 * P * qr::MP_PART;
    unsigned* counter = reinterpret_cast<unsigned*>(rowrec + 128);
    if (cudaMemsetAsync(counter, 0, sizeof(unsigned), st) != cudaSuccess) return JLC_E_LAUNCH;
    void* args[] = {&a, &lda, &m, &k0, &kb, &tau, &part, &rowrec, &counter, &status};
    // each CTA's rows in shared memory when the slab fits, else in place
    const int R = (m - k0 + P - 1) / P;
    const size_t slab = (size_t)R * kb * sizeof(double);
    cudaError_t e;
    if (slab <= (size_t)qr::SP_MAX_SLAB_BYTES && P <= qr::SP_MAX_CTAS) {
        e = cudaFuncSetAttribute((const void*)qr::qr_panel_sm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 qr::SP_MAX_SLAB_BYTES);
        if (e != cudaSuccess) return JLC_E_LAUNCH;
        e = cudaLaunchCooperativeKernel((const void*)qr::qr_panel_sm_kernel, dim3(P), dim3(qr::MP_THREADS), args,
                                        slab, st);
    } else {
        e = cudaLaunchCooperativeKernel((const void*)qr::qr_panel_mp_kernel, dim3(P), dim3(qr::MP_THREADS), args, 0,
                                        st);
    }
    return e == cudaSuccess ? JLC_OK : JLC_E_LAUNCH;
}

int launch_set_identity(double* q, long long ldq, long long m, long long cols, cudaStream_t st) {
    if (cudaMemset2DAsync(q, (size_t)ldq * sizeof(double), 0, (size_t)m * sizeof(double), (size_t)cols, st) !=
        cudaSuccess)
        return JLC_E_LAUNCH;
    const long long d = m < cols ? m : cols;
    qr::set_diag_kernel<<<(unsigned)((d + 255) / 256), 256, 0, st>>>(q, ldq, d);
    return cudaGetLastError() == cudaSuccess ? JLC_OK : JLC_E_LAUNCH;
}

size_t qr_gram_scratch_bytes(int sm_count) {
    return ((size_t)(sm_count > 0 ? sm_count : 1) + 1) * 64 * 64 * sizeof(double);
}

// V, T and V op(T) of the panels p0 .. p0 + panels - 1 (64 columns each) of the
// reflectors stored in a (below the diagonal shifted down by `shift` rows):
// panel p0 + i's at v + i 64 ldv, t + i 64^2 and vt + i 64 ldv.
int launch_qr_vt(const double* a, long long lda, int m, int kmax, int p0, int panels, int shift, const double* tau,
                 double* v, long long ldv, double* t, double* vt, bool trans, double* gram, int cluster_max,
                 int sm_count, cudaStream_t st, int* launches) {
    using namespace qr;
    const int rows = m - 64 * p0;  // of the tallest panel
    *launches = rows <= VT_MAX_ROWS ? 2 : 4 * panels + 1;
    if (rows <= VT_MAX_ROWS) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[2];
        const int cl = max(1, min((rows + 63) / 64, min(cluster_max, RG_MAX)));
        cfg.gridDim = dim3(cl * panels);
        cfg.blockDim = dim3(VT_THREADS);
        cfg.dynamicSmemBytes = VT_SMEM;
        cfg.stream = st;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1] = chained_launch();
        cfg.attrs = at;
        cfg.numAttrs = 2;
        const void* kern = (const void*)qr_vt_kernel;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, VT_SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaLaunchKernelEx(&cfg, qr_vt_kernel, a, lda, m, kmax, p0, shift, tau, v, ldv, t) != cudaSuccess)
            return JLC_E_LAUNCH;
    } else {
        if (cudaFuncSetAttribute((const void*)qr_build_t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 BT_SMEM) != cudaSuccess)
            return JLC_E_LAUNCH;
        for (int i = 0; i < panels; ++i) {
            const int k0 = 64 * (p0 + i), kb = min(64, kmax - k0);
            double* vi = v + (size_t)i * ldv * 64;
            qr_pack_v_kernel<<<(unsigned)((ldv * 64 + 255) / 256), 256, 0, st>>>(a, lda, m, k0, kb, shift, tau + k0, vi,
                                                                                 ldv);
            int parts = (m - k0 + GR_CHUNK - 1) / GR_CHUNK;
            if (parts > sm_count) parts = sm_count;
            const int slab = (m - k0 + parts - 1) / parts;
            parts = (m - k0 + slab - 1) / slab;
            double* g = gram + (size_t)sm_count * 64 * 64;
            qr_gram_partial_kernel<<<parts, GR_THREADS, 0, st>>>(vi, ldv, k0, m, slab, gram);
            qr_gram_sum_kernel<<<(64 * 64 + 255) / 256, 256, 0, st>>>(gram, parts, g);
            qr_build_t_kernel<<<1, BT_THREADS, BT_SMEM, st>>>(g, tau + k0, kb, t + (size_t)i * 64 * 64);
        }
    }
    if (cudaFuncSetAttribute((const void*)qr_vt_product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, VP_SMEM) !=
        cudaSuccess)
        return JLC_E_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = dim3((unsigned)((rows + 63) / 64), (unsigned)panels);
    cfg.blockDim = dim3(VT_THREADS);
    cfg.dynamicSmemBytes = VP_SMEM;
    cfg.stream = st;
    at[0] = chained_launch();
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, qr_vt_product_kernel, (const double*)v, ldv, m, p0, (const double*)t, trans ? 1 : 0,
                              vt) == cudaSuccess
               ? JLC_OK
               : JLC_E_LAUNCH;
}

}  // namespace jlc
