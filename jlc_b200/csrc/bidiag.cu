// Golub-Kahan bidiagonalisation on the device.
//
// The reference's tested class, Bidiagonalization.decomposeUpper
// (decomposition/bidiagonal/Bidiagonalization.java:180-309, m >= n), reduces A
// to upper bidiagonal B = U^T A V one column and one row at a time:
//   * column k: x = B(k:m, k); scale/ssq norm over all of x (x0 included),
//     beta = -copysign(xnorm, x0) (beta = xnorm when x0 < 0), tau = (beta -
//     x0) / beta, v = x / (x0 - beta) with v_0 = 1; no reflector when xnorm or
//     |tau| is at most Double.MIN_NORMAL; H = I - tau v v^T applied to the
//     columns k.. of B from the left (and to U from the right); B(k, k) = beta;
//   * row k (k < n - 1): the same recipe on x = B(k, k+1:n), applied to the
//     rows k.. of B from the right (and to V).
// That is a BLAS-2 algorithm: every reflector touches the whole trailing
// matrix.  Here all n steps run in one cooperative launch.  Row g lives on CTA
// g % P (at most one CTA per SM), so that every CTA keeps rows in play as the
// trailing matrix shrinks, and a CTA's rows -- its slab -- sit in shared
// memory for the whole reduction (row-major, a thread per column) while they
// fit, else in a global work array laid out the same way; where the device has
// no room for that array, they stay in the matrix (IN_PLACE: its columns are lda
// apart, so a thread per column reads 32 bytes for 8: 4096 x 4096 747 ms, 168
// with the array).
//
// A step needs two sums over all CTAs and no more, because everything else is
// formed redundantly from their results:
//   * the dots of column k with every trailing column, and its norm.  As the
//     raw column is all they need, the pass that finishes step k - 1 takes
//     them: w_j = tau (a_kj + sum_{i>k} x_i a_ij / (x0 - beta)) =
//     tau v^T A(:, j) follows from the sums.  A warp of some CTA sums 2
//     columns and publishes w_j;
//   * row k after the column reflector is a_kj - w_j: every CTA has both, forms
//     the row reflector u from them, then x = tau_p (A - v w^T) u on its own
//     rows (row-local), A - v w^T - x u^T, and the dots of column k + 1.
// The values cross the CTAs in tagged 16-byte slots (jlc_slab.cuh): a reader
// waits for the datum itself, and there is no barrier.
//
// What bounds a step is latency: two exchanges through L2 (about 1500 cycles
// each from store to load), two norms (a cross-warp sum, a square root, a
// division) and two short passes.  Hence
//   * A r (r the row before its reflector is known) and the norm of r are summed
//     in one pass between the same barriers: x = tau_p (t + (A r - v (w . r)) /
//     (x0 - beta)), t the pivot column, by the warps that have rows to finish
//     (before: norm, barrier, reflector, pass, barrier);
//   * few polls: what every CTA polls early delays the stores that it waits
//     for.  Only the dots are polled for in the first exchange, the pivot row is
//     fetched once the dots have come, and no warp polls for columns that it
//     does not have;
//   * short code, since a step runs straight through the kernel once: at 104 KB
//     (waits inlined with per-slot branches, two-level rescaling, integer
//     divisions for the row numbers) a step took 11 us, at 43 KB 7.0.
// Measured on B200, reflectors only, ms:        512^2  1152x1024  1400^2  4096^2
//   rows in place, four grid barriers per step    -      54.4       -     693.6
//   slabs, two grid barriers per step            5.3     11.8       -     172
//   slots instead of barriers                    5.4     11.4       -     227
//   the same in 43 KB of code                    3.1      7.1      13.4   191
//   one pass for A r and its norm, few polls,
//   3 columns per thread (this kernel)           2.4      5.3       8.8   166
// U and V are formed afterwards from the stored reflectors by the blocked
// compact-WY Q builder of the QR route (GEMM kernels).
//
// Rounding: the norms and dots are summed in a different order from the
// reference's serial loops, so B, U and V agree with it to rounding.
#include <cstdio>

#include "jlc_device.cuh"
#include "jlc_internal.h"
#include "jlc_slab.cuh"

namespace jlc {
namespace bidiag {

constexpr int BT = 512;  // threads per CTA
constexpr int WARPS = BT / 32;
constexpr int RC = 8;     // rows per register block: a CTA holds a multiple of RC rows
constexpr int QL = 16;    // lanes over the CTAs in the cross-CTA sums (a warp sums 2 columns)
constexpr int QMAX = 10;  // partials per lane: QL * QMAX >= 148 CTAs
constexpr int PAIRS = 5;  // (exponent, sum) pairs per lane: 32 * PAIRS >= 148 CTAs
static_assert(32 * PAIRS == QL * QMAX, "one scale factor per CTA");
constexpr int kMaxCtas = 148;
constexpr int kMaxRows = 256;  // rows per CTA
constexpr double kSafeMin = 2.2250738585072014e-308;  // Double.MIN_NORMAL
constexpr int kEmptyExp = -4096;                      // exponent of an empty sum
constexpr int kSmemLimit = 224 * 1024;

struct Args {
    double* a;  // column-major m x n, m >= n
    long long lda;
    int m, n;
    int rows;     // rows per CTA (a multiple of RC): CTA c holds rows c, c + P, c + 2P, ...
    int ld;       // leading dimension of the slots and slab rows (n rounded up to 4)
    double* d;    // n: the diagonal of B
    double* e;    // n - 1: the superdiagonal of B
    double* tauq; // n: the column reflectors' tau
    double* taup; // n: the row reflectors' tau (n - 1 used)
    Slot* part;   // [CTA][ld]: dots of the pivot column with the trailing columns
    Slot* cpair;  // [2][CTA]: exponent and sum of squares of its rows of the pivot column
    Slot* pivot;  // [2][ld]: the pivot row before the column reflector
    Slot* w;      // ld: w_j = tau (row k's entry + the dots, rescaled)
    double* slab; // global slabs (null: the slab sits in shared memory)
    int* status;
    int withhold;  // test hook: CTA 0 leaves its first pair out, so the waits run out
};

// Sums of squares and dots are formed from values scaled by 2^-e, e the
// exponent of a maximum, and carried with e: nothing overflows or underflows
// whatever the range of the input, and every rescaling is exact.
__device__ __forceinline__ int exp_of(double x) {  // 2^e <= x < 2^(e+1) for a positive normal x, in [-1000, 1022]
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    return x > 0.0 && ex != 0x7ff ? min(1022, max(-1000, ex - 1023)) : 0;
}
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// 2^d for d <= 0, 0 where a term scaled by it is negligible
__device__ __forceinline__ double down(int d) { return d >= -1022 ? pow2(d) : 0.0; }

// The reference's reflector recipe for a vector with norm 2^E sqrt(S) (x0
// included) and first entry x0: tau, beta and 2^E / (x0 - beta); tau = 0 and
// beta = x0 when there is no reflector.  By a whole warp: its halves take one of
// the two quotients each (a quotient is 135 cycles).
struct Reflector {
    double tau, beta, inv;
};
__device__ __noinline__ Reflector reflector(int E, double S, double x0) {
    Reflector h{0.0, x0, 0.0};
    if (!(S > 0.0)) return h;
    const double p2 = pow2(E);
    const double xnorm = p2 * sqrt(S);
    if (xnorm > kSafeMin) {
        const double b = x0 >= 0.0 ? -xnorm : xnorm;
        const bool lower = (threadIdx.x & 16) == 0;
        const double q = (lower ? b - x0 : p2) / (lower ? b : x0 - b);
        const double t = __shfl_sync(0xffffffffu, q, 0), inv = __shfl_sync(0xffffffffu, q, 16);
        if (fabs(t) > kSafeMin) {
            h.tau = t;
            h.beta = b;
            h.inv = inv;
        }
    }
    return h;
}

template <bool SMEM, int CB, bool IN_PLACE = false>
__global__ void __launch_bounds__(BT, 1) bidiag_kernel(const Args p) {
    extern __shared__ double dyn[];
    // (aligned for vector loads: the passes read 8 rows of each)
    __shared__ __align__(16) double s_v[kMaxRows];  // the column reflector on this CTA's rows
    __shared__ __align__(16) double s_x[kMaxRows];  // tau_p (A u) on this CTA's rows
    __shared__ __align__(16) double s_c[kMaxRows];  // the pivot column on this CTA's rows (0 above the pivot)
    __shared__ __align__(16) double s_t[kMaxRows];  // its tail (0 at the pivot too)
    __shared__ unsigned s_mx[kMaxRows / RC];        // high word of the column's maximum per row block
    __shared__ double s_sum[WARPS], s_wy[WARPS];
    __shared__ int s_exp[WARPS];
    __shared__ double s_f[QL * QMAX];  // 2^(e_q - E) per CTA q
    __shared__ int s_E;
    __shared__ double s_x0, s_wk;      // the row reflector's first entry before it, w there
    __shared__ Reflector s_h, s_hr;    // the column reflector, the row reflector (inv: 1 / (x0 - beta))
    const int P = gridDim.x, cta = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m = p.m, n = p.n, rows = p.rows, ld = p.ld;
    double* slab = SMEM ? dyn : p.slab + (size_t)cta * rows * ld;  // [local row][column]
    const int live = (m - cta + P - 1) / P;                        // IN_PLACE: the matrix has no rows past these
    auto at = [&](int l, int j) -> double& {
        return IN_PLACE ? p.a[(long long)l * P + cta + j * p.lda] : slab[(size_t)l * ld + j];
    };
    double* red = SMEM ? dyn + (size_t)rows * ld : dyn;            // [warp][local row]
    Slot* part = p.part + (size_t)cta * ld;
    // f(local row, global row, column) over the slab.  A matrix of few columns takes several rows at a
    // time, a power of two of threads each (37000 x 2: 197 us row by row, 95 so)
    auto over_slab = [&](auto f) {
        int span = BT;
        while (span >= 2 * ld) span >>= 1;
        for (int l = tid / span; l < rows; l += BT / span) {
#pragma unroll 1
            for (int j = tid & (span - 1); j < ld; j += span) f(l, l * P + cta, j);
        }
    };
    // this CTA's rows into its slab (rows past m are zero)
    if constexpr (!IN_PLACE)
        over_slab([&](int l, int g, int j) {
            slab[(size_t)l * ld + j] = g < m && j < n ? p.a[g + (long long)j * p.lda] : 0.0;
        });
    for (int l = tid; l < rows; l += BT) {
        s_v[l] = 0.0;
        s_x[l] = 0.0;
    }
    __syncthreads();

    // The warps' sums of a row block (red, scaled by 2^-e of each warp's exponent; f lane i: 2^(e_i - E)
    // of warp i): four lanes per row, all with its sum
    auto row_sum = [&](int b, double f) {
        const int l = b * RC + (lane >> 2);
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < WARPS / 4; ++i) {
            const int q = (lane & 3) * (WARPS / 4) + i;
            s = fma(red[q * rows + l], __shfl_sync(0xffffffffu, f, q), s);
        }
        s += shfl_xor(s, 1);
        s += shfl_xor(s, 2);
        return s;
    };
    // x = tau_p (A - v w^T) u = tau_p (t + hinv (sum - v wy)), t the pivot column kn after the column
    // reflector, wy = 2^-E w . r; then the column after both, 0 above the pivot, and its maximum per
    // row block.  A warp per row block; s: the sums of the warp's first one.
    auto finish_rows = [&](int kn, int b0, double s, double f, double wk, double wy, double tau, double hinv) {
#pragma unroll 1
        for (int b = b0 + warp; b < rows / RC; b += WARPS) {
            if (b >= b0 + WARPS) s = row_sum(b, f);
            const int l = b * RC + (lane >> 2), g = l * P + cta;
            const double v = s_v[l], t = IN_PLACE && g >= m ? 0.0 : fma(-v, wk, at(l, kn));
            const bool in = g >= kn && g < m;
            const double x = in && tau != 0.0 ? tau * fma(hinv, fma(-v, wy, s), t) : 0.0;
            const double c = in ? t - x : 0.0;
            if ((lane & 3) == 0) {
                s_x[l] = x;
                s_c[l] = c;
                s_t[l] = g > kn ? c : 0.0;
            }
            const unsigned mx = __reduce_max_sync(0xffffffffu, max((unsigned)__double2hiint(c) & 0x7fffffffu, c != 0.0 ? 1u : 0u));
            if (lane == 0) s_mx[b] = mx;
        }
    };
    finish_rows(0, 0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
    __syncthreads();

    double w[CB], u[CB];  // w and u of this thread's columns
    int l0 = 0, gl = cta;  // the first of this CTA's rows at or past the pivot: local, global
    bool fail = false;    // a wait of this thread ran out
    for (int k = -1; k < n - 1; ++k) {
        const int kn = k + 1;    // the pivot whose dots are published below
        const int c0 = kn;       // first column of this step's update
        // pivot rows and pairs alternate between two buffers: a CTA may still wait for step
        // k's while a faster one, which needs w only, publishes those of step k + 1
        const Slot* prow = p.pivot + (size_t)(k & 1) * ld;
        Slot* pnext = p.pivot + (size_t)(kn & 1) * ld;
        Slot* cnext = p.cpair + (size_t)(kn & 1) * P;
        double u0 = 0.0, ir = 0.0;  // u at column kn (1, or 0 without a row reflector), 1 / (x0 - beta)
        // not SMEM: w of a column block and the scaled pivot row - w (u0 at column kn), from the
        // slots this thread has waited for
        auto reload = [&](int j0, double first, double scale) {
#pragma unroll
            for (int i = 0; i < CB; ++i) {
                const int j = j0 + tid + i * BT;
                w[i] = j < n ? slot_value(p.w + j) : 0.0;
                u[i] = j >= n ? 0.0 : j == kn ? first : (slot_value(prow + j) - w[i]) * scale;
            }
        };
        if (k >= 0) {
            // ---- the row reflector of row k: w of this thread's columns as it arrives, r = the
            // pivot row - w, the norm of r over the CTA (every warp the same bits)
            double rmax = 0.0;
            if constexpr (SMEM) {
                fail |= !slot_wait_columns<BT>(p.w, c0, n, kn, w, p.status);
#pragma unroll
                for (int i = 0; i < CB; ++i) {
                    if (c0 + tid + i * BT >= n) w[i] = u[i] = 0.0;
                    u[i] -= w[i];  // r
                    rmax = fmax(rmax, fabs(u[i]));
                }
                if (tid == 0) {
                    s_x0 = u[0];
                    s_wk = w[0];
                }
            } else {
#pragma unroll 1
                for (int j = c0 + tid; j < n; j += BT) {
                    const Slot* at[1] = {p.w + j};
                    double wj[1];
                    fail |= !slot_wait(at, kn, wj, p.status);
                    const double r = slot_value(prow + j) - wj[0];
                    rmax = fmax(rmax, fabs(r));
                    if (j == c0) {
                        s_x0 = r;
                        s_wk = wj[0];
                    }
                }
            }
            const bool owner = gl == k;
            const int lk = l0;  // row k
            if (owner) {
                ++l0;
                gl += P;
            }
            const int b0 = l0 / RC;
            // ---- pass 1, ahead of the norm: A r beyond column kn on this CTA's rows below k, r scaled
            // by 2^-e of the warp's maximum; the sums of the norm and of w . r go with it
            const int ew = warp_max(rmax > 0.0 ? exp_of(rmax) : kEmptyExp);
            const double sc = ew > kEmptyExp ? pow2(-ew) : 0.0;
            double S = 0.0, wy = 0.0, y[CB];
            if constexpr (SMEM) {
#pragma unroll
                for (int i = 0; i < CB; ++i) {
                    y[i] = ew > kEmptyExp ? u[i] * sc : 0.0;
                    S = fma(y[i], y[i], S);
                }
                if (tid == 0) y[0] = 0.0;  // column kn: finish_rows adds it
#pragma unroll
                for (int i = 0; i < CB; ++i) wy = fma(w[i], y[i], wy);
            } else if (ew > kEmptyExp) {
                for (int j = c0 + tid; j < n; j += BT) {
                    const double wj = slot_value(p.w + j), t = (slot_value(prow + j) - wj) * sc;
                    S = fma(t, t, S);
                    wy = fma(wj, j == kn ? 0.0 : t, wy);
                }
            }
#pragma unroll 1
            for (int b = b0; b < rows / RC; ++b) {
                double acc[RC];
#pragma unroll
                for (int r = 0; r < RC; ++r) acc[r] = 0.0;
                for (int j0 = c0; j0 < n; j0 += CB * BT) {
                    if constexpr (!SMEM) reload(j0, 0.0, sc);
#pragma unroll
                    for (int i = 0; i < CB; ++i) {
                        const int j = j0 + tid + i * BT;
                        const double yi = SMEM ? y[i] : u[i];
                        if (IN_PLACE && j < n) {
#pragma unroll
                            for (int r = 0; r < RC; ++r)
                                if (b * RC + r < live) acc[r] = fma(at(b * RC + r, j), yi, acc[r]);
                        } else if (j < n) {
                            const double* q = slab + (size_t)b * RC * ld + j;
#pragma unroll
                            for (int r = 0; r < RC; ++r) acc[r] = fma(q[(size_t)r * ld], yi, acc[r]);
                        }
                    }
                    if constexpr (SMEM) break;
                }
                const double s = warp_sum8(acc);
                if ((lane & 3) == 0) red[warp * rows + b * RC + (lane >> 2)] = s;
            }
            S = warp_sum(S);
            wy = warp_sum(wy);
            if (lane == 0) {
                s_sum[warp] = S;
                s_wy[warp] = wy;
                s_exp[warp] = ew;
            }
            if (__syncthreads_or(fail)) return;
            // ---- the row reflector of row k, x and the pivot column, by the warps that have row
            // blocks (each the same bits)
            if (warp == 0 || b0 + warp < rows / RC) {
                const int e = lane < WARPS ? s_exp[lane] : kEmptyExp;
                const int E = warp_max(e);
                const double f = down(e - E);
                S = warp_sum(lane < WARPS ? (s_sum[lane] * f) * f : 0.0);
                wy = warp_sum(lane < WARPS ? s_wy[lane] * f : 0.0);
                const double s = row_sum(min(b0 + warp, rows / RC - 1), f);
                const Reflector h = reflector(E, S, s_x0);
                finish_rows(kn, b0, s, f, s_wk, wy, h.tau, h.inv);
                if (tid == 0) {
                    s_hr.tau = h.tau;
                    s_hr.inv = h.tau != 0.0 ? h.inv * pow2(-E) : 0.0;
                    if (cta == 0) {
                        p.taup[k] = h.tau;
                        p.e[k] = h.beta;
                    }
                }
            }
            __syncthreads();
            u0 = s_hr.tau != 0.0 ? 1.0 : 0.0;
            ir = s_hr.inv;
            // row k is finished: x0 beside the diagonal, the reflector's tail beyond it
            if constexpr (SMEM) {
#pragma unroll
                for (int i = 0; i < CB; ++i) {
                    const int j = c0 + tid + i * BT;
                    const double rj = u[i];
                    u[i] = j == kn ? u0 : u0 != 0.0 ? rj * ir : 0.0;
                    if (owner && j < n) at(lk, j) = u0 != 0.0 && j > kn ? u[i] : rj;
                }
            } else if (owner) {
                for (int j = c0 + tid; j < n; j += BT) {
                    const double rj = slot_value(prow + j) - slot_value(p.w + j);
                    at(lk, j) = u0 != 0.0 && j > kn ? rj * ir : rj;
                }
            }
        }
        // ---- the pivot column scaled by 2^-e, e the exponent of this CTA's maximum
        const int b0 = l0 / RC;
        unsigned mx = 0;
#pragma unroll 1
        for (int b = b0; b < rows / RC; ++b) mx = max(mx, s_mx[b]);
        const int ex = mx >> 20 >= 0x7ff ? 0 : min(1022, max(-1000, (int)(mx >> 20) - 1023));
        const double sc = pow2(-ex);
        if (warp == WARPS - 1) {
            double q = 0.0;
#pragma unroll 1
            for (int l = b0 * RC + lane; l < rows; l += 32) {
                const double c = s_c[l] * sc;
                q = fma(c, c, q);
            }
            q = warp_sum(q);
            if (lane == 0 && !(p.withhold && cta == 0 && kn == 0)) slot_put(cnext + cta, q, kn + 1, mx > 0 ? ex : kEmptyExp);
        }
        // ---- pass 2: A - v w^T - x u^T stored, and its dots with the pivot column
        const bool powner = gl == kn;
        for (int j0 = c0; j0 < n; j0 += CB * BT) {
            double s[CB];
#pragma unroll
            for (int i = 0; i < CB; ++i) s[i] = 0.0;
            if (k < 0) {
#pragma unroll
                for (int i = 0; i < CB; ++i) w[i] = u[i] = 0.0;
            } else if constexpr (!SMEM) {
                reload(j0, u0, ir);
            }
#pragma unroll 1
            for (int b = b0; b < rows / RC; ++b) {
                double vr[RC], xr[RC], cr[RC];
#pragma unroll
                for (int r = 0; r < RC; ++r) {
                    const int l = b * RC + r;
                    vr[r] = s_v[l];
                    xr[r] = s_x[l];
                    cr[r] = s_t[l] * sc;
                }
#pragma unroll
                for (int i = 0; i < CB; ++i) {
                    const int j = j0 + tid + i * BT;
                    if (j < n) {
                        double* q = slab + (size_t)b * RC * ld + j;
                        double x[RC];
#pragma unroll
                        for (int r = 0; r < RC; ++r)
                            x[r] = !IN_PLACE ? q[(size_t)r * ld] : b * RC + r < live ? at(b * RC + r, j) : 0.0;
#pragma unroll
                        for (int r = 0; r < RC; ++r) {
                            x[r] = fma(-xr[r], u[i], fma(-vr[r], w[i], x[r]));
                            s[i] = fma(cr[r], x[r], s[i]);
                        }
#pragma unroll
                        for (int r = 0; r < RC; ++r)
                            if (b * RC + r >= l0 && (!IN_PLACE || b * RC + r < live))
                                (IN_PLACE ? at(b * RC + r, j) : q[(size_t)r * ld]) = x[r];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < CB; ++i) {
                const int j = j0 + tid + i * BT;
                if (j < n) {
                    slot_put(part + j, s[i], kn + 1, 0);
                    if (powner) slot_put(pnext + j, at(l0, j), kn + 1, 0);
                }
            }
        }
        // ---- the column reflector of column kn (the last warp), while the
        // others wait for the dots: a warp sums those of 2 columns, 16 lanes over the CTAs
        const int qi = lane >> 1, jj = lane & 1;
        int gr = (kn + 1) / 2 + cta + warp * P;  // group of 2 columns, absolute
        const int glast = (n + 1) / 2;
        if (warp == WARPS - 1) {
            double q[PAIRS + 1];  // the CTAs' sums of squares, and the pivot
            int eq[PAIRS + 1];
            const Slot* at[PAIRS + 1];
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) at[i] = cnext + min(lane + 32 * i, P - 1);
            at[PAIRS] = pnext + kn;
            fail |= !slot_wait(at, kn + 1, q, p.status, eq);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < PAIRS; ++i)
                if (lane + 32 * i >= P) eq[i] = kEmptyExp;
            int E = kEmptyExp;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) E = max(E, eq[i]);
            E = warp_max(E);
            double S = 0.0;
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const double f = lane + 32 * i < P ? down(eq[i] - E) : 0.0;
                S = fma(q[i] * f, f, S);
                s_f[lane + 32 * i] = f;
            }
            S = warp_sum(S);
            const Reflector h = reflector(E, S, q[PAIRS]);
            if (lane == 0) {
                s_h = h;
                s_E = E;
                if (cta == 0) {
                    p.tauq[kn] = h.tau;
                    p.d[kn] = h.beta;
                }
            }
        }
        double tau = 0.0, vinv = 0.0;
#pragma unroll 1
        for (int trip = 0, left = glast - (kn + 1) / 2; trip == 0 || left > 0; ++trip, left -= P * WARPS, gr += P * WARPS) {
            const int j = gr * 2 + jj;
            double x[QMAX + 1];  // the dots, and the pivot row's entry
            if (gr < glast) {
                // (lanes past the last CTA or column wait for a live one and drop what they get)
                const int jl = min(max(j, kn + 1), n - 1);
                const Slot* at[QMAX + 1];
#pragma unroll
                for (int i = 0; i < QMAX; ++i) at[i] = p.part + (size_t)min(qi + QL * i, P - 1) * ld + jl;
                at[QMAX] = pnext + jl;
                fail |= !slot_wait(at, kn + 1, x, p.status);
            }
            if (trip == 0) {
                if (__syncthreads_or(fail)) return;
                tau = s_h.tau;
                vinv = s_h.inv;
            }
            if (gr < glast) {
                __syncwarp();
                double s0 = 0.0, s1 = 0.0;
#pragma unroll
                for (int i = 0; i < QMAX; i += 2) {
                    s0 = fma(x[i], s_f[qi + QL * i], s0);
                    s1 = fma(x[i + 1], s_f[qi + QL * (i + 1)], s1);
                }
                double s = s0 + s1;
#pragma unroll
                for (int o = 2; o < 32; o <<= 1) s += shfl_xor(s, o);
                if (qi == 0 && j > kn && j < n) slot_put(p.w + j, tau != 0.0 ? tau * fma(s, vinv, x[QMAX]) : 0.0, kn + 1, 0);
            }
        }
        // v on this CTA's rows, its tail stored below the diagonal
        if (tid >= BT - kMaxRows && tid - (BT - kMaxRows) < rows) {
            const int l = tid - (BT - kMaxRows), g = l * P + cta;
            double v = 0.0;
            if (tau != 0.0 && g >= kn && g < m) {
                v = g == kn ? 1.0 : (s_c[l] * pow2(-s_E)) * vinv;
                if (g > kn) at(l, kn) = v;
            }
            s_v[l] = v;
        }
        // the pivot row at this thread's columns of the next step, which has long arrived (waiting
        // for it ahead of the dots, every thread polls and delays them: 7.0 us a step against 6.3)
        if constexpr (SMEM) {
            fail |= !slot_wait_columns<BT>(pnext, kn + 1, n, kn + 1, u, p.status);
        } else {
#pragma unroll 1
            for (int c = kn + 1 + tid; c < n; c += BT) {
                const Slot* at[1] = {pnext + c};
                double y[1];
                fail |= !slot_wait(at, kn + 1, y, p.status);
            }
        }
    }
    __syncthreads();
    if constexpr (!IN_PLACE) over_slab([&](int l, int g, int j) {
        if (g < m && j < n) p.a[g + (long long)j * p.lda] = slab[(size_t)l * ld + j];
    });
}

// Right reflectors, stored in the rows of A beyond the superdiagonal, as the
// columns of a factor: W(r, k) = A(k, r) for r > k + 1 (k < n - 1).
__global__ void bidiag_right_factor_kernel(const double* a, long long lda, int n, double* w, long long ldw) {
    const int k = blockIdx.y;
    for (int r = k + 2 + blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        w[r + (long long)k * ldw] = a[k + (long long)r * lda];
}

}  // namespace bidiag

// The number of CTAs for an m-row reduction and the rows each holds (row g on
// CTA g % P, so that every CTA keeps rows in play to the last steps); 0 when
// a CTA would hold more than 256 rows.
int bidiag_grid(int m, int n, int sm_count, int* rows) {
    using namespace bidiag;
    const int most = sm_count < kMaxCtas ? sm_count : kMaxCtas;
    int per = ((m + most - 1) / most + RC - 1) / RC * RC;
    // past two columns per thread 16 rows per CTA (1168 x 1100: 6.7 ms, against 7.0 with 8: half as
    // many partials cross), below it 8 (1152 x 1024: 5.4 against 6.0; 512^2: 2.45 against 2.7)
    if (n > 2 * BT && per < 2 * RC) per = 2 * RC;
    if (per > kMaxRows) return 0;
    *rows = per;
    return (m + per - 1) / per;
}

namespace bidiag {
static size_t smem_bytes(int rows, int ld, bool slab) {
    return ((slab ? (size_t)rows * ld : 0) + (size_t)WARPS * rows) * sizeof(double);
}
static bool slab_in_smem(int rows, int n, int ld) {
    return n <= 4 * BT && smem_bytes(rows, ld, true) + 16 * 1024 <= (size_t)kSmemLimit;
}
}  // namespace bidiag

// Slots of the exchange: part, cpair, pivot and w.
static size_t bidiag_slots(int P, int ld) { return (size_t)P * ld + 2 * (size_t)P + 3 * (size_t)ld; }

// Work array: the slots, then (slab_doubles) the global slabs.
size_t bidiag_work_doubles(int m, int n, int sm_count, size_t* slab_doubles) {
    using namespace bidiag;
    int rows = 0;
    const int P = bidiag_grid(m, n, sm_count, &rows), ld = (n + 3) / 4 * 4;
    *slab_doubles = slab_in_smem(rows, n, ld) ? 0 : (size_t)P * rows * ld;
    return 2 * bidiag_slots(P, ld);
}

int launch_bidiag(double* a, long long lda, int m, int n, double* d, double* e, double* tauq, double* taup,
                  double* work, bool in_place, int sm_count, int* status, bool withhold, cudaStream_t st) {
    using namespace bidiag;
    Args p;
    int rows = 0;
    const int P = bidiag_grid(m, n, sm_count, &rows);
    if (P == 0) return JLC_E_UNSUPPORTED;
    p.a = a;
    p.lda = lda;
    p.m = m;
    p.n = n;
    p.rows = rows;
    p.ld = (n + 3) / 4 * 4;
    p.d = d;
    p.e = e;
    p.tauq = tauq;
    p.taup = taup;
    const size_t slots = bidiag_slots(P, p.ld);
    p.part = reinterpret_cast<Slot*>(work);
    p.cpair = p.part + (size_t)P * p.ld;
    p.pivot = p.cpair + 2 * P;
    p.w = p.pivot + 2 * (size_t)p.ld;
    const bool smem = slab_in_smem(rows, n, p.ld);
    p.slab = smem || in_place ? nullptr : work + 2 * slots;
    p.status = status;
    p.withhold = withhold ? 1 : 0;
    // (1400^2: 9.0 ms with 3 columns per thread, 11.4 with 4; up to 512 columns 1 gains nothing on 2)
    const void* kern = !smem        ? in_place ? (const void*)bidiag_kernel<false, 4, true> : (const void*)bidiag_kernel<false, 4>
                       : n > 3 * BT ? (const void*)bidiag_kernel<true, 4>
                       : n > 2 * BT ? (const void*)bidiag_kernel<true, 3>
                                    : (const void*)bidiag_kernel<true, 2>;
    const size_t bytes = smem_bytes(rows, p.ld, smem);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
        return JLC_E_LAUNCH;
    // no slot may hold a tag of an earlier call
    if (cudaMemsetAsync(work, 0, slots * sizeof(Slot), st) != cudaSuccess) return JLC_E_CUDA;
    void* args[] = {&p};
    cudaError_t err = cudaLaunchCooperativeKernel(kern, dim3(P), dim3(BT), args, bytes, st);
    return err == cudaSuccess ? JLC_OK : JLC_E_LAUNCH;
}

int launch_bidiag_right_factor(const double* a, long long lda, int n, double* w, long long ldw, cudaStream_t st) {
    if (n < 3) return JLC_OK;
    dim3 grid((unsigned)((n + 255) / 256 > 16 ? 16 : (n + 255) / 256), (unsigned)(n - 1));
    bidiag::bidiag_right_factor_kernel<<<grid, 256, 0, st>>>(a, lda, n, w, ldw);
    return cudaGetLastError() == cudaSuccess ? JLC_OK : JLC_E_LAUNCH;
}

}  // namespace jlc
