// HBM-bound kernels: matrix-vector product (the n == 1 / m == 1 shapes that
// GemmDispatch routes to SpecializedKernels.matvec, GemmDispatch.java:80-82,
// SpecializedKernels.java:27-71) and the beta-only update of C
// (PackingUtils.scaleCPanel, PackingUtils.java:159-183).
#include <cstdio>

#include <cooperative_groups.h>

#include "jlc_device.cuh"
#include "jlc_internal.h"

namespace jlc {
namespace {

namespace cg = cooperative_groups;

constexpr int GEMV_THREADS = 256, GEMV_WARPS = GEMV_THREADS / 32;
constexpr int GEMV_LOADS = 16;     // matrix loads a lane keeps in flight (dot form)
constexpr int GEMV_AXPY_CTAS = 8;  // resident CTAs per SM (axpy form)

// How a product's rows and columns are dealt to CTAs.  The kernels are bound by
// HBM, so every SM needs enough loads in flight and an equal share of the work: a
// wave of CTAs, or many short waves.  A dot-form CTA that owned 32 rows left 512
// CTAs for 16384 rows, 3.46 per SM, so that the SMs with three idled while the
// others ran a fourth, and 16 CTAs for 512 rows.  The warps of a CTA therefore
// split the columns wk ways as the rows run out, each warp takes fewer rows, and
// at last the columns are split over CTAs.  us before -> after, A row-major:
// 16384^2 371 -> 335 (6.4 TB/s), 4096 x 8192 145 -> 44, 512 x 16384 293 -> 16;
// column-major: 16384^2 457 -> 316, 2000 x 16000 67 -> 49, 512 x 16384 60 -> 26.
// (16384^2 by rows is 1024 CTAs, 6.9 per SM and four of them resident.)
struct GemvShape {
    int rows_per_warp;  // dot form: 4, 2 or 1
    int wk;             // warps that share a row group and split its columns (1, 2, 4, 8)
    int chunks;         // column chunks over CTAs (dot form: of a cluster; else partial sums in scratch when > 1)
    long long chunk;    // columns per chunk
};

__device__ __forceinline__ void gemv_store(const GemvDesc& g, long long row, double s) {
    double* y = g.y + row * g.incy;
    *y = (g.beta == 0.0) ? g.alpha * s : fma(g.alpha, s, g.beta * *y);
}

// Dot form: M(i,p) = mat[i*rs + p]; a warp takes R rows (x is loaded once for
// them) of its share of the columns, lanes along the row.
// U steps of 32 columns are in flight (U = 1, matrices of at most 64 columns: wk = 1).
// Four CTAs of the <4> form fit an SM at 64 registers (8192 x 16384: 159 us; 167 with three).
// CLUSTER: the chunks of the same rows are the CTAs of a cluster, the first of which adds their sums
// in order, so that a few long rows need neither scratch nor a second kernel.
template <int R, int U = GEMV_LOADS / R, bool CLUSTER = false>
__global__ void __launch_bounds__(GEMV_THREADS, R == 4 ? 4 : 1) gemv_dot_kernel(GemvDesc g, int lwk0, long long chunk) {
    __shared__ double red[GEMV_WARPS * R];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lwk = U == 1 ? 0 : lwk0, wk = 1 << lwk;  // (shifts: a 64-bit division is long)
    const long long row0 = ((long long)blockIdx.x * (GEMV_WARPS >> lwk) + (warp >> lwk)) * R;
    const long long c0 = (long long)blockIdx.y * chunk, c1 = c0 + chunk < g.cols ? c0 + chunk : g.cols;
    // this warp's columns: its share of the chunk in whole trips
    const long long trips = (c1 - c0 + 32 * U - 1) / (32 * U), per = ((trips + wk - 1) >> lwk) * (32 * U);
    const long long p0 = c0 + (warp & (wk - 1)) * per, p1 = p0 + per < c1 ? p0 + per : c1;
    double acc[R];
    const double* rowp[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        acc[r] = 0.0;
        const long long row = row0 + r < g.rows ? row0 + r : g.rows - 1;
        rowp[r] = g.mat + row * g.rs;
    }
    long long p = p0 + lane;
    for (; p + 32 * (U - 1) < p1; p += 32 * U) {
        double xv[U], m[R][U];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) m[r][u] = __ldcs(rowp[r] + p + 32 * u);
#pragma unroll
        for (int u = 0; u < U; ++u) xv[u] = __ldg(g.x + (p + 32 * u) * g.incx);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) acc[r] = fma(m[r][u], xv[u], acc[r]);
    }
    if (p < p1) {
        double xv[U], m[R][U];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) m[r][u] = p + 32 * u < p1 ? __ldcs(rowp[r] + p + 32 * u) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) xv[u] = p + 32 * u < p1 ? __ldg(g.x + (p + 32 * u) * g.incx) : 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (p + 32 * u < p1) acc[r] = fma(m[r][u], xv[u], acc[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    double mine = acc[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
        if (lane == r) mine = acc[r];
    const bool lead = (warp & (wk - 1)) == 0;
    if (wk > 1) {
        if (lane < R) red[warp * R + lane] = mine;
        __syncthreads();
        if (!CLUSTER && !lead) return;
        if (lead && lane < R) {
            mine = 0.0;
            for (int w = 0; w < wk; ++w) mine += red[(warp + w) * R + lane];
        }
    }
    if (CLUSTER) {
        __shared__ double sum[GEMV_WARPS * R];
        cg::cluster_group cluster = cg::this_cluster();
        double* slot = &sum[(warp >> lwk) * R + lane % R];
        if (lead && lane < R) *slot = mine;
        cluster.sync();
        const bool first = cluster.block_rank() == 0;
        if (first && lead && lane < R)
            for (unsigned q = 1; q < cluster.num_blocks(); ++q) mine += *cluster.map_shared_rank(slot, q);
        cluster.sync();  // (no CTA leaves while its sums are read)
        if (!first || !lead) return;
    }
    const long long row = row0 + lane;
    if (lane < R && row < g.rows) gemv_store(g, row, mine);
}

// Axpy form: M(i,p) = mat[i + p*cs]; lanes own rows, the WK warps of a row group
// split the chunk's columns, partial sums go to scratch[chunk][row] (one chunk:
// no scratch, 10^6 x 2 in 8.3 us against 28.8 with a second kernel).
template <int WK, bool DIRECT>
__global__ void __launch_bounds__(GEMV_THREADS) gemv_axpy_partial_kernel(GemvDesc g, double* partial, long long chunk) {
    __shared__ double red[WK > 1 ? GEMV_THREADS : 1];
    const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) % WK;
    const long long row = (long long)blockIdx.x * (GEMV_THREADS / WK) + (threadIdx.x >> 5) / WK * 32 + lane;
    if (WK == 1 && row >= g.rows) return;
    const long long c0 = (long long)blockIdx.y * chunk;
    const long long c1 = c0 + chunk < g.cols ? c0 + chunk : g.cols;
    const long long per = WK == 1 ? c1 - c0 : (c1 - c0 + WK - 1) / WK;
    const long long p0 = c0 + part * per;
    const long long p1 = WK == 1 || p0 + per > c1 ? c1 : p0 + per;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (WK == 1 || row < g.rows) {
        long long p = p0;
        for (; p + 3 < p1; p += 4) {
            a0 = fma(__ldcs(g.mat + row + (p + 0) * g.cs), __ldg(g.x + (p + 0) * g.incx), a0);
            a1 = fma(__ldcs(g.mat + row + (p + 1) * g.cs), __ldg(g.x + (p + 1) * g.incx), a1);
            a2 = fma(__ldcs(g.mat + row + (p + 2) * g.cs), __ldg(g.x + (p + 2) * g.incx), a2);
            a3 = fma(__ldcs(g.mat + row + (p + 3) * g.cs), __ldg(g.x + (p + 3) * g.incx), a3);
        }
        for (; p < p1; ++p) a0 = fma(__ldcs(g.mat + row + p * g.cs), __ldg(g.x + p * g.incx), a0);
    }
    double s = (a0 + a1) + (a2 + a3);
    if (WK > 1) {
        red[threadIdx.x] = s;
        __syncthreads();
        if (part != 0) return;
#pragma unroll
        for (int w = 1; w < WK; ++w) s += red[threadIdx.x + 32 * w];
    }
    if (WK == 1 || row < g.rows) {
        if (DIRECT) gemv_store(g, row, s);
        else partial[(long long)blockIdx.y * g.rows + row] = s;
    }
}

// y from the chunks' partial sums: 32 rows per CTA, its warps split the chunks
__global__ void __launch_bounds__(GEMV_THREADS) gemv_reduce_kernel(GemvDesc g, const double* partial, int nchunks) {
    __shared__ double red[GEMV_THREADS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long row = (long long)blockIdx.x * 32 + lane;
    double s = 0.0;
    if (row < g.rows) {
#pragma unroll 8
        for (int c = warp; c < nchunks; c += GEMV_WARPS) s += partial[(long long)c * g.rows + row];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    if (warp != 0 || row >= g.rows) return;
    s = 0.0;
    for (int w = 0; w < GEMV_WARPS; ++w) s += red[lane + 32 * w];
    gemv_store(g, row, s);
}

__global__ void scale_c_kernel(double* c, long long ldc, long long m, long long n, double beta) {
    const long long total = m * n;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long i = e / n, j = e % n;
        double* p = c + i * ldc + j;
        *p = (beta == 0.0) ? 0.0 : *p * beta;
    }
}

GemvShape gemv_shape(const GemvDesc& g, int sm_count) {
    const long long target = 6LL * sm_count;
    GemvShape s{4, 1, 1, g.cols};
    if (g.cs == 1) {
        auto ctas = [&] { return (g.rows * s.wk + (long long)GEMV_WARPS * s.rows_per_warp - 1) / (GEMV_WARPS * s.rows_per_warp); };
        // A warp keeps at least 128 columns, a trip at four rows.  With fewer rows a trip is 256 or 512
        // columns, and the last warps of a short row have none (512 x 1024: two of eight have).
        while (ctas() < target && s.wk < GEMV_WARPS && g.cols >= 2 * s.wk * 128) s.wk *= 2;
        while (ctas() < target && s.rows_per_warp > 1) s.rows_per_warp /= 2;
        const long long most = g.cols / (512 * s.wk);  // chunks of at least 512 columns per warp
        if (ctas() < target / 2 && most > 1) {
            long long want = (target + ctas() - 1) / ctas();
            if (want > most) want = most;
            if (want > 8) want = 8;  // CTAs of a cluster
            s.chunk = (g.cols + want - 1) / want;
        }
    } else {
        // CTAs of 256 rows (2 KB runs of each column) over column chunks, as many as are resident at
        // once and no more (a second wave of a few CTAs took 457 us at 16384^2, one wave 330); where
        // that is too few CTAs, the warps of a CTA split the columns.  At least 32 columns per warp.
        const long long groups = (g.rows + 31) / 32, resident = (long long)GEMV_AXPY_CTAS * sm_count;
        long long want = 1;
        for (s.wk = 1;; s.wk *= 2) {
            const long long ctas = (groups * s.wk + GEMV_WARPS - 1) / GEMV_WARPS;
            const long long most = g.cols / (32 * s.wk);
            want = resident / ctas;
            if (want > most) want = most;
            if (want > 256) want = 256;
            if (want < 1) want = 1;
            if (s.wk == GEMV_WARPS || 2 * ctas * want >= resident || g.cols < 64 * s.wk) break;
        }
        s.chunk = (g.cols + want - 1) / want;
    }
    s.chunks = (int)((g.cols + s.chunk - 1) / s.chunk);
    return s;
}

}  // namespace

// partial sums of the axpy form, when the columns are split over CTAs
size_t gemv_scratch_bytes(const GemvDesc& g, int sm_count) {
    if (g.rows <= 0 || g.cols <= 0) return 0;
    const GemvShape s = gemv_shape(g, sm_count);
    return g.cs == 1 || s.chunks == 1 ? 0 : (size_t)s.chunks * (size_t)g.rows * sizeof(double);
}

int launch_gemv(const GemvDesc& g, void* scratch, cudaStream_t st, int sm_count, char* err, size_t errlen) {
    if (g.rows <= 0) return JLC_OK;
    if (g.cs != 1 && g.rs != 1) {
        snprintf(err, errlen, "gemv needs a unit row or column stride");
        return JLC_E_UNSUPPORTED;
    }
    const GemvShape s = gemv_shape(g, sm_count);
    double* partial = g.cs == 1 || s.chunks == 1 ? nullptr : static_cast<double*>(scratch);
    const long long groups = g.cs == 1 ? (g.rows + s.rows_per_warp - 1) / s.rows_per_warp : (g.rows + 31) / 32;
    const dim3 grid((unsigned)((groups * s.wk + GEMV_WARPS - 1) / GEMV_WARPS), (unsigned)s.chunks);
    if (g.cs == 1) {
        const int lwk = s.wk == 8 ? 3 : s.wk >> 1;
        if (s.chunks > 1) {  // (few rows: one per warp)
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            cfg.gridDim = grid;
            cfg.blockDim = dim3(GEMV_THREADS);
            cfg.stream = st;
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 1;
            at[0].val.clusterDim.y = (unsigned)s.chunks;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, gemv_dot_kernel<1, GEMV_LOADS, true>, g, lwk, s.chunk);
        } else {
            // (rows of at most 64 columns keep fewer loads than registers would be held for: 10^6 x 2
            // 122 -> 80 us, 200000 x 16 27.8 -> 18.8)
            auto kern = s.rows_per_warp == 4   ? g.cols <= 64 ? gemv_dot_kernel<4, 1> : gemv_dot_kernel<4>
                        : s.rows_per_warp == 2 ? gemv_dot_kernel<2>
                                               : gemv_dot_kernel<1>;
            kern<<<grid, GEMV_THREADS, 0, st>>>(g, lwk, s.chunk);
        }
    } else {
        auto kern = s.wk == 1   ? partial ? gemv_axpy_partial_kernel<1, false> : gemv_axpy_partial_kernel<1, true>
                    : s.wk == 2 ? partial ? gemv_axpy_partial_kernel<2, false> : gemv_axpy_partial_kernel<2, true>
                    : s.wk == 4 ? partial ? gemv_axpy_partial_kernel<4, false> : gemv_axpy_partial_kernel<4, true>
                    : partial   ? gemv_axpy_partial_kernel<8, false>
                                : gemv_axpy_partial_kernel<8, true>;
        kern<<<grid, GEMV_THREADS, 0, st>>>(g, partial, s.chunk);
    }
    if (partial)
        gemv_reduce_kernel<<<(unsigned)((g.rows + 31) / 32), GEMV_THREADS, 0, st>>>(g, partial, s.chunks);
    if (cudaGetLastError() != cudaSuccess) {
        snprintf(err, errlen, "gemv launch failed");
        return JLC_E_LAUNCH;
    }
    return JLC_OK;
}

int launch_scale_c(double* c, long long ldc, long long m, long long n, double beta, cudaStream_t st) {
    if (m <= 0 || n <= 0 || beta == 1.0) return JLC_OK;
    long long total = m * n;
    long long blocks = (total + 255) / 256;
    if (blocks > 148LL * 16) blocks = 148LL * 16;
    scale_c_kernel<<<(unsigned)blocks, 256, 0, st>>>(c, ldc, m, n, beta);
    return cudaGetLastError() == cudaSuccess ? JLC_OK : JLC_E_LAUNCH;
}

}  // namespace jlc
