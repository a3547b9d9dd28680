// libjlcgpu C ABI: contexts, argument validation, host staging and dispatch.
//
// The host entries replace net.faulj.compute.CudaGemm (CudaGemm.java:53-134),
// which paid cublasCreate + cudaMalloc x3 + free x3 on every call: here a
// context keeps its stream, its device buffers (grow-only) and its workspace
// across calls, and only the copies of the operands remain per call.
#include <cudaTypedefs.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "jlc_internal.h"

using namespace jlc;

namespace {

int set_err(jlc_ctx* ctx, int code, const char* fmt, ...) {
    if (ctx) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(ctx->err, sizeof(ctx->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

int cuda_err(jlc_ctx* ctx, cudaError_t e, const char* what) {
    if (e == cudaErrorMemoryAllocation) return set_err(ctx, JLC_E_OOM, "%s: %s", what, cudaGetErrorString(e));
    return set_err(ctx, JLC_E_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int reserve(jlc_ctx* ctx, DevBuf& b, size_t bytes, const char* what) {
    if (fault_hit(ctx, JLC_FAULT_ALLOC)) return set_err(ctx, JLC_E_OOM, "%s: injected allocation failure", what);
    if (bytes <= b.bytes) return JLC_OK;
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
    size_t want = bytes + bytes / 8;  // grow with slack, like GemmWorkspace's grow-only buffers
    cudaError_t e = cudaMalloc(&b.ptr, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        e = cudaMalloc(&b.ptr, bytes);
        if (e != cudaSuccess) {
            cudaGetLastError();
            b.ptr = nullptr;
            return cuda_err(ctx, e, what);
        }
        want = bytes;
    }
    b.bytes = want;
    return JLC_OK;
}

inline long long round_up(long long v, long long m) { return (v + m - 1) / m * m; }

// the context workspace, grown on demand (and the allocation test hook)
int ws_reserve(jlc_ctx* ctx, size_t bytes) {
    if (fault_hit(ctx, JLC_FAULT_ALLOC)) return set_err(ctx, JLC_E_OOM, "workspace: injected allocation failure");
    return workspace_reserve(ctx->ws, bytes, ctx->err, sizeof(ctx->err));
}

bool capturing(jlc_ctx* ctx) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(ctx->stream, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusActive;
}

// The counters of a split product about to be launched.  Each launch has a number
// of its own, so that nothing an earlier one left in them matters, whichever
// stream it ran on and however it ended.  A captured launch keeps its number
// from replay to replay: its counters are cleared in the graph.
SplitCounters split_counters(jlc_ctx* ctx) {
    if (capturing(ctx)) cudaMemsetAsync(ctx->d_counters, 0, kSplitTiles * sizeof(*ctx->d_counters), ctx->stream);
    return {ctx->d_counters, ++ctx->split_launches << kSplitShift};
}

// a failed copy of the single-shot host entry: the stream is drained so the
// context is idle when the error returns
int copy_failed(jlc_ctx* ctx, cudaError_t e, const char* what) {
    const int rc = cuda_err(ctx, e, what);
    cudaStreamSynchronize(ctx->stream);
    cudaGetLastError();
    return rc;
}

// Phase markers for the profiler: begin() records the start event of a new
// record, end() its stop event.  Both are no-ops when profiling is off or the
// record buffer is full.
struct Phase {
    jlc_ctx* ctx;
    cudaStream_t st;
    int idx = -1;
    Phase(jlc_ctx* c, int phase, cudaStream_t s = nullptr) : ctx(c), st(s ? s : c->stream) {
        if (!ctx->profiling || ctx->nrec >= jlc_ctx::kMaxRec) return;
        idx = ctx->nrec++;
        for (int e = 0; e < 2; ++e)
            if (!ctx->rec_ev[2 * idx + e]) cudaEventCreate(&ctx->rec_ev[2 * idx + e]);
        ctx->rec_phase[idx] = phase;
        cudaEventRecord(ctx->rec_ev[2 * idx], st);
    }
    ~Phase() {
        if (idx >= 0) cudaEventRecord(ctx->rec_ev[2 * idx + 1], st);
    }
};

// Validation shared by host and device entries: the IllegalArgumentException
// cases of CudaGemm.gemm / OptimizedBLAS3.gemm (null matrices, negative sizes,
// leading dimensions too small for the declared shape).
int validate(jlc_ctx* ctx, int la, int lb, long long m, long long n, long long k, const void* a, long long lda,
             const void* b, long long ldb, const void* c, long long ldc) {
    if (!ctx) return JLC_E_ARG;
    if (m < 0 || n < 0 || k < 0) return set_err(ctx, JLC_E_ARG, "dimensions must be non-negative");
    if ((la != JLC_ROW_MAJOR && la != JLC_COL_MAJOR) || (lb != JLC_ROW_MAJOR && lb != JLC_COL_MAJOR))
        return set_err(ctx, JLC_E_ARG, "layout must be JLC_ROW_MAJOR or JLC_COL_MAJOR");
    if (m > 0 && n > 0 && c == nullptr) return set_err(ctx, JLC_E_ARG, "Matrices must not be null");
    if (m > 0 && n > 0 && ldc < n) return set_err(ctx, JLC_E_ARG, "ldc (%lld) < n (%lld)", ldc, n);
    if (m > 0 && n > 0 && k > 0) {
        if (a == nullptr || b == nullptr) return set_err(ctx, JLC_E_ARG, "Matrices must not be null");
        const long long need_a = la == JLC_ROW_MAJOR ? k : m;
        const long long need_b = lb == JLC_ROW_MAJOR ? n : k;
        if (lda < need_a) return set_err(ctx, JLC_E_ARG, "lda (%lld) too small (need >= %lld)", lda, need_a);
        if (ldb < need_b) return set_err(ctx, JLC_E_ARG, "ldb (%lld) too small (need >= %lld)", ldb, need_b);
    }
    if (m > INT32_MAX / 2 || n > INT32_MAX / 2 || k > INT32_MAX / 2)
        return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^30");
    return JLC_OK;
}

void report_init(jlc_report* rep) {
    if (rep) memset(rep, 0, sizeof(*rep));
}

}  // namespace

namespace jlc {

// a host <-> device copy of a host entry (and the copy test hook)
cudaError_t copy2d(jlc_ctx* ctx, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                   size_t height, cudaMemcpyKind kind, cudaStream_t st) {
    if (fault_hit(ctx, JLC_FAULT_COPY)) return cudaErrorUnknown;
    return cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, height, kind, st);
}
// The matrix-vector form of a GEMM with n == 1 or m == 1.
GemvDesc gemv_desc(const GemmDesc& g) {
    GemvDesc v;
    if (g.n == 1) {
        // y = C(:,0), rows of op(A) dotted with x = B(:,0)
        v.rows = g.m;
        v.cols = g.k;
        v.mat = g.a;
        v.rs = g.layout_a == JLC_ROW_MAJOR ? g.lda : 1;
        v.cs = g.layout_a == JLC_ROW_MAJOR ? 1 : g.lda;
        v.x = g.b;
        v.incx = g.layout_b == JLC_ROW_MAJOR ? g.ldb : 1;
        v.y = g.c;
        v.incy = g.ldc;
    } else {
        // y^T = C(0,:) = A(0,:) * B  ->  y = B^T x with x = A(0,:)
        v.rows = g.n;
        v.cols = g.k;
        v.mat = g.b;
        v.rs = g.layout_b == JLC_ROW_MAJOR ? 1 : g.ldb;
        v.cs = g.layout_b == JLC_ROW_MAJOR ? g.ldb : 1;
        v.x = g.a;
        v.incx = g.layout_a == JLC_ROW_MAJOR ? 1 : g.lda;
        v.y = g.c;
        v.incy = 1;
    }
    v.alpha = g.alpha;
    v.beta = g.beta;
    if (v.cs != 1 && v.rs != 1) {
        // single row/column with both strides > 1 cannot happen for a
        // matrix operand; k == 1 makes either stride irrelevant
        if (v.cols == 1) v.cs = 1;
        else if (v.rows == 1) v.rs = 1;
    }
    return v;
}
}  // namespace jlc

namespace {

bool use_ozaki(int precision, long long m, long long n, long long k) {
    if (precision == JLC_PREC_OZAKI || precision == JLC_PREC_OZAKI_CRT) return true;
    if (precision == JLC_PREC_NATIVE) return false;
    return m >= 2048 && n >= 2048 && k >= 1024;  // AUTO: large products only
}

// Device dispatch on already-validated device operands.
int run_device(jlc_ctx* ctx, const GemmDesc& g0, int precision, int slices, jlc_report* rep) {
    GemmDesc g = g0;
    ctx->cert_pending = false;
    if (rep) rep->precision = JLC_PREC_NATIVE;
    if (g.m == 0 || g.n == 0) {
        if (rep) rep->kernel = JLC_KERNEL_NONE;
        return JLC_OK;
    }
    if (fault_hit(ctx, JLC_FAULT_LAUNCH)) return set_err(ctx, JLC_E_LAUNCH, "injected kernel launch failure");
    if (g.alpha == 0.0 || g.k == 0) {
        if (rep) rep->kernel = JLC_KERNEL_NONE;
        if (g.beta == 1.0) return JLC_OK;
        Phase ph(ctx, JLC_PHASE_SCALE);
        ctx->launches += 1;
        int rc = launch_scale_c(g.c, g.ldc, g.m, g.n, g.beta, ctx->stream);
        return rc ? set_err(ctx, rc, "scale kernel launch failed") : JLC_OK;
    }
    if (g.n == 1 || g.m == 1) {
        const GemvDesc v = gemv_desc(g);
        size_t need = gemv_scratch_bytes(v, ctx->sm_count);
        if (need) {
            int rc = ws_reserve(ctx, need);
            if (rc) return rc;
        }
        if (rep) rep->kernel = JLC_KERNEL_GEMV;
        Phase ph(ctx, JLC_PHASE_GEMV);
        ctx->launches += need == 0 ? 1 : 2;
        return launch_gemv(v, ctx->ws.ptr, ctx->stream, ctx->sm_count, ctx->err, sizeof(ctx->err));
    }
    // a row block of a pipelined product follows the whole product's choice
    const long long whole_m = g.ws_m > g.m ? g.ws_m : g.m;
    // AUTO takes the residue scheme: fewer INT8 products for the same bound;
    // an automatic count that cannot reach the bound for this k means FP64
    const bool crt_req = precision != JLC_PREC_OZAKI;
    const bool ozaki = use_ozaki(precision, whole_m, g.n, g.k) && (slices > 0 || ozaki_reaches_bound(g.k, crt_req));
    const bool crt = ozaki && crt_req;
    // Small products split k across CTAs, partials in the workspace (after
    // the Ozaki split data when the FP64 kernel is the gated fallback, so
    // that its split choice, and with it its sums, match the native route).
    int ksplit = g.dot_mat ? 1 : dmma_splitk(whole_m, g.n, g.k, ctx->sm_count, ctx->dmma_k);
    size_t splitk_bytes = dmma_splitk_bytes(g.m, whole_m, g.n, g.k, ksplit, ctx->sm_count, ctx->dmma_k);
    size_t splitk_off = 0;
    int rc = JLC_OK;
    if (ozaki) {
        // The higher count re-splits op(B): not for row blocks that share
        // one split of it (they fall back to FP64 instead).
        const OzakiPlan pl = ozaki_plan(g.k, crt, slices, whole_m == g.m);
        size_t need = ozaki_workspace_bytes(whole_m, g.n, g.k, pl, ctx->sm_count);
        splitk_off = (need + 255) / 256 * 256;
        if (splitk_bytes) need = splitk_off + splitk_bytes;
        rc = ws_reserve(ctx, need);
        if (rc) return rc;
        void* ws = ctx->ws.ptr;
        const size_t wsb = ctx->ws.bytes;
        int nl = 0;
        {
            Phase ph(ctx, JLC_PHASE_OZAKI_SPLIT);
            rc = launch_ozaki_split(g, pl, 0, ws, wsb, ctx->stream, ctx->sm_count, ctx->d_flags, ctx->err,
                                    sizeof(ctx->err), &nl);
        }
        if (!rc) {
            Phase ph(ctx, JLC_PHASE_OZAKI_CERT);
            nl += 1;
            rc = launch_ozaki_cert(g, pl, ws, wsb, ctx->stream, ctx->sm_count, ctx->d_status, ctx->d_flags, ctx->err,
                                   sizeof(ctx->err));
        }
        if (!rc) {
            Phase ph(ctx, JLC_PHASE_OZAKI_GEMM);
            nl += 1;
            rc = launch_ozaki_gemm(g, pl, 0, ws, wsb, ctx->stream, ctx->sm_count, ctx->d_status, ctx->d_flags,
                                   ctx->err, sizeof(ctx->err));
        }
        if (!rc && pl.hi > 0) {
            {
                Phase ph(ctx, JLC_PHASE_OZAKI_SPLIT_HI);
                rc = launch_ozaki_split(g, pl, 1, ws, wsb, ctx->stream, ctx->sm_count, ctx->d_flags, ctx->err,
                                        sizeof(ctx->err), &nl);
            }
            if (!rc) {
                Phase ph(ctx, JLC_PHASE_OZAKI_GEMM_HI);
                nl += 1;
                rc = launch_ozaki_gemm(g, pl, 1, ws, wsb, ctx->stream, ctx->sm_count, ctx->d_status, ctx->d_flags,
                                       ctx->err, sizeof(ctx->err));
            }
        }
        ctx->launches += nl;
        if (rc) return rc;
        ctx->cert_rec = reinterpret_cast<CertRecord*>(static_cast<char*>(ws) +
                                                      ozaki_cert_offset(whole_m, g.n, g.k, pl));
        ctx->cert_plan = pl;
        ctx->cert_pending = true;
        if (rep) {
            // a-priori figures; replaced by the certificate's when the caller reads it
            rep->precision = crt ? JLC_PREC_OZAKI_CRT : JLC_PREC_OZAKI;
            rep->kernel = JLC_KERNEL_OZAKI;
            rep->slices = pl.lo;
            rep->products = crt ? pl.lo : pl.lo * (pl.lo + 1) / 2;
            const double u = std::ldexp(1.0, -53);
            rep->est_err_ratio = crt ? ozaki_crt_est_ratio(pl.lo, g.k)
                                     : (pl.lo + 3) * std::ldexp(1.0, -7 * pl.lo) / (2.0 * u * (double)g.k / 16.0);
        }
    }
    // the DMMA kernel reads A/B through TMA: 16-byte aligned bases, even lds
    RepackDesc packs[2];
    int np = 0;
    auto repack = [&](DevBuf& buf, const double*& x, long long& ld, long long rows, long long cols, const char* what) {
        if (dmma_operand_ok(x, ld)) return (int)JLC_OK;
        RepackDesc d{x, ld, nullptr, round_up(cols, 8), rows, cols};
        const int r = reserve(ctx, buf, (size_t)(rows * d.ld_dst) * 8, what);
        if (r) return r;
        d.dst = static_cast<double*>(buf.ptr);
        packs[np++] = d;
        x = d.dst;
        ld = d.ld_dst;
        return (int)JLC_OK;
    };
    const bool a_row = g.layout_a == JLC_ROW_MAJOR, b_row = g.layout_b == JLC_ROW_MAJOR;
    if ((rc = repack(ctx->bufA, g.a, g.lda, a_row ? g.m : g.k, a_row ? g.k : g.m, "repack A"))) return rc;
    if ((rc = repack(ctx->bufB, g.b, g.ldb, b_row ? g.k : g.n, b_row ? g.n : g.k, "repack B"))) return rc;
    if (np > 0) {
        rc = launch_repack(packs[0], packs[1], ozaki ? ctx->d_flags : nullptr, ctx->stream);
        if (rc) return set_err(ctx, rc, "repack launch failed");
        ctx->launches += 1;
    }
    if (!ozaki && rep) rep->kernel = JLC_KERNEL_DMMA;
    if (!ozaki && fault_hit(ctx, JLC_FAULT_WAIT)) g.withhold_stage = true;
    if (!ozaki && splitk_bytes > 0) {
        // Without room for the partials -- a capture cannot allocate -- the product runs unsplit.
        const bool grow = splitk_bytes > ctx->ws.bytes;
        if ((grow && capturing(ctx)) || ws_reserve(ctx, splitk_bytes) != JLC_OK) {
            ctx->err[0] = 0;
            ksplit = 1;
            splitk_bytes = 0;
        }
    }
    // After an Ozaki launch the FP64 kernel is gated on the split's
    // non-finite flag: it only runs when Inf/NaN made slicing impossible.
    Phase ph(ctx, ozaki ? JLC_PHASE_FP64_GATED : JLC_PHASE_DMMA);
    ctx->launches += 1;
    return launch_dgemm_dmma(g, ctx->stream, ctx->sm_count, ctx->d_status, ozaki ? ctx->d_flags : nullptr,
                             ctx->dmma_k, ctx->err, sizeof(ctx->err), ksplit,
                             splitk_bytes ? static_cast<char*>(ctx->ws.ptr) + splitk_off : nullptr, splitk_bytes,
                             splitk_bytes ? split_counters(ctx) : SplitCounters{});
}

int finish_sync(jlc_ctx* ctx) {
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_err(ctx, e, "stream synchronize");
    int st = 0;
    e = cudaMemcpy(&st, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_err(ctx, e, "status read");
    if (st != 0) {
        // (on the context's stream, which the legacy stream is not ordered with)
        e = cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_err(ctx, e, "status reset");
        if (st & JLC_DEV_TIMEOUT) return set_err(ctx, JLC_E_TIMEOUT, "a device wait timed out (status 0x%x)", st);
        return set_err(ctx, JLC_E_CUDA, "device status 0x%x", st);
    }
    return JLC_OK;
}

// Fills rep from the certificate record of the Ozaki call just enqueued
// (waits for the device).  Not while the stream is being captured: the
// a-priori figures stay.
int read_cert(jlc_ctx* ctx, jlc_report* rep) {
    if (!ctx->cert_pending) return JLC_OK;
    ctx->cert_pending = false;
    if (!rep) return JLC_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return JLC_OK;
    CertRecord r;
    cudaError_t e = cudaMemcpyAsync(&r, ctx->cert_rec, sizeof(r), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_err(ctx, e, "certificate read");
    const OzakiPlan& pl = ctx->cert_plan;
    auto as_double = [](unsigned long long b) {
        double d;
        memcpy(&d, &b, 8);
        return d;
    };
    if (r.blocks == 0 || r.fb_blocks == r.blocks) {
        // Inf/NaN operands (no certificate) or every block certified only in FP64
        rep->precision = JLC_PREC_NATIVE;
        rep->kernel = JLC_KERNEL_DMMA;
        rep->slices = 0;
        rep->products = 0;
        rep->est_err_ratio = r.blocks == 0 ? 0.0 : as_double(r.fb_est_bits);
        return JLC_OK;
    }
    const int used = r.hi_blocks > 0 ? pl.hi : pl.lo;
    rep->precision = pl.crt ? JLC_PREC_OZAKI_CRT : JLC_PREC_OZAKI;
    rep->kernel = JLC_KERNEL_OZAKI;
    rep->slices = used;
    rep->products = pl.crt ? used : used * (used + 1) / 2;
    rep->est_err_ratio = as_double(r.oz_est_bits);
    return JLC_OK;
}

// Host entry: stage op(A), op(B) (and C when beta != 0) into context buffers
// with 16-byte-aligned, padded leading dimensions, run, copy C back into the
// caller's m x n window only.
// Smallest row block of the host-entry pipeline: below two of these (or for a
// matrix-vector shape) the copies and the GEMM run back to back.
constexpr long long kPipeBlockRows = 512;

int pipe_ready(jlc_ctx* ctx) {
    if (!ctx->cin && cudaStreamCreateWithFlags(&ctx->cin, cudaStreamNonBlocking) != cudaSuccess)
        return cuda_err(ctx, cudaGetLastError(), "copy stream");
    if (!ctx->cout && cudaStreamCreateWithFlags(&ctx->cout, cudaStreamNonBlocking) != cudaSuccess)
        return cuda_err(ctx, cudaGetLastError(), "copy stream");
    for (cudaEvent_t& ev : ctx->pev)
        if (!ev && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)
            return cuda_err(ctx, cudaGetLastError(), "pipeline event");
    return JLC_OK;
}

// Host entry in row blocks of C: B (whole) and then the rows of op(A) (and of
// C when beta != 0) of each block go to the device on a copy-in stream, each
// block's GEMM runs on the context stream as soon as its rows have arrived,
// and its rows of C return on a copy-out stream while later blocks compute.
// PCIe is full duplex, so the time approaches the larger of the two copy
// directions plus one block.  Every block computes exactly what the
// single-shot path computes for its rows (same kernels, per-row and
// per-column Ozaki scaling, same k order), so results are bitwise identical.
// The Ozaki split of B is made once, by the first block, and reused.
int run_host_pipelined(jlc_ctx* ctx, int la, int lb, long long m, long long n, long long k, double alpha,
                       const double* a, long long lda, const double* b, long long ldb, double beta, double* c,
                       long long ldc, int precision, jlc_report* rep, long long dlda, long long dldb, long long dldc,
                       int64_t& h2d, int64_t& d2h) {
    int rc = pipe_ready(ctx);
    if (rc) return rc;
    // pageable operands go through the context's pinned chunks (staging.cu)
    const bool pa = host_pageable(a), pb = host_pageable(b), pc = host_pageable(c);
    if ((pa || pb || pc) && !ctx->stager) ctx->stager = stager_create();  // null: the driver stages instead
    auto h2d_copy = [&](bool pageable, void* dst, long long dp, const void* src, long long sp, long long w,
                        long long h) {
        return pageable ? staged_h2d(ctx, dst, (size_t)dp, src, (size_t)sp, (size_t)w, (size_t)h, ctx->cin)
                        : copy2d(ctx, dst, (size_t)dp, src, (size_t)sp, (size_t)w, (size_t)h, cudaMemcpyHostToDevice,
                                 ctx->cin);
    };
    const int maxb = jlc_ctx::kPipeMaxBlocks;
    long long rb = round_up((m + maxb - 1) / maxb, 128);
    if (rb < kPipeBlockRows) rb = kPipeBlockRows;
    const int nb = (int)((m + rb - 1) / rb);
    const long long b_rows = lb == JLC_ROW_MAJOR ? k : n, b_cols = lb == JLC_ROW_MAJOR ? n : k;
    cudaStream_t cs = ctx->stream, ci = ctx->cin, co = ctx->cout;
    auto drain = [&] {
        cudaStreamSynchronize(ci);
        cudaStreamSynchronize(cs);
        cudaStreamSynchronize(co);
        stager_abort(ctx);
    };
    cudaError_t e = cudaEventRecord(ctx->ev0, cs);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ci, ctx->ev0, 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(co, ctx->ev0, 0);
    if (e != cudaSuccess) return cuda_err(ctx, e, "pipeline start");
    {
        Phase ph(ctx, JLC_PHASE_H2D, ci);
        e = h2d_copy(pb, ctx->bufB.ptr, dldb * 8, b, ldb * 8, b_cols * 8, b_rows);
    }
    if (e != cudaSuccess) {
        drain();
        return cuda_err(ctx, e, "copy B to device");
    }
    h2d += b_rows * b_cols * 8;
    double* dA = static_cast<double*>(ctx->bufA.ptr);
    double* dC = static_cast<double*>(ctx->bufC.ptr);
    auto block_rows = [&](int i, long long& r0, long long& mr) {
        r0 = (long long)i * rb;
        mr = (m - r0 < rb) ? m - r0 : rb;
    };
    // Every block's inputs and GEMM are enqueued before any block's rows of C
    // are: a call that fails while enqueueing leaves the caller's C as it was.
    // (Enqueueing takes microseconds; block 0's GEMM is still running when its
    // copy-out is queued, so the overlap is unchanged.)
    for (int i = 0; i < nb; ++i) {
        long long r0, mr;
        block_rows(i, r0, mr);
        const double* blk_a;
        {
            Phase ph(ctx, JLC_PHASE_H2D, ci);
            if (la == JLC_ROW_MAJOR) {
                e = h2d_copy(pa, dA + r0 * dlda, dlda * 8, a + r0 * lda, lda * 8, k * 8, mr);
                blk_a = dA + r0 * dlda;
            } else {
                e = h2d_copy(pa, dA + r0, dlda * 8, a + r0, lda * 8, mr * 8, k);
                blk_a = dA + r0;
            }
            if (e == cudaSuccess && beta != 0.0)
                e = h2d_copy(pc, dC + r0 * dldc, dldc * 8, c + r0 * ldc, ldc * 8, n * 8, mr);
        }
        if (e == cudaSuccess) e = cudaEventRecord(ctx->pev[i], ci);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(cs, ctx->pev[i], 0);
        if (e != cudaSuccess) {
            drain();
            return cuda_err(ctx, e, "copy A block to device");
        }
        h2d += mr * k * 8 + (beta != 0.0 ? mr * n * 8 : 0);
        GemmDesc g{la, lb, mr, n, k, alpha, beta, blk_a, dlda, (const double*)ctx->bufB.ptr, dldb, dC + r0 * dldc,
                   dldc};
        g.ws_m = m;
        g.b_split_ready = i > 0;
        rc = run_device(ctx, g, precision, 0, rep);
        if (rc) {
            drain();
            return rc;
        }
        e = cudaEventRecord(ctx->pev[maxb + i], cs);
        if (e != cudaSuccess) {
            drain();
            return cuda_err(ctx, e, "pipeline event");
        }
    }
    for (int i = 0; i < nb; ++i) {
        long long r0, mr;
        block_rows(i, r0, mr);
        e = cudaStreamWaitEvent(co, ctx->pev[maxb + i], 0);
        if (e == cudaSuccess) {
            Phase ph(ctx, JLC_PHASE_D2H, co);
            e = pc ? staged_d2h(ctx, c + r0 * ldc, ldc * 8, dC + r0 * dldc, dldc * 8, n * 8, mr, co)
                   : copy2d(ctx, c + r0 * ldc, ldc * 8, dC + r0 * dldc, dldc * 8, n * 8, mr, cudaMemcpyDeviceToHost,
                            co);
        }
        if (e != cudaSuccess) {
            drain();
            return cuda_err(ctx, e, "copy C block to host");
        }
        d2h += mr * n * 8;
    }
    if (pc) {
        e = stager_flush(ctx);  // the host copies of the last chunks of C
        if (e != cudaSuccess) {
            drain();
            return cuda_err(ctx, e, "copy C to host");
        }
    }
    e = cudaEventRecord(ctx->pev[2 * maxb], co);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(cs, ctx->pev[2 * maxb], 0);
    if (e != cudaSuccess) {
        drain();
        return cuda_err(ctx, e, "pipeline end");
    }
    return JLC_OK;
}

int run_host(jlc_ctx* ctx, int la, int lb, long long m, long long n, long long k, double alpha, const double* a,
             long long lda, const double* b, long long ldb, double beta, double* c, long long ldc, int precision,
             jlc_report* rep) {
    report_init(rep);
    int rc = validate(ctx, la, lb, m, n, k, a, lda, b, ldb, c, ldc);
    if (rc) return rc;
    if (m == 0 || n == 0) return JLC_OK;
    ctx->err[0] = 0;
    cudaError_t e;
    const bool need_ab = alpha != 0.0 && k > 0;
    const long long a_rows = la == JLC_ROW_MAJOR ? m : k, a_cols = la == JLC_ROW_MAJOR ? k : m;
    const long long b_rows = lb == JLC_ROW_MAJOR ? k : n, b_cols = lb == JLC_ROW_MAJOR ? n : k;
    const long long dlda = round_up(a_cols, 8), dldb = round_up(b_cols, 8), dldc = round_up(n, 8);
    int64_t h2d = 0, d2h = 0;
    if (need_ab) {
        if ((rc = reserve(ctx, ctx->bufA, (size_t)(a_rows * dlda) * 8, "device A"))) return rc;
        if ((rc = reserve(ctx, ctx->bufB, (size_t)(b_rows * dldb) * 8, "device B"))) return rc;
    }
    if ((rc = reserve(ctx, ctx->bufC, (size_t)(m * dldc) * 8, "device C"))) return rc;
    if (need_ab && n > 1 && m >= 2 * kPipeBlockRows) {
        rc = run_host_pipelined(ctx, la, lb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, precision, rep, dlda,
                                dldb, dldc, h2d, d2h);
        if (rc) return rc;
        cudaEventRecord(ctx->ev1, ctx->stream);
        rc = finish_sync(ctx);
        if (!rc) rc = read_cert(ctx, rep);
        if (rc) return rc;
        if (rep) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
            rep->device_ms = ms;
            rep->h2d_bytes = h2d;
            rep->d2h_bytes = d2h;
        }
        return JLC_OK;
    }
    cudaEventRecord(ctx->ev0, ctx->stream);
    {
    Phase ph(ctx, JLC_PHASE_H2D);
    if (need_ab) {
        e = copy2d(ctx, ctx->bufA.ptr, dlda * 8, a, lda * 8, a_cols * 8, a_rows, cudaMemcpyHostToDevice,
                              ctx->stream);
        if (e != cudaSuccess) return copy_failed(ctx, e, "copy A to device");
        e = copy2d(ctx, ctx->bufB.ptr, dldb * 8, b, ldb * 8, b_cols * 8, b_rows, cudaMemcpyHostToDevice,
                              ctx->stream);
        if (e != cudaSuccess) return copy_failed(ctx, e, "copy B to device");
        h2d += (a_rows * a_cols + b_rows * b_cols) * 8;
    }
    if (beta != 0.0) {
        e = copy2d(ctx, ctx->bufC.ptr, dldc * 8, c, ldc * 8, n * 8, m, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) return copy_failed(ctx, e, "copy C to device");
        h2d += m * n * 8;
    }
    }
    GemmDesc g{la, lb, m, n, k, alpha, beta, (const double*)ctx->bufA.ptr, dlda, (const double*)ctx->bufB.ptr,
               dldb, (double*)ctx->bufC.ptr, dldc};
    rc = run_device(ctx, g, precision, 0, rep);
    if (rc) {
        cudaStreamSynchronize(ctx->stream);
        return rc;
    }
    {
        Phase ph(ctx, JLC_PHASE_D2H);
        e = copy2d(ctx, c, ldc * 8, ctx->bufC.ptr, dldc * 8, n * 8, m, cudaMemcpyDeviceToHost, ctx->stream);
    }
    if (e != cudaSuccess) return copy_failed(ctx, e, "copy C to host");
    d2h += m * n * 8;
    cudaEventRecord(ctx->ev1, ctx->stream);
    rc = finish_sync(ctx);
    if (!rc) rc = read_cert(ctx, rep);
    if (rc) return rc;
    if (rep) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        rep->device_ms = ms;
        rep->h2d_bytes = h2d;
        rep->d2h_bytes = d2h;
    }
    return JLC_OK;
}

}  // namespace

namespace jlc {

int workspace_reserve(Workspace& w, size_t bytes, char* err, size_t errlen) {
    if (bytes <= w.bytes) return JLC_OK;
    if (w.ptr) cudaFree(w.ptr);
    w.ptr = nullptr;
    w.bytes = 0;
    cudaError_t e = cudaMalloc(&w.ptr, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        w.ptr = nullptr;
        snprintf(err, errlen, "workspace allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
        return JLC_E_OOM;
    }
    w.bytes = bytes;
    return JLC_OK;
}

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

int make_tmap_2d(CUtensorMap* map, CUtensorMapDataType dt, int elem_bytes, void* base, uint64_t inner,
                 uint64_t outer, uint64_t ld_elems, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle sw,
                 char* err, size_t errlen) {
    auto fn = encode_fn();
    if (!fn) {
        snprintf(err, errlen, "cuTensorMapEncodeTiled unavailable");
        return JLC_E_CUDA;
    }
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {ld_elems * (uint64_t)elem_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(err, errlen, "cuTensorMapEncodeTiled(2d) failed (%d): dims %llu x %llu ld %llu box %u x %u",
                 (int)r, (unsigned long long)inner, (unsigned long long)outer, (unsigned long long)ld_elems,
                 box_inner, box_outer);
        return JLC_E_CUDA;
    }
    return JLC_OK;
}

int make_tmap_3d(CUtensorMap* map, CUtensorMapDataType dt, int elem_bytes, void* base, uint64_t d0, uint64_t d1,
                 uint64_t d2, uint64_t stride1_elems, uint64_t stride2_elems, uint32_t b0, uint32_t b1, uint32_t b2,
                 CUtensorMapSwizzle sw, char* err, size_t errlen) {
    auto fn = encode_fn();
    if (!fn) {
        snprintf(err, errlen, "cuTensorMapEncodeTiled unavailable");
        return JLC_E_CUDA;
    }
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {stride1_elems * (uint64_t)elem_bytes, stride2_elems * (uint64_t)elem_bytes};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, dt, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(err, errlen, "cuTensorMapEncodeTiled(3d) failed (%d)", (int)r);
        return JLC_E_CUDA;
    }
    return JLC_OK;
}

}  // namespace jlc

// ======================================================================== C ABI
namespace {

constexpr int kQrPanel = 64;  // panel width (HouseholderQR.java BLOCK_SIZE)

struct QrWork {
    double *v, *vt, *t, *w;
    long long ldv, ldw;
    int batch;            // panels whose V, T and V op(T) fit
    void* panel_scratch;  // multi-CTA panel: partials, row records, barrier counter
    double* gram;         // row-slab partials of V^T V (tall panels)
};

// Workspace for an m-row factor applied to `cols` columns, with V, T and V op(T)
// of up to `panels` panels at a time, within 256 MB (one panel at least, and no
// more than the device has room for).
int qr_work(jlc_ctx* ctx, long long m, long long cols, long long panels, QrWork& q) {
    q.ldv = round_up(m > 0 ? m : 1, 8);
    q.ldw = round_up(cols > 0 ? cols : 1, 8);
    const long long per = 2 * q.ldv * kQrPanel + kQrPanel * kQrPanel;  // doubles per panel
    const long long most = (256LL << 20) / (per * (long long)sizeof(double));
    q.batch = (int)(panels < 1 ? 1 : (most < 1 ? 1 : (panels < most ? panels : most)));
    const size_t scratch = round_up(qr_panel_mp_scratch_bytes(ctx->sm_count > 0 ? ctx->sm_count : 1), 256);
    const size_t gram = qr_gram_scratch_bytes(ctx->sm_count);
    for (int rc;; q.batch = (q.batch + 1) / 2) {
        const size_t doubles = (size_t)(per * q.batch + kQrPanel * q.ldw);
        rc = reserve(ctx, ctx->bufQ, doubles * sizeof(double) + scratch + gram, "QR workspace");
        if (rc == JLC_OK) break;
        if (rc != JLC_E_OOM || q.batch == 1) return rc;
    }
    ctx->err[0] = 0;
    if (ctx->qr_cluster_max == 0) ctx->qr_cluster_max = qr_panel_cluster_max();
    q.v = static_cast<double*>(ctx->bufQ.ptr);
    q.vt = q.v + q.ldv * kQrPanel * q.batch;
    q.t = q.vt + q.ldv * kQrPanel * q.batch;
    q.w = q.t + kQrPanel * kQrPanel * q.batch;
    q.panel_scratch = q.w + kQrPanel * q.ldw;
    q.gram = reinterpret_cast<double*>(static_cast<char*>(q.panel_scratch) + scratch);
    return JLC_OK;
}

// V, T and V op(T) of panels p0 .. p0 + panels - 1 of the factor f (m rows, kmax
// reflectors, reflector k's unit entry in row k + shift).
int qr_panels_vt(jlc_ctx* ctx, const double* f, long long ldf, long long m, long long kmax, long long p0, int panels,
                 int shift, const double* tau, bool trans, const QrWork& q) {
    Phase ph(ctx, JLC_PHASE_QR_VT);
    int nl = 0;
    const int rc = launch_qr_vt(f, ldf, (int)m, (int)kmax, (int)p0, panels, shift, tau, q.v, q.ldv, q.t, q.vt, trans,
                                q.gram, ctx->qr_cluster_max, ctx->sm_count, ctx->stream, &nl);
    ctx->launches += nl;
    return rc ? set_err(ctx, rc, "QR: V / T launch failed") : JLC_OK;
}

// C (rows k0.. of a column-major m x cols block, ld ldc) <- H C with H = I - V T
// V^T, or H^T C, by the i-th panel of the workspace, whose vt is V T or V T^T:
// W = V^T C, C -= (V op(T)) W, the latter as C^T -= W^T (V op(T))^T so that the
// column-major C is the GEMM's row-major output.
int qr_apply_wy(jlc_ctx* ctx, long long m, long long k0, long long cols, double* c, long long ldc, const QrWork& q,
                int i, int precision) {
    if (cols <= 0) return JLC_OK;
    const long long rows = m - k0;
    const double* v = q.v + i * q.ldv * kQrPanel + k0;
    const double* vt = q.vt + i * q.ldv * kQrPanel + k0;
    GemmDesc w{JLC_ROW_MAJOR, JLC_COL_MAJOR, kQrPanel, cols, rows, 1.0, 0.0, v, q.ldv, c + k0, ldc, q.w, q.ldw};
    w.chained = true;
    int rc = run_device(ctx, w, precision, 0, nullptr);
    if (rc) return rc;
    GemmDesc u{JLC_COL_MAJOR, JLC_ROW_MAJOR, cols, rows, kQrPanel, -1.0, 1.0, q.w, q.ldw, vt, q.ldv, c + k0, ldc};
    u.chained = true;
    return run_device(ctx, u, precision, 0, nullptr);
}

}  // namespace

extern "C" {

int jlc_version(void) { return JLCGPU_VERSION; }

int jlc_device_count(int* count) {
    if (!count) return JLC_E_ARG;
    *count = 0;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return JLC_OK;
    }
    int usable = 0;
    for (int d = 0; d < n; ++d) {
        int major = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, d) == cudaSuccess && major == 10)
            ++usable;
    }
    *count = usable;
    return JLC_OK;
}

int jlc_init(int device, jlc_ctx** out) {
    if (!out) return JLC_E_ARG;
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
        cudaGetLastError();
        return JLC_E_NODEV;
    }
    int major = 0, minor = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device);
    if (major != 10 || minor != 0) return JLC_E_NODEV;  // sm_100a code only
    if (cudaSetDevice(device) != cudaSuccess) return JLC_E_NODEV;
    jlc_ctx* ctx = new (std::nothrow) jlc_ctx();
    if (!ctx) return JLC_E_OOM;
    ctx->device = device;
    cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (const char* e = getenv("JLCGPU_DMMA_K")) {
        int v = atoi(e);
        if (v == 4 || v == 8 || v == 16) ctx->dmma_k = v;
    }
    bool ok = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&ctx->d_status, 4 * sizeof(int)) == cudaSuccess &&
              cudaMalloc(&ctx->d_flags, 4 * sizeof(int)) == cudaSuccess &&
              cudaMalloc(&ctx->d_counters, kSplitTiles * sizeof(*ctx->d_counters)) == cudaSuccess &&
              cudaEventCreate(&ctx->ev0) == cudaSuccess && cudaEventCreate(&ctx->ev1) == cudaSuccess;
    if (ok) ok = cudaMemsetAsync(ctx->d_status, 0, 4 * sizeof(int), ctx->own_stream) == cudaSuccess &&
                 cudaMemsetAsync(ctx->d_flags, 0, 4 * sizeof(int), ctx->own_stream) == cudaSuccess &&
                 cudaMemsetAsync(ctx->d_counters, 0, kSplitTiles * sizeof(*ctx->d_counters), ctx->own_stream) ==
                     cudaSuccess &&
                 cudaStreamSynchronize(ctx->own_stream) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        jlc_destroy(ctx);
        return JLC_E_CUDA;
    }
    ctx->stream = ctx->own_stream;
    // JLCGPU_FAULT=alloc|launch|copy|wait[:after] arms the failure test hook
    if (const char* f = getenv("JLCGPU_FAULT")) {
        static const char* names[] = {"none", "alloc", "launch", "copy", "wait"};
        for (int kind = 1; kind <= 4; ++kind) {
            const size_t len = strlen(names[kind]);
            if (strncmp(f, names[kind], len) == 0 && (f[len] == 0 || f[len] == ':')) {
                ctx->fault_kind = kind;
                ctx->fault_after = f[len] == ':' ? atoi(f + len + 1) : 0;
            }
        }
    }
    *out = ctx;
    return JLC_OK;
}

int jlc_set_wait_limit(jlc_ctx* ctx, double seconds) {
    if (!ctx) return JLC_E_ARG;
    if (!(seconds >= 0.0) || seconds > 600.0) return set_err(ctx, JLC_E_ARG, "wait limit must be in [0, 600] s");
    cudaSetDevice(ctx->device);
    const unsigned long long ns = (unsigned long long)(seconds * 1e9);
    // the limit sits beside the status bits (byte 8 of the status block)
    cudaError_t e = cudaMemcpyAsync(ctx->d_status + 2, &ns, sizeof(ns), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e == cudaSuccess ? JLC_OK : cuda_err(ctx, e, "wait limit");
}

int jlc_splitk_choice(jlc_ctx* ctx, int64_t m, int64_t n, int64_t k, int* split) {
    if (!ctx || !split || m < 1 || n < 1 || k < 1) return set_err(ctx, JLC_E_ARG, "splitk_choice: bad arguments");
    *split = dmma_splitk(m, n, k, ctx->sm_count, ctx->dmma_k);
    return JLC_OK;
}

int jlc_autotune_splitk(jlc_ctx* ctx, int64_t m, int64_t n, int64_t k, int* split) {
    if (!ctx || !split || m < 2 || n < 2 || k < 1 || m > (1 << 20) || n > (1 << 20) || k > (1 << 20))
        return set_err(ctx, JLC_E_ARG, "autotune_splitk: bad arguments");
    cudaSetDevice(ctx->device);
    const long long lda = round_up(k, 8), ldb = round_up(n, 8), ldc = n;
    int rc = reserve(ctx, ctx->bufA, (size_t)(m * lda) * 8, "autotune A");
    if (!rc) rc = reserve(ctx, ctx->bufB, (size_t)(k * ldb) * 8, "autotune B");
    if (!rc) rc = reserve(ctx, ctx->bufC, (size_t)(m * ldc) * 8, "autotune C");
    if (rc) return rc;
    // the kernel's time does not depend on the values: zeros will do
    cudaMemsetAsync(ctx->bufA.ptr, 0, (size_t)(m * lda) * 8, ctx->stream);
    cudaMemsetAsync(ctx->bufB.ptr, 0, (size_t)(k * ldb) * 8, ctx->stream);
    GemmDesc g{JLC_ROW_MAJOR, JLC_ROW_MAJOR, m, n, k, 1.0, 0.0, (const double*)ctx->bufA.ptr, lda,
               (const double*)ctx->bufB.ptr, ldb, (double*)ctx->bufC.ptr, ldc};
    int best = 1;
    float best_ms = 0.f;
    for (int s = 1; s <= 8; ++s) {
        if (!dmma_splitk_legal(m, n, k, s, ctx->sm_count)) continue;
        const size_t wsb = dmma_splitk_bytes(m, m, n, k, s, ctx->sm_count, ctx->dmma_k);
        if (wsb && (rc = ws_reserve(ctx, wsb))) return rc;
        float ms_min = 0.f;
        for (int rep = 0; rep < 4; ++rep) {  // one warm-up, three timed
            cudaEventRecord(ctx->ev0, ctx->stream);
            rc = launch_dgemm_dmma(g, ctx->stream, ctx->sm_count, ctx->d_status, nullptr, ctx->dmma_k, ctx->err,
                                   sizeof(ctx->err), s, wsb ? ctx->ws.ptr : nullptr, wsb,
                                   wsb ? split_counters(ctx) : SplitCounters{});
            if (rc) return rc;
            cudaEventRecord(ctx->ev1, ctx->stream);
            cudaError_t e = cudaEventSynchronize(ctx->ev1);
            if (e != cudaSuccess) return cuda_err(ctx, e, "autotune");
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
            if (rep == 1 || (rep > 1 && ms < ms_min)) ms_min = ms;
        }
        ctx->launches += 4;
        if (s == 1 || ms_min < best_ms) {
            best = s;
            best_ms = ms_min;
        }
    }
    rc = finish_sync(ctx);
    if (rc) return rc;
    const std::string cls = dmma_splitk_class(ctx->sm_count, m, n, k, ctx->dmma_k);
    grp::tune_store(cls, best);
    dmma_splitk_remember(cls, best);
    *split = best;
    return JLC_OK;
}

int jlc_inject_fault(jlc_ctx* ctx, int kind, int after) {
    if (!ctx) return JLC_E_ARG;
    if (kind < JLC_FAULT_NONE || kind > JLC_FAULT_WAIT || after < 0)
        return set_err(ctx, JLC_E_ARG, "fault kind must be JLC_FAULT_* and after >= 0");
    ctx->fault_kind = kind;
    ctx->fault_after = after;
    return JLC_OK;
}

void jlc_destroy(jlc_ctx* ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    if (ctx->stream) cudaStreamSynchronize(ctx->stream);
    if (ctx->bufA.ptr) cudaFree(ctx->bufA.ptr);
    if (ctx->bufH.ptr) cudaFree(ctx->bufH.ptr);
    if (ctx->bufB.ptr) cudaFree(ctx->bufB.ptr);
    if (ctx->bufC.ptr) cudaFree(ctx->bufC.ptr);
    if (ctx->bufR.ptr) cudaFree(ctx->bufR.ptr);
    if (ctx->bufQ.ptr) cudaFree(ctx->bufQ.ptr);
    if (ctx->ws.ptr) cudaFree(ctx->ws.ptr);
    if (ctx->d_status) cudaFree(ctx->d_status);
    if (ctx->d_flags) cudaFree(ctx->d_flags);
    if (ctx->d_counters) cudaFree(ctx->d_counters);
    stager_destroy(ctx->stager);
    for (int i = 0; i < 2 * jlc_ctx::kMaxRec; ++i)
        if (ctx->rec_ev[i]) cudaEventDestroy(ctx->rec_ev[i]);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    for (cudaEvent_t ev : ctx->pev)
        if (ev) cudaEventDestroy(ev);
    if (ctx->cin) cudaStreamDestroy(ctx->cin);
    if (ctx->cout) cudaStreamDestroy(ctx->cout);
    if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
    delete ctx;
}

const char* jlc_last_error(const jlc_ctx* ctx) { return ctx ? ctx->err : "null context"; }

int jlc_set_stream(jlc_ctx* ctx, void* cuda_stream) {
    if (!ctx) return JLC_E_ARG;
    ctx->stream = cuda_stream ? static_cast<cudaStream_t>(cuda_stream) : ctx->own_stream;
    return JLC_OK;
}

int jlc_synchronize(jlc_ctx* ctx) {
    if (!ctx) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    return finish_sync(ctx);
}

int jlc_device_status(jlc_ctx* ctx) { return jlc_synchronize(ctx); }

int jlc_host_register(jlc_ctx* ctx, void* ptr, size_t bytes) {
    if (!ctx || !ptr || bytes == 0) return set_err(ctx, JLC_E_ARG, "host_register: bad arguments");
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaHostRegister(ptr, bytes, cudaHostRegisterPortable);
    return e == cudaSuccess ? JLC_OK : cuda_err(ctx, e, "cudaHostRegister");
}

int jlc_host_unregister(jlc_ctx* ctx, void* ptr) {
    if (!ctx || !ptr) return set_err(ctx, JLC_E_ARG, "host_unregister: bad arguments");
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaHostUnregister(ptr);
    return e == cudaSuccess ? JLC_OK : cuda_err(ctx, e, "cudaHostUnregister");
}

int jlc_gemm(jlc_ctx* ctx, const double* a, const double* b, double* c, int64_t m, int64_t k, int64_t n,
             double alpha, double beta, int precision, jlc_report* rep) {
    if (!ctx) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    return run_host(ctx, JLC_ROW_MAJOR, JLC_ROW_MAJOR, m, n, k, alpha, a, k, b, n, beta, c, n, precision, rep);
}

int jlc_dgemm(jlc_ctx* ctx, int layout_a, int layout_b, int64_t m, int64_t n, int64_t k, double alpha,
              const double* a, int64_t lda, const double* b, int64_t ldb, double beta, double* c, int64_t ldc,
              int precision, jlc_report* rep) {
    if (!ctx) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    return run_host(ctx, layout_a, layout_b, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, precision, rep);
}

static int strided_entry(jlc_ctx* ctx, int la, int lb, const double* a, int64_t a_off, int64_t lda,
                         const double* b, int64_t b_off, int64_t ldb, double* c, int64_t c_off, int64_t ldc,
                         int64_t m, int64_t n, int64_t k, double alpha, double beta, int precision,
                         jlc_report* rep) {
    if (!ctx) return JLC_E_ARG;
    if (a_off < 0 || b_off < 0 || c_off < 0) return set_err(ctx, JLC_E_ARG, "offsets must be non-negative");
    cudaSetDevice(ctx->device);
    return run_host(ctx, la, lb, m, n, k, alpha, a ? a + a_off : nullptr, lda, b ? b + b_off : nullptr, ldb, beta,
                    c ? c + c_off : nullptr, ldc, precision, rep);
}

int jlc_gemm_strided(jlc_ctx* ctx, const double* a, int64_t a_off, int64_t lda, const double* b, int64_t b_off,
                     int64_t ldb, double* c, int64_t c_off, int64_t ldc, int64_t m, int64_t k, int64_t n,
                     double alpha, double beta, int precision, jlc_report* rep) {
    return strided_entry(ctx, JLC_ROW_MAJOR, JLC_ROW_MAJOR, a, a_off, lda, b, b_off, ldb, c, c_off, ldc, m, n, k,
                         alpha, beta, precision, rep);
}

int jlc_gemm_strided_transa(jlc_ctx* ctx, const double* a, int64_t a_off, int64_t lda, const double* b,
                            int64_t b_off, int64_t ldb, double* c, int64_t c_off, int64_t ldc, int64_t m,
                            int64_t k, int64_t n, double alpha, double beta, int precision, jlc_report* rep) {
    // output k x n, contraction over m: op(A)(i,p) = A(p,i) = a[p*lda + i] (column-major view)
    return strided_entry(ctx, JLC_COL_MAJOR, JLC_ROW_MAJOR, a, a_off, lda, b, b_off, ldb, c, c_off, ldc, k, n, m,
                         alpha, beta, precision, rep);
}

int jlc_gemm_strided_colmajor_a(jlc_ctx* ctx, const double* a, int64_t a_off, int64_t lda, const double* b,
                                int64_t b_off, int64_t ldb, double* c, int64_t c_off, int64_t ldc, int64_t m,
                                int64_t k, int64_t n, double alpha, double beta, int precision,
                                jlc_report* rep) {
    return strided_entry(ctx, JLC_COL_MAJOR, JLC_ROW_MAJOR, a, a_off, lda, b, b_off, ldb, c, c_off, ldc, m, n, k,
                         alpha, beta, precision, rep);
}

int jlc_gemm_strided_colmajor_b(jlc_ctx* ctx, const double* a, int64_t a_off, int64_t lda, const double* b,
                                int64_t b_off, int64_t ldb, double* c, int64_t c_off, int64_t ldc, int64_t m,
                                int64_t k, int64_t n, double alpha, double beta, int precision,
                                jlc_report* rep) {
    return strided_entry(ctx, JLC_ROW_MAJOR, JLC_COL_MAJOR, a, a_off, lda, b, b_off, ldb, c, c_off, ldc, m, n, k,
                         alpha, beta, precision, rep);
}

int jlc_dgemm_device(jlc_ctx* ctx, int layout_a, int layout_b, int64_t m, int64_t n, int64_t k, double alpha,
                     const double* a, int64_t lda, const double* b, int64_t ldb, double beta, double* c,
                     int64_t ldc, int precision, jlc_report* rep) {
    report_init(rep);
    int rc = validate(ctx, layout_a, layout_b, m, n, k, a, lda, b, ldb, c, ldc);
    if (rc) return rc;
    cudaSetDevice(ctx->device);
    GemmDesc g{layout_a, layout_b, m, n, k, alpha, beta, a, lda, b, ldb, c, ldc};
    rc = run_device(ctx, g, precision, 0, rep);
    return rc ? rc : read_cert(ctx, rep);
}

int jlc_dgemm_ozaki_crt_device(jlc_ctx* ctx, int layout_a, int layout_b, int64_t m, int64_t n, int64_t k,
                               double alpha, const double* a, int64_t lda, const double* b, int64_t ldb, double beta,
                               double* c, int64_t ldc, int moduli, jlc_report* rep) {
    report_init(rep);
    int rc = validate(ctx, layout_a, layout_b, m, n, k, a, lda, b, ldb, c, ldc);
    if (rc) return rc;
    if (moduli != 0 && (moduli < 2 || moduli > 15)) return set_err(ctx, JLC_E_ARG, "moduli must be 0 or in [2,15]");
    cudaSetDevice(ctx->device);
    GemmDesc g{layout_a, layout_b, m, n, k, alpha, beta, a, lda, b, ldb, c, ldc};
    rc = run_device(ctx, g, JLC_PREC_OZAKI_CRT, moduli, rep);
    return rc ? rc : read_cert(ctx, rep);
}

int jlc_dgemm_ozaki_device(jlc_ctx* ctx, int layout_a, int layout_b, int64_t m, int64_t n, int64_t k,
                           double alpha, const double* a, int64_t lda, const double* b, int64_t ldb, double beta,
                           double* c, int64_t ldc, int slices, jlc_report* rep) {
    report_init(rep);
    int rc = validate(ctx, layout_a, layout_b, m, n, k, a, lda, b, ldb, c, ldc);
    if (rc) return rc;
    if (slices != 0 && (slices < 3 || slices > 8)) return set_err(ctx, JLC_E_ARG, "slices must be 0 or in [3,8]");
    cudaSetDevice(ctx->device);
    GemmDesc g{layout_a, layout_b, m, n, k, alpha, beta, a, lda, b, ldb, c, ldc};
    rc = run_device(ctx, g, JLC_PREC_OZAKI, slices, rep);
    return rc ? rc : read_cert(ctx, rep);
}

int jlc_set_profiling(jlc_ctx* ctx, int on) {
    if (!ctx) return JLC_E_ARG;
    ctx->profiling = on != 0;
    return JLC_OK;
}

int jlc_profile_collect(jlc_ctx* ctx, int* phases, double* ms, int max) {
    if (!ctx || max < 0 || (max > 0 && (!phases || !ms))) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_err(ctx, e, "profile synchronize");
    const int n = ctx->nrec < max ? ctx->nrec : max;
    for (int i = 0; i < n; ++i) {
        float t = 0.f;
        e = cudaEventElapsedTime(&t, ctx->rec_ev[2 * i], ctx->rec_ev[2 * i + 1]);
        if (e != cudaSuccess) return cuda_err(ctx, e, "profile event");
        phases[i] = ctx->rec_phase[i];
        ms[i] = t;
    }
    ctx->nrec = 0;
    return n;
}

int jlc_profile_timeline(jlc_ctx* ctx, int* phases, double* start_ms, double* end_ms, int max) {
    if (!ctx || max < 0 || (max > 0 && (!phases || !start_ms || !end_ms))) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    cudaError_t e = cudaDeviceSynchronize();  // records may sit on the copy streams
    if (e != cudaSuccess) return cuda_err(ctx, e, "profile synchronize");
    const int n = ctx->nrec < max ? ctx->nrec : max;
    for (int i = 0; i < n; ++i) {
        float t0 = 0.f, t1 = 0.f;
        e = cudaEventElapsedTime(&t0, ctx->rec_ev[0], ctx->rec_ev[2 * i]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t1, ctx->rec_ev[0], ctx->rec_ev[2 * i + 1]);
        if (e != cudaSuccess) return cuda_err(ctx, e, "profile event");
        phases[i] = ctx->rec_phase[i];
        start_ms[i] = t0;
        end_ms[i] = t1;
    }
    ctx->nrec = 0;
    return n;
}

int jlc_check_fp64_bound_device(jlc_ctx* ctx, int layout_a, int layout_b, int64_t m, int64_t n, int64_t k,
                                double alpha, const double* a, int64_t lda, const double* b, int64_t ldb,
                                double beta, const double* c_in, int64_t ldc_in, const double* c_out,
                                int64_t ldc_out, int64_t count, const int64_t* rows, const int64_t* cols,
                                double* max_ratio, double* max_abs, int64_t* over) {
    int rc = validate(ctx, layout_a, layout_b, m, n, k, a, lda, b, ldb, c_out, ldc_out);
    if (rc) return rc;
    if (count < 0 || (count > 0 && (!rows || !cols)) || !max_ratio || !max_abs || !over)
        return set_err(ctx, JLC_E_ARG, "check: bad sample arguments");
    if (beta != 0.0 && (!c_in || ldc_in < n)) return set_err(ctx, JLC_E_ARG, "check: beta != 0 needs C_in");
    for (int64_t e = 0; e < count; ++e)
        if (rows[e] < 0 || rows[e] >= m || cols[e] < 0 || cols[e] >= n)
            return set_err(ctx, JLC_E_ARG, "check: sample entry %lld out of range", (long long)e);
    cudaSetDevice(ctx->device);
    const size_t bytes = (size_t)count * 16 + 64;
    DevBuf tmp;
    if ((rc = reserve(ctx, tmp, bytes, "check buffers"))) return rc;
    auto* d_rows = static_cast<long long*>(tmp.ptr);
    auto* d_cols = d_rows + count;
    auto* d_out = reinterpret_cast<unsigned long long*>(d_cols + count);
    cudaError_t e = cudaMemcpyAsync(d_rows, rows, count * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_cols, cols, count * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_out, 0, 24, ctx->stream);
    if (e != cudaSuccess) {
        cudaFree(tmp.ptr);
        return cuda_err(ctx, e, "check setup");
    }
    GemmDesc g{layout_a, layout_b, m, n, k, alpha, beta, a, lda, b, ldb, nullptr, 0};
    rc = check_fp64_bound(g, c_in, ldc_in, c_out, ldc_out, count, d_rows, d_cols, d_out, ctx->stream);
    unsigned long long h[3] = {0, 0, 0};
    if (!rc) e = cudaMemcpyAsync(h, d_out, 24, cudaMemcpyDeviceToHost, ctx->stream);
    if (!rc && e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(tmp.ptr);
    if (rc) return set_err(ctx, rc, "check kernel launch failed");
    if (e != cudaSuccess) return cuda_err(ctx, e, "check");
    double r, ab;
    memcpy(&r, &h[0], 8);
    memcpy(&ab, &h[1], 8);
    *max_ratio = r;
    *max_abs = ab;
    *over = (int64_t)h[2];
    return JLC_OK;
}

int jlc_qr_factor_device(jlc_ctx* ctx, int64_t m, int64_t n, double* a, int64_t lda, double* tau, int precision,
                         jlc_report* rep) {
    report_init(rep);
    if (!ctx) return JLC_E_ARG;
    if (m < 0 || n < 0) return set_err(ctx, JLC_E_ARG, "dimensions must be non-negative");
    if (m == 0 || n == 0) return JLC_OK;
    if (!a || !tau || lda < m) return set_err(ctx, JLC_E_ARG, "A and tau must not be null and lda must be >= m");
    if (m > INT32_MAX / 2 || n > INT32_MAX / 2) return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^30");
    cudaSetDevice(ctx->device);
    ctx->err[0] = 0;
    QrWork q;
    int rc = qr_work(ctx, m, n, 1, q);
    if (rc) return rc;
    cudaEventRecord(ctx->ev0, ctx->stream);
    const long long kmax = m < n ? m : n;
    for (long long k0 = 0; k0 < kmax; k0 += kQrPanel) {
        const int kb = (int)(kmax - k0 < kQrPanel ? kmax - k0 : kQrPanel);
        {
            // one cluster of CTAs of >= 64 rows each while the rows fit its
            // registers or shared memory, else up to one CTA per SM, of >= 128
            // rows each, in one cooperative launch
            Phase ph(ctx, JLC_PHASE_QR_PANEL);
            ctx->launches += 1;
            long long ctas = (m - k0) / 128;
            if (ctas > ctx->sm_count) ctas = ctx->sm_count;
            if (ctas < 1) ctas = 1;
            const bool withhold =
                qr_panel_waits((int)m, (int)k0, ctx->qr_cluster_max) && fault_hit(ctx, JLC_FAULT_WAIT);
            rc = launch_qr_panel(a, lda, (int)m, (int)k0, kb, tau, (int)ctas, ctx->qr_cluster_max, q.panel_scratch,
                                 ctx->d_status, withhold, ctx->stream);
            if (rc) return set_err(ctx, rc, "QR: panel launch failed");
        }
        const long long trail = n - (k0 + kb);
        if (trail <= 0) continue;
        rc = qr_panels_vt(ctx, a, lda, m, kmax, k0 / kQrPanel, 1, 0, tau, true, q);
        if (!rc) rc = qr_apply_wy(ctx, m, k0, trail, a + (k0 + kb) * lda, lda, q, 0, precision);
        if (rc) return rc;
    }
    cudaEventRecord(ctx->ev1, ctx->stream);
    rc = finish_sync(ctx);
    if (rc) return rc;
    if (rep) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        rep->device_ms = ms;
        rep->kernel = JLC_KERNEL_DMMA;
    }
    return JLC_OK;
}

// The block reflector of one Hessenberg panel applied as the reference does
// (BlockedHessenbergQR.applyBlockLeft / applyBlockRight, :277-345), on
// column-major matrices.  Left, rows r0.. and columns c0.. of h:
// W = V^T C, W2 = T^T W, C -= V W2 (the last as C^T -= W2^T V^T).  Right,
// columns r0.. (all rows) of mat: W = B V, W2 = W T, B -= W2 V^T (as
// B^T -= V W2^T).
constexpr int kHessPanel = 32;

int hess_apply_left(jlc_ctx* ctx, double* h, long long ldh, long long n, long long k, int pw, const double* V,
                    long long ldv, const double* T, double* W, double* W2, long long ldw, int precision) {
    const long long m = n - k - 1, cols = n - k;
    double* c = h + (k + 1) + k * ldh;
    GemmDesc w{JLC_ROW_MAJOR, JLC_COL_MAJOR, pw, cols, m, 1.0, 0.0, V, ldv, c, ldh, W, ldw};
    int rc = run_device(ctx, w, precision, 0, nullptr);
    if (rc) return rc;
    GemmDesc t{JLC_COL_MAJOR, JLC_ROW_MAJOR, pw, cols, pw, 1.0, 0.0, T, kHessPanel, W, ldw, W2, ldw};
    rc = run_device(ctx, t, JLC_PREC_NATIVE, 0, nullptr);
    if (rc) return rc;
    GemmDesc u{JLC_COL_MAJOR, JLC_ROW_MAJOR, cols, m, pw, -1.0, 1.0, W2, ldw, V, ldv, c, ldh};
    return run_device(ctx, u, precision, 0, nullptr);
}

int hess_apply_right(jlc_ctx* ctx, double* mat, long long ldm, long long n, long long k, int pw, const double* V,
                     long long ldv, const double* T, double* W, double* W2, int precision) {
    // W = X V and W2 = W T are formed transposed, W^T = V^T X^T (pw x n) and
    // W2^T = T^T W^T, so that their GEMMs have pw rows (thin tiles) rather
    // than pw columns; W and W2 hold them row-major with leading dimension ldv
    const long long m = n - k - 1;
    double* b = mat + (k + 1) * ldm;
    GemmDesc w{JLC_ROW_MAJOR, JLC_ROW_MAJOR, pw, n, m, 1.0, 0.0, V, ldv, b, ldm, W, ldv};
    int rc = run_device(ctx, w, precision, 0, nullptr);
    if (rc) return rc;
    GemmDesc t{JLC_COL_MAJOR, JLC_ROW_MAJOR, pw, n, pw, 1.0, 0.0, T, kHessPanel, W, ldv, W2, ldv};
    rc = run_device(ctx, t, JLC_PREC_NATIVE, 0, nullptr);
    if (rc) return rc;
    // X_sub^T (the column-major block read row-major) -= V W2^T
    GemmDesc u{JLC_COL_MAJOR, JLC_ROW_MAJOR, m, n, pw, -1.0, 1.0, V, ldv, W2, ldv, b, ldm};
    return run_device(ctx, u, precision, 0, nullptr);
}

}  // extern "C"

namespace {
// Q (first qcols columns) of kmax reflectors stored in f (QR style; reflector
// k's unit entry, implied, in row k + shift and its tail below) with scales tau,
// enqueued on the context stream without a sync: the identity, then the panels'
// block reflectors in reverse order.  The panels' V and T do not depend on one
// another: a batch of panels forms them in two launches.
int qr_build_q_enqueue(jlc_ctx* ctx, long long m, long long kmax, long long qcols, const double* f, long long ldf,
                       int shift, const double* tau, double* q_out, long long ldq, int precision) {
    const long long live = kmax < qcols ? kmax : qcols;  // a panel past the last column has nothing to change
    const long long panels = (live + kQrPanel - 1) / kQrPanel;
    QrWork q;
    int rc = qr_work(ctx, m, qcols, panels, q);
    if (rc) return rc;
    rc = launch_set_identity(q_out, ldq, m, qcols, ctx->stream);
    if (rc) return set_err(ctx, rc, "QR: identity launch failed");
    for (long long last = panels; last > 0;) {
        const int nb = (int)(last < q.batch ? last : q.batch);
        const long long first = last - nb;
        rc = qr_panels_vt(ctx, f, ldf, m, kmax, first, nb, shift, tau, false, q);
        for (int i = nb - 1; i >= 0 && !rc; --i) {
            // (the columns of Q up to k0 + shift are the identity's and have no entry in these rows)
            const long long k0 = (first + i) * kQrPanel, c0 = k0 + shift;
            rc = qr_apply_wy(ctx, m, k0, qcols - c0, q_out + c0 * ldq, ldq, q, i, precision);
        }
        if (rc) return rc;
        last = first;
    }
    return JLC_OK;
}
}  // namespace

extern "C" {

int jlc_hessenberg_device(jlc_ctx* ctx, int64_t n, double* a, int64_t lda, double* q, int64_t ldq, int precision,
                          jlc_report* rep) {
    report_init(rep);
    if (!ctx) return JLC_E_ARG;
    if (n < 0) return set_err(ctx, JLC_E_ARG, "dimension must be non-negative");
    if (n == 0) return JLC_OK;
    if (!a || lda < n) return set_err(ctx, JLC_E_ARG, "A must not be null and lda must be >= n");
    if (q && ldq < n) return set_err(ctx, JLC_E_ARG, "ldq must be >= n");
    if (n > INT32_MAX / 4) return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^29");
    cudaSetDevice(ctx->device);
    ctx->err[0] = 0;
    cudaStream_t st = ctx->stream;
    cudaEventRecord(ctx->ev0, st);
    int rc = JLC_OK;
    const bool slab = n > 2 && hess_slab_fits((int)n, ctx->sm_count);
    // (the Q builder behind the one-launch reduction starts from an identity of its own)
    if (q && !slab && (rc = launch_set_identity(q, ldq, n, n, st)))
        return set_err(ctx, rc, "Hessenberg: identity launch failed");
    if (slab) {
        // the whole reduction in one launch, then Q from the reflectors below the subdiagonal
        const long long ldt = round_up(n, 8);
        if ((rc = reserve(ctx, ctx->bufH, (ldt + hess_slab_work_doubles((int)n, ctx->sm_count)) * sizeof(double),
                          "Hessenberg workspace")))
            return rc;
        double* tau = static_cast<double*>(ctx->bufH.ptr);
        {
            Phase ph(ctx, JLC_PHASE_HESS_PANEL);
            rc = launch_hess_slab(a, lda, (int)n, tau, tau + ldt, ctx->sm_count, ctx->d_status,
                                  fault_hit(ctx, JLC_FAULT_WAIT), st);
            if (rc) return set_err(ctx, rc, "Hessenberg: launch failed");
            ctx->launches += 1;
        }
        if (q && (rc = qr_build_q_enqueue(ctx, n, n - 2, n, a, lda, 1, tau, q, ldq, precision))) return rc;
        if ((rc = launch_hess_clear(a, lda, (int)n, st))) return set_err(ctx, rc, "Hessenberg: clear launch failed");
        ctx->launches += 1;
    } else if (n > 2) {
        const long long ldv = round_up(n, 8), ldw = ldv;
        const size_t work_bytes = hess_work_doubles(n) * sizeof(double);
        if ((rc = reserve(ctx, ctx->bufH, work_bytes + hess_panel_scratch_bytes(ctx->sm_count),
                          "Hessenberg workspace")))
            return rc;
        double* V = static_cast<double*>(ctx->bufH.ptr);
        double* Y = V + ldv * kHessPanel;
        double* W = Y + ldv * kHessPanel;
        double* W2 = W + ldv * kHessPanel;
        double* T = W2 + ldv * kHessPanel;
        double* tau = T + kHessPanel * kHessPanel;
        double* wbuf = tau + 2 * kHessPanel;
        void* panel_scratch = static_cast<char*>(ctx->bufH.ptr) + work_bytes;
        for (long long k = 0; k < n - 2; k += kHessPanel) {
            const int pw = (int)((n - 2 - k) < kHessPanel ? (n - 2 - k) : kHessPanel);
            {
                // the panel's reflectors, V, T and Y in one cooperative launch
                Phase ph(ctx, JLC_PHASE_HESS_PANEL);
                if (cudaMemsetAsync(T, 0, kHessPanel * kHessPanel * sizeof(double), st) != cudaSuccess)
                    return set_err(ctx, JLC_E_CUDA, "Hessenberg: T reset failed");
                rc = launch_hess_panel(a, lda, (int)n, (int)k, pw, V, ldv, Y, T, tau, wbuf, panel_scratch,
                                       ctx->sm_count, ctx->d_status, st);
                if (rc) return set_err(ctx, rc, "Hessenberg: panel launch failed");
                ctx->launches += 1;
            }
            rc = hess_apply_left(ctx, a, lda, n, k, pw, V, ldv, T, W, W2, ldw, precision);
            if (!rc) rc = hess_apply_right(ctx, a, lda, n, k, pw, V, ldv, T, W, W2, precision);
            if (!rc && q) rc = hess_apply_right(ctx, q, ldq, n, k, pw, V, ldv, T, W, W2, precision);
            if (rc) return rc;
        }
        if ((rc = launch_hess_clear(a, lda, (int)n, st))) return set_err(ctx, rc, "Hessenberg: clear launch failed");
        ctx->launches += 1;
    }
    cudaEventRecord(ctx->ev1, st);
    rc = finish_sync(ctx);
    if (rc) return rc;
    if (rep) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        rep->device_ms = ms;
        rep->kernel = JLC_KERNEL_DMMA;
    }
    return JLC_OK;
}

int jlc_qr_build_q_device(jlc_ctx* ctx, int64_t m, int64_t n, int64_t qcols, const double* f, int64_t ldf,
                          const double* tau, double* q_out, int64_t ldq, int precision, jlc_report* rep) {
    report_init(rep);
    if (!ctx) return JLC_E_ARG;
    if (m < 0 || n < 0 || qcols < 0 || qcols > m) return set_err(ctx, JLC_E_ARG, "need 0 <= qcols <= m");
    if (m == 0 || qcols == 0) return JLC_OK;
    if (!q_out || ldq < m) return set_err(ctx, JLC_E_ARG, "Q must not be null and ldq must be >= m");
    const long long kmax = m < n ? m : n;
    if (kmax > 0 && (!f || !tau || ldf < m)) return set_err(ctx, JLC_E_ARG, "F and tau must not be null, ldf >= m");
    if (m > INT32_MAX / 2 || n > INT32_MAX / 2) return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^30");
    cudaSetDevice(ctx->device);
    ctx->err[0] = 0;
    cudaEventRecord(ctx->ev0, ctx->stream);
    int rc = qr_build_q_enqueue(ctx, m, kmax, qcols, f, ldf, 0, tau, q_out, ldq, precision);
    if (rc) return rc;
    cudaEventRecord(ctx->ev1, ctx->stream);
    rc = finish_sync(ctx);
    if (rc) return rc;
    if (rep) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        rep->device_ms = ms;
        rep->kernel = JLC_KERNEL_DMMA;
    }
    return JLC_OK;
}

int jlc_bidiag_device(jlc_ctx* ctx, int64_t m, int64_t n, double* a, int64_t lda, double* d, double* e, double* u,
                      int64_t ldu, double* v, int64_t ldv, int precision, jlc_report* rep) {
    report_init(rep);
    if (!ctx) return JLC_E_ARG;
    if (m < 0 || n < 0) return set_err(ctx, JLC_E_ARG, "dimensions must be non-negative");
    if (n > m) return set_err(ctx, JLC_E_ARG, "need m >= n (a wide matrix is reduced through its transpose)");
    if (m > 0 && n > 0 && (!a || lda < m)) return set_err(ctx, JLC_E_ARG, "A must not be null and lda must be >= m");
    if (n > 0 && (!d || (n > 1 && !e))) return set_err(ctx, JLC_E_ARG, "d and e must not be null");
    if (u && ldu < m) return set_err(ctx, JLC_E_ARG, "ldu must be >= m");
    if (v && ldv < n) return set_err(ctx, JLC_E_ARG, "ldv must be >= n");
    if (m > INT32_MAX / 4) return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^29");
    cudaSetDevice(ctx->device);
    ctx->err[0] = 0;
    cudaStream_t st = ctx->stream;
    int rows_per_cta = 0;
    if (m > 0 && n > 0 && bidiag_grid((int)m, (int)n, ctx->sm_count, &rows_per_cta) == 0)
        return set_err(ctx, JLC_E_UNSUPPORTED, "bidiagonalisation: more than 256 rows per SM");
    cudaEventRecord(ctx->ev0, st);
    int rc = JLC_OK;
    if (m > 0 && n > 0) {
        // workspace: tau of the column and row reflectors, the kernel's slots,
        // and a region for its copy of the rows (past shared memory), which the
        // row reflectors rearranged as a QR factor take over.  Without room for
        // the copy the reduction runs in place.
        const long long ldw = round_up(n, 8);
        const long long ldt = round_up(n, 8);
        size_t sdoubles = 0;
        const size_t kdoubles = bidiag_work_doubles((int)m, (int)n, ctx->sm_count, &sdoubles);
        const size_t wdoubles = v ? (size_t)ldw * (size_t)n : 0, base = 2 * (size_t)ldt + kdoubles;
        bool in_place = false;
        rc = reserve(ctx, ctx->bufH, (base + (sdoubles > wdoubles ? sdoubles : wdoubles)) * sizeof(double),
                     "bidiagonalisation workspace");
        if (rc == JLC_E_OOM && sdoubles > 0) {
            in_place = true;
            rc = reserve(ctx, ctx->bufH, (base + wdoubles) * sizeof(double), "bidiagonalisation workspace");
        }
        if (rc) return rc;
        ctx->err[0] = 0;
        double* tauq = static_cast<double*>(ctx->bufH.ptr);
        double* taup = tauq + ldt;
        double* kwork = taup + ldt;
        double* wr = kwork + kdoubles;
        {
            Phase ph(ctx, JLC_PHASE_BIDIAG);
            rc = launch_bidiag(a, lda, (int)m, (int)n, d, e, tauq, taup, kwork, in_place, ctx->sm_count, ctx->d_status,
                               fault_hit(ctx, JLC_FAULT_WAIT), st);
            if (rc) return set_err(ctx, rc, "bidiagonalisation: launch failed");
            ctx->launches += 1;
        }
        // U = H_0 H_1 ... H_{n-1}: the column reflectors sit below the diagonal as in a QR factor
        if (u && (rc = qr_build_q_enqueue(ctx, m, n, m, a, lda, 0, tauq, u, ldu, precision))) return rc;
        if (v) {
            // V = G_0 ... G_{n-2}: row k's reflector acts on columns k+1..
            if (n > 1) {
                if ((rc = launch_bidiag_right_factor(a, lda, (int)n, wr, ldw, st)))
                    return set_err(ctx, rc, "bidiagonalisation: right factor launch failed");
                if ((rc = qr_build_q_enqueue(ctx, n, n - 1, n, wr, ldw, 1, taup, v, ldv, precision))) return rc;
            } else if ((rc = launch_set_identity(v, ldv, n, n, st))) {
                return set_err(ctx, rc, "identity launch failed");
            }
        }
    } else {
        if (u && (rc = launch_set_identity(u, ldu, m, m, st))) return set_err(ctx, rc, "identity launch failed");
        if (v && (rc = launch_set_identity(v, ldv, n, n, st))) return set_err(ctx, rc, "identity launch failed");
    }
    cudaEventRecord(ctx->ev1, st);
    rc = finish_sync(ctx);
    if (rc) return rc;
    if (rep) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        rep->device_ms = ms;
        rep->kernel = JLC_KERNEL_DMMA;
    }
    return JLC_OK;
}

int jlc_dgemm_adjoint_device(jlc_ctx* ctx, int64_t m, int64_t n, int64_t k, double alpha, double beta,
                             const double* a, int64_t lda, const double* b, int64_t ldb, const double* c_in,
                             int64_t ldc_in, const double* dc, int64_t lddc, double* da, int64_t ldda, double* db,
                             int64_t lddb, double* dalpha, double* dbeta, double* dc_in, int64_t lddc_in,
                             int precision, jlc_report* rep) {
    report_init(rep);
    if (!ctx) return JLC_E_ARG;
    if (m < 0 || n < 0 || k < 0) return set_err(ctx, JLC_E_ARG, "dimensions must be non-negative");
    if (!dalpha || !dbeta) return set_err(ctx, JLC_E_ARG, "dalpha and dbeta must not be null");
    if (m > 0 && n > 0 && (!dc || lddc < n || !c_in || ldc_in < n))
        return set_err(ctx, JLC_E_ARG, "dC and C_in must not be null and their ld must be >= n");
    if (m > 0 && k > 0 && (!a || lda < k || !da || ldda < k))
        return set_err(ctx, JLC_E_ARG, "A and dA must not be null and their ld must be >= k");
    if (k > 0 && n > 0 && (!b || ldb < n || !db || lddb < n))
        return set_err(ctx, JLC_E_ARG, "B and dB must not be null and their ld must be >= n");
    if (dc_in && lddc_in < n) return set_err(ctx, JLC_E_ARG, "lddc_in must be >= n");
    if (m > INT32_MAX / 2 || n > INT32_MAX / 2 || k > INT32_MAX / 2)
        return set_err(ctx, JLC_E_UNSUPPORTED, "dimension above 2^30");
    cudaSetDevice(ctx->device);
    ctx->err[0] = 0;
    cudaStream_t st = ctx->stream;
    const int np = ctx->sm_count > 0 ? ctx->sm_count : 1;  // the GEMM kernels never launch more CTAs
    int rc = reserve(ctx, ctx->bufR, (size_t)(4 * np) * sizeof(double), "reduction partials");
    if (rc) return rc;
    double* parts_a = static_cast<double*>(ctx->bufR.ptr);
    double* parts_b = parts_a + 2 * np;
    jlc_report sub;

    // 1) G = dC * B^T (m x k, contraction n): dA = alpha * G, dalpha = <A, G>
    if (m > 0 && k > 0 && n > 0) {
        GemmDesc g{JLC_ROW_MAJOR, JLC_COL_MAJOR, m, k, n, 1.0, 0.0, dc, lddc, b, ldb, da, ldda};
        const bool gemv_shape = (k == 1 || m == 1);
        if (!gemv_shape) {
            // fused: the GEMM epilogue scales and reduces; partials of a kernel
            // that did not run (the gated FP64 twin of an Ozaki call) stay 0
            if (cudaMemsetAsync(parts_a, 0, np * sizeof(double), st) != cudaSuccess)
                return set_err(ctx, JLC_E_CUDA, "partials reset failed");
            g.epi_scale = alpha;
            g.dot_mat = a;
            g.dot_ld = lda;
            g.dot_partials = parts_a;
            rc = run_device(ctx, g, precision, 0, &sub);
            if (!rc) {
                Phase ph(ctx, JLC_PHASE_REDUCE);
                rc = launch_sum(parts_a, np, dalpha, st);
            }
        } else {
            rc = run_device(ctx, g, precision, 0, &sub);
            Phase ph(ctx, JLC_PHASE_REDUCE);
            if (!rc)
                rc = launch_dot2d(da, ldda, a, lda, m, k, parts_a, 2 * np, dalpha, alpha != 1.0 ? da : nullptr, ldda,
                                  alpha, st);
        }
        if (rc) return rc;
    } else {
        if (m > 0 && k > 0) {
            rc = launch_scale_c(da, ldda, m, k, 0.0, st);  // n == 0: dA = 0
            if (rc) return set_err(ctx, rc, "dA reset failed");
        }
        if (cudaMemsetAsync(dalpha, 0, sizeof(double), st) != cudaSuccess)
            return set_err(ctx, JLC_E_CUDA, "dalpha reset failed");
    }
    if (rep) *rep = sub;
    // 2) dB = alpha * A^T * dC (k x n, contraction m)
    if (k > 0 && n > 0) {
        GemmDesc g2{JLC_COL_MAJOR, JLC_ROW_MAJOR, k, n, m, alpha, 0.0, a, lda, dc, lddc, db, lddb};
        rc = run_device(ctx, g2, precision, 0, &sub);
        if (rc) return rc;
    }
    // 3) dbeta = <dC, C_in>;  4) dC_in = beta * dC
    {
        Phase ph(ctx, JLC_PHASE_REDUCE);
        rc = launch_dot2d(dc, lddc, c_in, ldc_in, m, n, parts_b, 2 * np, dbeta, dc_in, lddc_in, beta, st);
    }
    if (rc) return set_err(ctx, rc, "adjoint reduction launch failed");
    ctx->launches += 2;
    return JLC_OK;
}

int jlc_measure_peaks(jlc_ctx* ctx, double* out4) {
    if (!ctx || !out4) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    int rc = measure_peaks(ctx->sm_count, ctx->stream, ctx->d_status, out4, ctx->err, sizeof(ctx->err));
    if (rc) return rc;
    return finish_sync(ctx);
}

int jlc_measure_int8_sustained(jlc_ctx* ctx, double seconds, double* tops) {
    if (!ctx || !tops || !(seconds > 0.0) || seconds > 60.0) return JLC_E_ARG;
    cudaSetDevice(ctx->device);
    int rc = measure_int8_sustained(ctx->sm_count, ctx->stream, ctx->d_status, seconds, tops, ctx->err,
                                    sizeof(ctx->err));
    if (rc) return rc;
    return finish_sync(ctx);
}

int jlc_launch_count(jlc_ctx* ctx, int64_t* launches) {
    if (!ctx || !launches) return JLC_E_ARG;
    *launches = ctx->launches;
    return JLC_OK;
}

}  // extern "C"
