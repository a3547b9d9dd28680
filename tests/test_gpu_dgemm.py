"""GPU parity of the native FP64 route (DMMA tensor-core kernel and GEMV).

Cases follow the reference's own GEMM tests (GemmParityTest, GemmStridedParityTest,
GemmOffHeapParityTest, GemmNumericEdgeTest, GemmCudaParityTest), run through the
reference-shaped API (jlc_b200.compute -> C ABI).  Each result is held to
(a) the reference's CUDA tolerance against GemmReference (GemmReference.java:179-181)
and (b) the componentwise FP64 bound |C - C_dd| <= 2 k u (|alpha||A||B| + |beta||C|)
against the double-double oracle.
"""
import json
import os

import numpy as np
import pytest

from parity import assert_fp64_bound, assert_reference_parity

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
SHAPES = [(4, 4, 4), (12, 12, 12), (64, 64, 64), (128, 64, 16), (16, 64, 128), (96, 96, 1), (128, 3, 128)]
GRID = [0.0, 1.0, -0.5, 2.5]


def test_parity_grid_optimized_blas3(ctx, oracle):
    """GemmParityTest.gemmParityAgainstIndependentReference (GemmParityTest.java:38-72)."""
    from jlc_b200 import Matrix, OptimizedBLAS3, BLAS3Kernels
    seed = 20260603
    for (m, k, n) in SHAPES:
        a = Matrix.wrap(oracle.seeded_array(m * k, seed + 11), m, k)
        b = Matrix.wrap(oracle.seeded_array(k * n, seed + 29), k, n)
        c0 = oracle.seeded_array(m * n, seed + 47)
        for alpha in GRID:
            for beta in GRID:
                expected = oracle.gemm_reference(a.to_numpy(), b.to_numpy(), c0.reshape(m, n), alpha, beta)
                for api in (OptimizedBLAS3.gemm, BLAS3Kernels.gemm):
                    out = Matrix.wrap(c0.copy(), m, n)
                    api(a, b, out, alpha, beta)
                    label = f"{api.__qualname__} {m}x{k}x{n} a={alpha} b={beta}"
                    assert_reference_parity(label, expected, out.getRawData(), k)
                    assert_fp64_bound(label, out.to_numpy(), a.to_numpy(), b.to_numpy(), c0.reshape(m, n),
                                      alpha, beta)
        seed += 101


def test_known_answers(ctx):
    from jlc_b200 import CudaGemm, Matrix
    with open(os.path.join(GOLDEN, "reference_known_answers.json")) as f:
        cases = json.load(f)["cases"]
    for case in cases:
        if "expected" not in case:
            continue
        m, k, n = case["m"], case["k"], case["n"]
        a = Matrix.wrap(np.array([float(x) for x in case["a"]]), m, k)
        b = Matrix.wrap(np.array([float(x) for x in case["b"]]), k, n)
        c = Matrix.wrap(np.array([float(x) for x in case["c"]]), m, n)
        assert CudaGemm.gemm(a, b, c, case["alpha"], case["beta"]), CudaGemm.last_error
        exp = np.array([float(x) for x in case["expected"]])
        np.testing.assert_array_equal(np.isnan(c.getRawData()), np.isnan(exp), err_msg=case["name"])
        np.testing.assert_allclose(np.nan_to_num(c.getRawData()), np.nan_to_num(exp), atol=1e-12,
                                   err_msg=case["name"])


def test_cuda_parity_64(ctx, oracle):
    """GemmCudaParityTest (GemmCudaParityTest.java:8-26): 64^3, alpha=1, beta=-0.5, seeds 7001-7003."""
    from jlc_b200 import CudaGemm, Matrix
    a = Matrix.wrap(oracle.seeded_array(64 * 64, 7001), 64, 64)
    b = Matrix.wrap(oracle.seeded_array(64 * 64, 7002), 64, 64)
    c = oracle.seeded_array(64 * 64, 7003)
    expected = oracle.gemm_reference(a.to_numpy(), b.to_numpy(), c.reshape(64, 64), 1.0, -0.5)
    out = Matrix.wrap(c.copy(), 64, 64)
    assert CudaGemm.gemm(a, b, out, 1.0, -0.5)
    assert_reference_parity("CudaGemm.gemm", expected, out.getRawData(), 64)
    prod = CudaGemm.multiply(a, b)
    assert_fp64_bound("CudaGemm.multiply", prod.to_numpy(), a.to_numpy(), b.to_numpy(), None, 1.0, 0.0)


def test_strided_row_major(ctx, oracle):
    """GemmStridedParityTest.stridedRowMajorParity (GemmStridedParityTest.java:7-29)."""
    from jlc_b200 import BLAS3Kernels
    m, k, n, off = 9, 7, 11, 13
    lda, ldb, ldc = k + 5, n + 7, n + 3
    a = oracle.seeded_array(off + lda * m + 17, 4102)
    b = oracle.seeded_array(off + ldb * k + 17, 4103)
    c = oracle.seeded_array(off + ldc * m + 17, 4104)
    A = a[off:off + lda * m].reshape(m, lda)[:, :k]
    B = b[off:off + ldb * k].reshape(k, ldb)[:, :n]
    C = c[off:off + ldc * m].reshape(m, ldc)[:, :n].copy()
    expected = oracle.gemm_reference(A, B, C, 2.5, -0.5)
    before = c.copy()
    BLAS3Kernels.gemmStrided(a, off, lda, b, off, ldb, c, off, ldc, m, k, n, 2.5, -0.5, 19)
    got = c[off:off + ldc * m].reshape(m, ldc)[:, :n]
    assert_reference_parity("gemmStrided", expected, got, k)
    assert_fp64_bound("gemmStrided", np.ascontiguousarray(got), A, B, C, 2.5, -0.5)
    # guard band: nothing outside the m x n window changed
    inside = np.zeros(c.size, dtype=bool)
    for i in range(m):
        inside[off + i * ldc:off + i * ldc + n] = True
    np.testing.assert_array_equal(c[~inside], before[~inside])


def test_strided_transposed_a(ctx, oracle):
    """GemmStridedParityTest.stridedTransposedAParity (GemmStridedParityTest.java:31-54)."""
    from jlc_b200 import BLAS3Kernels
    m, k, n, off = 8, 5, 6, 13
    lda, ldb, ldc = k + 7, n + 5, n + 3
    a = oracle.seeded_array(off + lda * m + 9, 4202)
    b = oracle.seeded_array(off + ldb * m + 9, 4203)
    c = oracle.seeded_array(off + ldc * k + 9, 4204)
    A = a[off:off + lda * m].reshape(m, lda)[:, :k]
    B = b[off:off + ldb * m].reshape(m, ldb)[:, :n]
    C = c[off:off + ldc * k].reshape(k, ldc)[:, :n].copy()
    expected = oracle.gemm_reference(A.T, B, C, 1.0, 2.5)
    BLAS3Kernels.gemmStridedTransA(a, off, lda, b, off, ldb, c, off, ldc, m, k, n, 1.0, 2.5, 17)
    got = c[off:off + ldc * k].reshape(k, ldc)[:, :n]
    assert_reference_parity("gemmStridedTransA", expected, got, m)
    assert_fp64_bound("gemmStridedTransA", np.ascontiguousarray(got), A.T, B, C, 1.0, 2.5)


def test_strided_column_major_variants(ctx, oracle):
    """GemmStridedParityTest.stridedColumnMajorVariantsParity (GemmStridedParityTest.java:56-107)."""
    from jlc_b200 import BLAS3Kernels
    m, k, n = 10, 6, 7
    rldA, rldB, cldA, cldB, ldc, off = k + 4, n + 7, m + 5, k + 3, n + 5, 13
    A = oracle.seeded_array(m * k, 4302).reshape(m, k)
    B = oracle.seeded_array(k * n, 4303).reshape(k, n)
    cA = oracle.seeded_array(off + ldc * m + 9, 4304)
    cB = oracle.seeded_array(off + ldc * m + 9, 4305)
    a_col = np.zeros(k * cldA)
    a_col.reshape(k, cldA)[:, :m] = A.T
    b_col = np.zeros(n * cldB)
    b_col.reshape(n, cldB)[:, :k] = B.T
    b_rs = np.zeros(off + rldB * k + 9)
    b_rs[off:off + rldB * k].reshape(k, rldB)[:, :n] = B
    a_rs = np.zeros(off + rldA * m + 9)
    a_rs[off:off + rldA * m].reshape(m, rldA)[:, :k] = A

    CA = cA[off:off + ldc * m].reshape(m, ldc)[:, :n].copy()
    expA = oracle.gemm_reference(A, B, CA, -0.5, 1.0)
    BLAS3Kernels.gemmStridedColMajorA(a_col, 0, cldA, b_rs, off, rldB, cA, off, ldc, m, k, n, -0.5, 1.0, 15)
    gotA = cA[off:off + ldc * m].reshape(m, ldc)[:, :n]
    assert_reference_parity("gemmStridedColMajorA", expA, gotA, k)
    assert_fp64_bound("gemmStridedColMajorA", np.ascontiguousarray(gotA), A, B, CA, -0.5, 1.0)

    CB = cB[off:off + ldc * m].reshape(m, ldc)[:, :n].copy()
    expB = oracle.gemm_reference(A, B, CB, 2.5, 0.0)
    BLAS3Kernels.gemmStridedColMajorB(a_rs, off, rldA, b_col, 0, cldB, cB, off, ldc, m, k, n, 2.5, 0.0, 15)
    gotB = cB[off:off + ldc * m].reshape(m, ldc)[:, :n]
    assert_reference_parity("gemmStridedColMajorB", expB, gotB, k)
    assert_fp64_bound("gemmStridedColMajorB", np.ascontiguousarray(gotB), A, B, CB, 2.5, 0.0)


def test_optimized_strided(ctx, oracle):
    """GemmStridedParityTest.optimizedStridedParity (GemmStridedParityTest.java:109-130)."""
    from jlc_b200 import OptimizedBLAS3
    m, k, n, off = 13, 9, 8, 13
    lda, ldb, ldc = k + 7, n + 5, n + 1
    a = oracle.seeded_array(off + lda * m + 5, 4402)
    b = oracle.seeded_array(off + ldb * k + 5, 4403)
    c = oracle.seeded_array(off + ldc * m + 5, 4404)
    A = a[off:off + lda * m].reshape(m, lda)[:, :k]
    B = b[off:off + ldb * k].reshape(k, ldb)[:, :n]
    C = c[off:off + ldc * m].reshape(m, ldc)[:, :n].copy()
    expected = oracle.gemm_reference(A, B, C, 1.0, -0.5)
    OptimizedBLAS3.gemmStrided(a, off, lda, b, off, ldb, c, off, ldc, m, k, n, 1.0, -0.5)
    assert_reference_parity("OptimizedBLAS3.gemmStrided", expected, c[off:off + ldc * m].reshape(m, ldc)[:, :n], k)


def test_offheap_operands(ctx, oracle):
    """GemmOffHeapParityTest (GemmOffHeapParityTest.java:22-78), both storage orders."""
    from jlc_b200 import BLAS3Kernels, OffHeapMatrix, OptimizedBLAS3

    def fill(mat, seed):
        data = oracle.seeded_array(mat.rows * mat.cols, seed)
        for i in range(mat.rows):
            for j in range(mat.cols):
                mat.set(i, j, data[i * mat.cols + j])
        mat.syncToOffHeap()

    for order in (OffHeapMatrix.ROW_MAJOR, OffHeapMatrix.COL_MAJOR):
        a, b = OffHeapMatrix(24, 16, order=order), OffHeapMatrix(16, 10, order=order)
        fill(a, 5101)
        fill(b, 5102)
        prod = BLAS3Kernels.gemm(a, b)
        assert isinstance(prod, OffHeapMatrix)
        expected = oracle.gemm_reference(a.to_numpy(), b.to_numpy(), np.zeros((24, 10)), 1.0, 0.0)
        assert_reference_parity("BLAS3Kernels.gemm off-heap", expected, prod.getRawData(), 16)

        a, b, c = (OffHeapMatrix(18, 12, order=order, ld=15 if order == "ROW_MAJOR" else 21),
                   OffHeapMatrix(12, 14, order=order), OffHeapMatrix(18, 14))
        fill(a, 5201)
        fill(b, 5202)
        fill(c, 5203)
        expected = oracle.gemm_reference(a.to_numpy(), b.to_numpy(), c.to_numpy(), -0.5, 2.5)
        OptimizedBLAS3.gemm(a, b, c, -0.5, 2.5)
        assert_reference_parity("OptimizedBLAS3.gemm off-heap", expected, c.getRawData(), 12)
        for (i, j) in [(0, 0), (9, 7), (17, 13)]:
            assert abs(c.getOffHeap(i, j) - expected[i, j]) <= 1e-12


def test_numeric_edges(ctx):
    """GemmNumericEdgeTest semantics on the GPU route: beta == 0 does not read C,
    alpha == 0 does not read A/B, no zero-skip (0*Inf = NaN)."""
    from jlc_b200 import Matrix, OptimizedBLAS3
    a = Matrix.wrap(np.array([1.0, 2.0, 3.0, 4.0]), 2, 2)
    b = Matrix.wrap(np.array([5.0, 6.0, 7.0, 8.0]), 2, 2)
    c = Matrix.wrap(np.full(4, np.nan), 2, 2)
    OptimizedBLAS3.gemm(a, b, c, 1.0, 0.0)
    np.testing.assert_array_equal(c.getRawData(), [19.0, 22.0, 43.0, 50.0])
    c = Matrix.wrap(np.array([4.0]), 1, 1)
    OptimizedBLAS3.gemm(Matrix.wrap(np.array([np.nan]), 1, 1), Matrix.wrap(np.array([np.nan]), 1, 1), c, 0.0, -0.5)
    assert c.get(0, 0) == -2.0
    c = Matrix.wrap(np.array([7.0]), 1, 1)
    OptimizedBLAS3.gemm(Matrix.wrap(np.array([0.0]), 1, 1), Matrix.wrap(np.array([np.inf]), 1, 1), c, 1.0, 1.0)
    assert np.isnan(c.get(0, 0))
    # a larger tile with an Inf in B: only the products that touch it become non-finite
    A = np.ones((130, 70))
    B = np.ones((70, 90))
    B[3, 5] = np.inf
    C = np.zeros((130, 90))
    ctx.gemm(A, B, C, 1.0, 0.0)
    assert np.isinf(C[:, 5]).all() and np.isfinite(np.delete(C, 5, axis=1)).all()


def test_zero_and_degenerate_dimensions(ctx, oracle):
    """GemmParityTest.gemmSupportsZeroAndDegenerateDimensions (GemmParityTest.java:117-146)."""
    from jlc_b200 import BLAS3Kernels, Matrix, OptimizedBLAS3
    a, b, c = Matrix(0, 3), Matrix(3, 2), Matrix(0, 2)
    BLAS3Kernels.gemm(a, b, c, 1.0, 0.0)
    OptimizedBLAS3.gemm(a, b, c, 1.0, 0.0)
    assert c.getRawData().size == 0
    c0 = oracle.seeded_array(20, 901)
    for api in (BLAS3Kernels.gemm, OptimizedBLAS3.gemm):
        out = Matrix.wrap(c0.copy(), 5, 4)
        api(Matrix(5, 0), Matrix(0, 4), out, 2.5, -0.5)
        np.testing.assert_array_equal(out.getRawData(), c0 * -0.5)
    empty = BLAS3Kernels.gemm(Matrix(2, 0), Matrix(0, 0))
    assert empty.getRowCount() == 2 and empty.getColumnCount() == 0


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (7, 7, 7), (31, 33, 17), (33, 31, 129), (129, 127, 31),
                                   (128, 128, 16), (257, 129, 300), (1, 300, 65), (300, 1, 65), (2, 513, 3)])
def test_edge_tiles(ctx, oracle, m, n, k):
    a = oracle.uniform((m, k), m * 1000 + n)
    b = oracle.uniform((k, n), k * 1000 + m)
    c = oracle.uniform((m, n), 77)
    out = c.copy()
    ctx.gemm(a, b, out, -1.25, 0.75)
    assert_fp64_bound(f"edge {m}x{n}x{k}", out, a, b, c, -1.25, 0.75)


@pytest.mark.parametrize("la,lb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_layouts_host_and_device(ctx, oracle, la, lb):
    """All four operand orders, on host entries and on device entries whose
    operands are deliberately misaligned (odd offsets and odd leading
    dimensions force the repack path)."""
    import torch
    m, n, k = 300, 257, 129
    A = oracle.uniform((m, k), 31)
    B = oracle.uniform((k, n), 32)
    C = oracle.uniform((m, n), 33)
    a_store = A if la == 0 else np.ascontiguousarray(A.T)
    b_store = B if lb == 0 else np.ascontiguousarray(B.T)
    out = C.copy()
    ctx.dgemm(la, lb, m, n, k, 1.5, a_store, a_store.shape[1], b_store, b_store.shape[1], 0.5, out, n)
    assert_fp64_bound(f"host layouts {la}{lb}", out, A, B, C, 1.5, 0.5)

    def padded(x, pad_cols, off):
        buf = torch.zeros(off + x.shape[0] * (x.shape[1] + pad_cols), dtype=torch.float64, device="cuda")
        view = buf[off:].view(x.shape[0], x.shape[1] + pad_cols)
        view[:, :x.shape[1]] = torch.from_numpy(x).cuda()
        return buf, x.shape[1] + pad_cols, off

    abuf, lda, aoff = padded(a_store, 3, 1)   # odd ld, 8-byte (not 16-byte) aligned base
    bbuf, ldb, boff = padded(b_store, 2, 0)
    cdev = torch.from_numpy(C.copy()).cuda()
    rep = ctx.dgemm_device(la, lb, m, n, k, 1.5, abuf.data_ptr() + 8 * aoff, lda, bbuf.data_ptr() + 8 * boff, ldb,
                           0.5, cdev.data_ptr(), n)
    ctx.synchronize()
    assert rep["kernel"] == 1
    assert_fp64_bound(f"device layouts {la}{lb}", cdev.cpu().numpy(), A, B, C, 1.5, 0.5)


def test_config1_1024(ctx, oracle):
    """1024^3, alpha=1.5, beta=0.5, seed 20260604: sampled entries against the
    double-double oracle, the full matrix against the OptimizedBLAS3 order."""
    n = 1024
    A = oracle.uniform((n, n), 20260604 + 1)
    B = oracle.uniform((n, n), 20260604 + 2)
    C = oracle.uniform((n, n), 20260604 + 3)
    out = C.copy()
    rep = ctx.gemm(A, B, out, 1.5, 0.5)
    assert rep["kernel"] == 1 and rep["h2d_bytes"] == 3 * n * n * 8 and rep["d2h_bytes"] == n * n * 8
    rows, cols = oracle.sample_entries(n, n, 4096, 1)
    assert_fp64_bound("config1 sampled", out, A, B, C, 1.5, 0.5, rows=rows, cols=cols)
    fma = oracle.gemm_fmachain(A, B, C, 1.5, 0.5)
    bound = 2 * n * 2.0 ** -53 * (1.5 * (np.abs(A) @ np.abs(B)) + 0.5 * np.abs(C))
    assert np.all(np.abs(out - fma) <= 2 * bound)


@pytest.mark.parametrize("la", [0, 1])
def test_gemv_shapes(ctx, oracle, la):
    """n == 1 (MATVEC, SpecializedKernels.java:27-71) and m == 1."""
    for (m, n, k) in [(777, 1, 1531), (1, 913, 1029), (4096, 1, 4096)]:
        A = oracle.uniform((m, k), 1)
        B = oracle.uniform((k, n), 2)
        C = oracle.uniform((m, n), 3)
        a_store = A if la == 0 else np.ascontiguousarray(A.T)
        out = C.copy()
        rep = ctx.dgemm(la, 0, m, n, k, 0.75, a_store, a_store.shape[1], B, n, -1.5, out, n)
        assert rep["kernel"] == 2
        assert_fp64_bound(f"gemv {m}x{n}x{k} la={la}", out, A, B, C, 0.75, -1.5)


def test_device_entry_on_caller_stream(ctx, oracle):
    import torch
    m = n = k = 512
    A = torch.from_numpy(oracle.uniform((m, k), 5)).cuda()
    B = torch.from_numpy(oracle.uniform((k, n), 6)).cuda()
    C = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    try:
        ctx.dgemm_device(0, 0, m, n, k, 1.0, A.data_ptr(), k, B.data_ptr(), n, 0.0, C.data_ptr(), n)
        s.synchronize()
    finally:
        ctx.set_stream(None)
    assert_fp64_bound("caller stream", C.cpu().numpy(), A.cpu().numpy(), B.cpu().numpy(), None, 1.0, 0.0)


@pytest.mark.parametrize("m,n,k,alpha,beta", [
    (1024, 1024, 1024, 1.5, 0.5),   # 64 tiles: two k parts
    (300, 200, 3000, 1.0, 0.0),     # 6 tiles, ragged edges: eight k parts
    (512, 768, 2000, -0.75, 2.0),   # 24 tiles, parts of uneven length
    (128, 128, 4096, 1.0, -1.0),    # one tile
])
def test_split_k_small_products(ctx, oracle, m, n, k, alpha, beta):
    """Products with fewer tiles than half the SMs split k across CTAs; the
    last part to arrive sums the parts in index order: inside the FP64 bound,
    and bitwise the same on every run (and through the host entry)."""
    import torch
    A = oracle.uniform((m, k), 71)
    B = oracle.uniform((k, n), 72)
    C = oracle.uniform((m, n), 73)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    runs = []
    for _ in range(3):
        dC = torch.from_numpy(C.copy()).cuda()
        rep = ctx.dgemm_device(0, 0, m, n, k, alpha, dA.data_ptr(), k, dB.data_ptr(), n, beta, dC.data_ptr(), n,
                               precision=0)
        ctx.synchronize()
        assert rep["kernel"] == 1
        runs.append(dC.cpu().numpy())
    for r in runs[1:]:
        np.testing.assert_array_equal(r, runs[0])
    rows, cols = oracle.sample_entries(m, n, 2048, 5)
    assert_fp64_bound(f"split-K {m}x{n}x{k}", runs[0], A, B, C, alpha, beta, rows=rows, cols=cols)
    host = C.copy()
    ctx.dgemm(0, 0, m, n, k, alpha, A, k, B, n, beta, host, n, precision=0)
    np.testing.assert_array_equal(host, runs[0])


def test_splitk_autotune_caches_and_is_used(ctx, oracle, tmp_path, monkeypatch):
    """The split-K tuner (the per-shape-class counterpart of
    GemmDispatch.computeBlockSizes, GemmDispatch.java:118-149): it times the
    legal factors for a class, stores the fastest in the tuning cache, and
    products of that class use it from then on, inside the FP64 bound and
    bitwise repeatable."""
    import torch
    monkeypatch.setenv("JLCGPU_TUNE_CACHE", str(tmp_path / "tune.txt"))
    m, n, k = 640, 512, 2048  # 20 tiles: split-K matters
    s = ctx.autotune_splitk(m, n, k)
    assert 1 <= s <= 8
    text = (tmp_path / "tune.txt").read_text()
    assert "dmma-splitk|t20|kb7" in text and text.strip().endswith(str(s))
    assert ctx.splitk_choice(m, n, k) == s
    assert ctx.splitk_choice(m, n, k + 100) == s  # same class (k to a power of two)
    A = oracle.uniform((m, k), 1601)
    B = oracle.uniform((k, n), 1602)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    outs = []
    for _ in range(2):
        dC = torch.zeros((m, n), dtype=torch.float64, device="cuda")
        ctx.dgemm_device(0, 0, m, n, k, 1.0, dA.data_ptr(), k, dB.data_ptr(), n, 0.0, dC.data_ptr(), n)
        ctx.synchronize()
        outs.append(dC.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])
    assert_fp64_bound("tuned split-K", outs[0], A, B, None, 1.0, 0.0)


@pytest.mark.parametrize("m", [2, 20, 32, 33, 50, 64, 65])
@pytest.mark.parametrize("la,lb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_thin_tiles(ctx, oracle, m, la, lb):
    """Products of at most 64 rows run 32- or 64-row tiles (the panel GEMMs of
    the blocked factorisations): every operand order, rows on and just past
    the tile heights, beta != 0, and a k long enough for split-K.  Inside the
    FP64 bound, and the same bits on a second run."""
    import torch
    n, k = 1000, 3000
    A = oracle.uniform((m, k), 81 + m)
    B = oracle.uniform((k, n), 82)
    C = oracle.uniform((m, n), 83)
    a_store = A if la == 0 else np.ascontiguousarray(A.T)
    b_store = B if lb == 0 else np.ascontiguousarray(B.T)
    dA, dB = torch.from_numpy(a_store).cuda(), torch.from_numpy(b_store).cuda()
    runs = []
    for _ in range(2):
        dC = torch.from_numpy(C.copy()).cuda()
        rep = ctx.dgemm_device(la, lb, m, n, k, -0.5, dA.data_ptr(), a_store.shape[1], dB.data_ptr(),
                               b_store.shape[1], 1.25, dC.data_ptr(), n, precision=0)
        ctx.synchronize()
        assert rep["kernel"] == 1
        runs.append(dC.cpu().numpy())
    np.testing.assert_array_equal(runs[1], runs[0])
    assert_fp64_bound(f"thin {m} {la}{lb}", runs[0], A, B, C, -0.5, 1.25)


@pytest.mark.parametrize("la,lb", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k", [
    (31, 33, 17), (97, 79, 113),                  # 32 x 32 tiles, one k-block and a k tail
    (32, 9001, 20), (41, 2500, 100),              # 32 x 64, 64 x 32
    (700, 651, 200), (32, 4737, 33),              # 64 x 64, 32 x 128
    (999, 1100, 520), (64, 9473, 33),             # 128 x 64, 64 x 128
    (1501, 1500, 33),                             # 128 x 128
    (33, 65, 4100), (130, 257, 1537),             # split k on the smallest tiles
])
def test_tile_shapes(ctx, oracle, la, lb, m, n, k):
    """Products whose tile shapes differ, ragged at every edge, in all four
    layouts with padded leading dimensions, alpha and beta: inside the FP64
    bound, and the padding of C untouched."""
    import torch
    rng = np.random.default_rng(m * 7 + n)
    a, b, c = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n)), rng.uniform(-1, 1, (m, n))

    def stored(x, layout, pad):
        x = x if layout == 0 else x.T
        out = np.full((x.shape[0], (x.shape[1] + pad + 1) // 2 * 2), 7.5)
        out[:, :x.shape[1]] = x
        return torch.from_numpy(out).cuda()

    at, bt, ct = stored(a, la, 3), stored(b, lb, 5), stored(c, 0, 1)
    torch.cuda.synchronize()
    ctx.dgemm_device(la, lb, m, n, k, 1.5, at.data_ptr(), at.shape[1], bt.data_ptr(), bt.shape[1], -0.5,
                     ct.data_ptr(), ct.shape[1])
    ctx.synchronize()
    out = ct.cpu().numpy()
    assert (out[:, n:] == 7.5).all()
    rows = rng.integers(0, m, 400)
    cols = rng.integers(0, n, 400)
    rows[:4], cols[:4] = (0, 0, m - 1, m - 1), (0, n - 1, 0, n - 1)
    assert_fp64_bound(f"{m}x{n}x{k}", out[:, :n], a, b, c, 1.5, -0.5, rows=rows, cols=cols)


@pytest.mark.parametrize("m,n,k", [(3, 5, 2), (9, 513, 511), (600, 7, 8)])
def test_operands_copied_for_tma(ctx, oracle, m, n, k):
    """Odd leading dimensions and 8-byte aligned bases of either operand, at
    the edges of the copy's row and column blocks: bit for bit the product of
    aligned operands."""
    import torch
    rng = np.random.default_rng(m + n + k)
    a, b = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))
    outs = []
    for lda, ldb, off in ((k + k % 2, n + n % 2, 0), (k + 1 + k % 2, n + 1 + n % 2, 0), (k + k % 2, n + n % 2, 1)):
        bufs = []
        for x, ld in ((a, lda), (b, ldb)):
            flat = torch.full((off + x.shape[0] * ld,), 3.5, dtype=torch.float64)
            flat[off:].view(x.shape[0], ld)[:, :x.shape[1]] = torch.from_numpy(x)
            bufs.append(flat.cuda())
        c = torch.zeros(m, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.dgemm_device(0, 0, m, n, k, 1.0, bufs[0].data_ptr() + 8 * off, lda, bufs[1].data_ptr() + 8 * off, ldb, 0.0,
                         c.data_ptr(), n)
        ctx.synchronize()
        outs.append(c.cpu().numpy())
    assert_fp64_bound("aligned", outs[0], a, b, None, 1.0, 0.0)
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])


@pytest.mark.parametrize("la", [0, 1])
@pytest.mark.parametrize("m,k", [
    (2, 1), (31, 33), (33, 1000), (257, 70),    # fewer rows or columns than a warp's share
    (512, 4100), (1100, 513), (5000, 300),      # warps, then CTAs, that split the columns; whole rows
    (65, 40001), (3, 70000),                    # column chunks over CTAs in both forms
])
def test_matvec_shapes(ctx, oracle, la, m, k):
    """Matrix-vector products over the row and column splits of both forms,
    with a strided x and y, and the row-vector product with the transpose."""
    import torch
    rng = np.random.default_rng(m + k)
    a, x, c = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, 1)), rng.uniform(-1, 1, (m, 1))
    stored = a if la == 0 else a.T
    at = torch.from_numpy(np.ascontiguousarray(stored)).cuda()
    xt = torch.full((k, 3), 9.0, dtype=torch.float64)
    xt[:, 0] = torch.from_numpy(x[:, 0])
    yt = torch.full((m, 2), 7.0, dtype=torch.float64)
    yt[:, 0] = torch.from_numpy(c[:, 0])
    xt, yt = xt.cuda(), yt.cuda()
    row = torch.from_numpy(c.T.copy()).cuda()
    torch.cuda.synchronize()
    ctx.dgemm_device(la, 0, m, 1, k, 1.5, at.data_ptr(), at.shape[1], xt.data_ptr(), 3, -0.5, yt.data_ptr(), 2)
    # y^T = x^T A^T: B = A^T is stored as A is, in the other layout
    ctx.dgemm_device(1, 1 - la, 1, m, k, 1.5, xt.data_ptr(), 3, at.data_ptr(), at.shape[1], -0.5, row.data_ptr(), m)
    ctx.synchronize()
    y = yt.cpu().numpy()
    assert (y[:, 1] == 7.0).all()
    assert_fp64_bound(f"matvec {m}x{k}", y[:, :1], a, x, c, 1.5, -0.5)
    assert_fp64_bound(f"vecmat {m}x{k}", row.cpu().numpy(), x.T, a.T, c.T, 1.5, -0.5)


@pytest.mark.parametrize("la", [0, 1])
@pytest.mark.parametrize("m,k", [(20001, 2), (9000, 31), (5000, 64), (5000, 65), (300, 700), (50, 50), (12345, 1)])
def test_gemv_of_few_columns(ctx, oracle, la, m, k):
    """Tall matrices of few columns: the row form's short tail (up to two steps
    of 32 columns) and the column form that needs no partial sums."""
    import torch
    A, B, C = oracle.uniform((m, k), 61 + k), oracle.uniform((k, 1), 62 + k), oracle.uniform((m, 1), 63 + k)
    dA = torch.from_numpy(np.ascontiguousarray(A if la == 0 else A.T)).cuda()
    dB, dC = torch.from_numpy(B).cuda(), torch.from_numpy(C.copy()).cuda()
    ctx.dgemm_device(la, 0, m, 1, k, 1.5, dA.data_ptr(), dA.shape[1], dB.data_ptr(), 1, 0.5, dC.data_ptr(), 1)
    ctx.synchronize()
    assert_fp64_bound(f"gemv {m}x{k} la={la}", dC.cpu().numpy(), A, B, C, 1.5, 0.5)


def test_captured_split_products_among_others(oracle):
    """A captured split product, replayed between eager split products of the
    same context: every result has the bits of the first."""
    import jlc_b200
    import torch
    ctx, st = jlc_b200.Context(0), torch.cuda.Stream()
    try:
        ctx.set_stream(st.cuda_stream)
        shapes = [(640, 512, 2048), (256, 256, 4096)]
        ops = [(torch.from_numpy(oracle.uniform((m, k), 71 + i)).cuda(),
                torch.from_numpy(oracle.uniform((k, n), 81 + i)).cuda(),
                torch.zeros(m, n, dtype=torch.float64, device="cuda")) for i, (m, n, k) in enumerate(shapes)]
        torch.cuda.synchronize()

        def product(i):
            (m, n, k), (a, b, c) = shapes[i], ops[i]
            assert ctx.splitk_choice(m, n, k) > 1
            ctx.dgemm_device(0, 0, m, n, k, 1.0, a.data_ptr(), k, b.data_ptr(), n, 0.0, c.data_ptr(), n, report=False)

        def result(i):
            ctx.synchronize()
            c = ops[i][2].clone()
            ops[i][2].zero_()
            torch.cuda.synchronize()
            return c

        first = []
        for i in (0, 1):
            product(i)
            first.append(result(i))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            product(0)
        for step in (0, 0, 1, 0, "eager 0", 0, 1, 1, 0):
            if step == 1 or step == "eager 0":
                i = 1 if step == 1 else 0
                product(i)
            else:
                i = 0
                with torch.cuda.stream(st):
                    graph.replay()
            assert torch.equal(result(i), first[i]), step
    finally:
        ctx.close()


@pytest.mark.parametrize("m,k", [(1, 100001), (7, 40000), (100, 16384), (443, 9000), (33, 4097)])
def test_few_long_rows_captured_by_a_new_context(oracle, m, k):
    """A matrix-vector product of few rows, whose columns are split over the
    CTAs of a cluster, takes no device memory: the first call of a context can
    be captured.  The replay and an eager call give the same bits."""
    import jlc_b200
    import torch
    ctx, st = jlc_b200.Context(0), torch.cuda.Stream()
    try:
        ctx.set_stream(st.cuda_stream)
        A, B, C = oracle.uniform((m, k), 91), oracle.uniform((k, 1), 92), oracle.uniform((m, 1), 93)
        dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
        dC = [torch.from_numpy(C.copy()).cuda() for _ in range(2)]

        def product(c):
            ctx.dgemm_device(0, 0, m, 1, k, 1.5, dA.data_ptr(), k, dB.data_ptr(), 1, 0.5, c.data_ptr(), 1, report=False)

        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            product(dC[0])
        with torch.cuda.stream(st):
            graph.replay()
        product(dC[1])
        ctx.synchronize()
        assert torch.equal(dC[0], dC[1])
        assert_fp64_bound(f"gemv {m}x{k}", dC[0].cpu().numpy(), A, B, C, 1.5, 0.5)
    finally:
        ctx.close()


def test_tuned_splits_are_those_of_the_shape(ctx, tmp_path, monkeypatch):
    """65 x 300 and 128 x 384 products have as many 128-column tiles, but the
    kernel cuts them into different numbers of smaller ones: an entry tuned for
    one is not the other's.  An entry that names 128-column tiles alone, as an
    earlier kernel stored it, is nobody's."""
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("JLCGPU_TUNE_CACHE", str(cache))
    ctx.autotune_splitk(96, 100, 1024)
    prefix = cache.read_text().split("dmma-splitk")[0] + "dmma-splitk"
    cache.write_text(f"{prefix}|t3|kb8 5\n{prefix}|t3|kb8|r4x12 5\n")
    assert ctx.splitk_choice(128, 384, 4096) == 5
    assert ctx.splitk_choice(65, 300, 4096) != 5
    assert ctx.splitk_choice(100, 300, 4096) != 5   # r4x10


@pytest.mark.parametrize("k_step", [4, 16])
@pytest.mark.parametrize("m,n,k", [(2048, 1024, 512), (1064, 1024, 512), (1536, 1100, 300)])
def test_k_step_setting_in_row_blocks(oracle, monkeypatch, k_step, m, n, k):
    """JLCGPU_DMMA_K: the row blocks of a pipelined host product, the last one
    of 40 rows too, sum in the same steps of k as the device entry's product."""
    import jlc_b200
    import torch
    monkeypatch.setenv("JLCGPU_DMMA_K", str(k_step))
    ctx = jlc_b200.Context(0)
    monkeypatch.delenv("JLCGPU_DMMA_K")
    try:
        A, B = oracle.uniform((m, k), 95), oracle.uniform((k, n), 96)
        dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
        dC = torch.zeros((m, n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.dgemm_device(0, 0, m, n, k, 1.0, dA.data_ptr(), k, dB.data_ptr(), n, 0.0, dC.data_ptr(), n, report=False)
        ctx.synchronize()
        host = np.zeros((m, n))
        ctx.dgemm(0, 0, m, n, k, 1.0, A, k, B, n, 0.0, host, n, precision=0)
        np.testing.assert_array_equal(host, dC.cpu().numpy())
        assert_fp64_bound(f"k step {k_step}", host, A, B, None, 1.0, 0.0)
    finally:
        ctx.close()


@pytest.mark.parametrize("m,n,k", [(301, 6144, 1614), (256, 256, 4096)])
def test_split_product_without_a_workspace(oracle, m, n, k):
    """A product that would be split along k runs unsplit where the partial
    sums find no room: as the first call of a context, captured into a graph,
    and where the allocation fails."""
    import jlc_b200
    import torch
    ctx, st = jlc_b200.Context(0), torch.cuda.Stream()
    try:
        ctx.set_stream(st.cuda_stream)
        assert ctx.splitk_choice(m, n, k) > 1
        A, B = oracle.uniform((m, k), 97), oracle.uniform((k, n), 98)
        dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
        dC = [torch.zeros((m, n), dtype=torch.float64, device="cuda") for _ in range(3)]

        def product(c):
            ctx.dgemm_device(0, 0, m, n, k, 1.0, dA.data_ptr(), k, dB.data_ptr(), n, 0.0, c.data_ptr(), n, report=False)

        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            product(dC[0])
        with torch.cuda.stream(st):
            graph.replay()
        ctx.inject_fault(1)   # the next allocation
        product(dC[1])
        product(dC[2])        # with a workspace: split
        ctx.synchronize()
        assert torch.equal(dC[0], dC[1])
        rows, cols = oracle.sample_entries(m, n, 2000, 3)
        for c in (dC[0], dC[2]):
            assert_fp64_bound(f"{m}x{n}x{k}", c.cpu().numpy(), A, B, None, 1.0, 0.0, rows=rows, cols=cols)
    finally:
        ctx.close()
