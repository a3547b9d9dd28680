"""The blocked Hessenberg reduction on the device against the reference's own
tests and the oracle's restatement (BlockedHessenbergQR.decompose,
eigen/qr/BlockedHessenbergQR.java:99-146).

The reference's cases (DecompositionTests.testHessenberg_*Random,
DecompositionTests.java:1150-1183, sizes 2..200 on java.util.Random(700/800/900
+ n); stress/HessenbergDebugTest) run through BlockedHessenbergQR.decompose on
their exact inputs with the reference's four checks and tolerances: H upper
Hessenberg, Q orthogonal, the trace kept, A = Q H Q^T.  Larger matrices
(several panels, a partial last panel, a zero column that skips reflectors)
are compared with the oracle's restatement entry by entry."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tolerance(n):
    # DecompositionTests.getTolerance (decomposition/DecompositionTests.java:183-188)
    if n <= 10:
        return 1e-10 * math.sqrt(n)
    if n <= 30:
        return 1e-8 * math.sqrt(n)
    if n <= 100:
        return 1e-6 * math.sqrt(n)
    return 1e-5 * math.sqrt(n)


def _check_hessenberg(a, h, q, tol):
    # testHessenbergReduction (DecompositionTests.java:1193-1224)
    n = a.shape[0]
    assert np.abs(np.tril(h, -2)).max(initial=0.0) <= tol
    assert np.linalg.norm(q.T @ q - np.eye(n)) < tol
    assert abs(np.trace(a) - np.trace(h)) <= tol * abs(np.trace(a)) + tol
    assert np.linalg.norm(a - q @ h @ q.T) / np.linalg.norm(a) < tol


def _device(a, ctx=None, precision=0):
    from jlc_b200 import BlockedHessenbergQR, Matrix
    n = a.shape[0]
    res = BlockedHessenbergQR.decompose(Matrix.wrap(np.ascontiguousarray(a).ravel().copy(), n, n), ctx=ctx,
                                        precision=precision)
    return res.getH().to_numpy(), res.getQ().to_numpy(), res


CASES = [(n, 700 + n) for n in (2, 3, 4, 5, 6, 7, 8, 9, 10)] + \
        [(n, 800 + n) for n in (15, 20, 25, 30)] + \
        [(n, 900 + n) for n in (50, 100, 200)]


@pytest.mark.parametrize("n,seed", CASES)
def test_reference_hessenberg_cases(oracle, n, seed):
    a = oracle.java_random_matrix(seed, n, n)
    h, q, _ = _device(a)
    _check_hessenberg(a, h, q, _tolerance(n))
    h_ref, q_ref = oracle.blocked_hessenberg(a)
    scale = max(1.0, np.abs(a).max())
    np.testing.assert_allclose(h, h_ref, rtol=0, atol=1e-11 * scale * n)
    np.testing.assert_allclose(q, q_ref, rtol=0, atol=1e-11 * n)


def test_reference_hessenberg_debug_case(oracle):
    d = oracle.java_random_doubles(1234567, 4 + 9 + 16) * 2.0 - 1.0
    o = 0
    for n in (2, 3, 4):
        a = d[o:o + n * n].reshape(n, n)
        o += n * n
        h, q, res = _device(a)
        assert np.linalg.norm(a - q @ h @ q.T) < 0.01
        assert res.residualNorm() < 1e-12
        _check_hessenberg(a, h, q, _tolerance(n))


@pytest.mark.parametrize("n", [97, 256, 513])
def test_matches_restatement_on_larger_matrices(ctx, oracle, n):
    """Several panels and a partial last panel; A's eigenvalues kept."""
    a = oracle.uniform((n, n), 2000 + n)
    h, q, _ = _device(a, ctx)
    h_ref, q_ref = oracle.blocked_hessenberg(a)
    np.testing.assert_allclose(h, h_ref, rtol=0, atol=1e-12 * n)
    np.testing.assert_allclose(q, q_ref, rtol=0, atol=1e-12 * n)
    assert np.linalg.norm(a - q @ h @ q.T) / np.linalg.norm(a) < 1e-13
    assert np.linalg.norm(q.T @ q - np.eye(n)) < 1e-12 * n
    if n <= 256:
        ev_a = np.sort_complex(np.linalg.eigvals(a))
        ev_h = np.sort_complex(np.linalg.eigvals(h))
        np.testing.assert_allclose(ev_h, ev_a, rtol=0, atol=1e-9)


def test_skipped_reflectors(ctx, oracle):
    """Columns already in Hessenberg form below the subdiagonal give sigma = 0:
    the reference skips those reflectors (tau = 0), and so does the device."""
    n = 70
    a = oracle.uniform((n, n), 2101)
    a[3:, 1] = 0.0     # column 1: nothing below its subdiagonal
    a[36:, 33] = 0.0   # inside the second panel
    h, q, _ = _device(a, ctx)
    h_ref, q_ref = oracle.blocked_hessenberg(a)
    np.testing.assert_allclose(h, h_ref, rtol=0, atol=1e-12 * n)
    np.testing.assert_allclose(q, q_ref, rtol=0, atol=1e-12 * n)


def test_ozaki_precision_block_updates(ctx, oracle):
    """The block updates on the Ozaki route (certified, or FP64 where the
    certificate cannot prove the bound) give the same reduction."""
    n = 300
    a = oracle.uniform((n, n), 2201)
    h, q, _ = _device(a, ctx, precision=3)
    h_ref, q_ref = oracle.blocked_hessenberg(a)
    np.testing.assert_allclose(h, h_ref, rtol=0, atol=1e-11 * n)
    assert np.linalg.norm(a - q @ h @ q.T) / np.linalg.norm(a) < 1e-13


def test_device_entry_arguments(ctx):
    import torch
    from jlc_b200 import ArithmeticException, BlockedHessenbergQR, IllegalArgumentException, Matrix
    with pytest.raises(IllegalArgumentException):
        BlockedHessenbergQR.decompose(None)
    with pytest.raises(ArithmeticException):
        BlockedHessenbergQR.decompose(Matrix(3, 4))
    a = torch.zeros((4, 4), dtype=torch.float64, device="cuda")
    with pytest.raises(IllegalArgumentException):
        ctx.hessenberg_device(4, a.data_ptr(), 3, None, 4)
    # without Q
    a = torch.from_numpy(np.arange(16, dtype=np.float64).reshape(4, 4) % 5 + 1.0).cuda()
    ctx.hessenberg_device(4, a.data_ptr(), 4, None, 4)
    h = a.cpu().numpy().T  # the buffer is column-major
    assert np.all(np.tril(h, -2) == 0.0)


@pytest.mark.parametrize("n,with_q", [
    (3, True), (9, True),            # one CTA, two CTAs
    (512, True),                     # one column per thread
    (513, True), (1024, False),      # one column past a thread's first; 8 rows per CTA
    (1025, True), (1184, False),     # three columns per thread, 8 rows per CTA
    (1200, True), (1537, True),      # 16 rows per CTA, three columns per thread; four
    (1744, True), (1745, True),      # the largest order in shared memory, the smallest of the panel route
])
def test_route_edges(ctx, n, with_q):
    """A = Q H Q^T (or the eigenvalue-preserving norms without Q) at the sizes
    where the one-launch kernel's layout or the route changes, checked with
    torch in FP64 against a backward stable reduction's residual (a small
    multiple of n u)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(2300 + n)
    a = torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1   # column-major
    f = torch.zeros(n, n + 3, dtype=torch.float64, device="cuda")                   # padded leading dimension
    f[:, :n] = a
    q = torch.empty(n, n, dtype=torch.float64, device="cuda") if with_q else None
    torch.cuda.synchronize()
    ctx.hessenberg_device(n, f.data_ptr(), n + 3, q.data_ptr() if with_q else None, n)
    assert float(f[:, n:].abs().max()) == 0.0
    h = f[:, :n].T
    assert float(torch.tril(h, -2).abs().max()) == 0.0
    tol = 1e-14 * n
    assert abs(float(h.norm() / a.norm()) - 1.0) < tol
    assert abs(float(h.trace() - a.trace())) < tol * float(a.norm())
    if with_q:
        q = q.T
        assert float((a.T - q @ h @ q.T).norm() / a.norm()) < tol
        assert float((q.T @ q - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) < tol * n ** 0.5


@pytest.mark.parametrize("n", [40, 200])
@pytest.mark.parametrize("i,j,bad", [(0, 7, np.nan), (0, 7, np.inf), (5, 7, np.nan), (5, 0, np.nan), (39, 38, np.nan)])
def test_q_of_a_matrix_with_a_non_finite_entry(ctx, oracle, n, i, j, bad):
    """A column whose norm is a NaN has no reflector: Q is the product of the
    others, finite and orthogonal.  (An infinity below the diagonal makes the
    reflector itself NaN: only Q's first column is left.)"""
    import torch
    a = oracle.uniform((n, n), 1800 + n)
    a[i, j] = bad
    h = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    q = torch.zeros_like(h)
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    ctx.hessenberg_device(n, h.data_ptr(), n, q.data_ptr(), n)
    assert float((q.T @ q - eye).abs().max()) < 1e-14 * n
    a[i, j] = 0.5
    a[5, 0] = np.inf
    h = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    ctx.hessenberg_device(n, h.data_ptr(), n, q.data_ptr(), n)
    assert torch.equal(q[0], eye[0])   # column-major: Q's first column


@pytest.mark.parametrize("n", [40, 200, 700])   # 8 rows per CTA; one and two columns per thread
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_entries_stay_where_a_reduction_leaves_them(ctx, oracle, n, bad):
    """Row 0 takes part in no reflector's dots: an entry there that is not
    finite changes row 0 alone, and Q not at all.  An entry below it reaches
    the rows from 1 on, but not row 0.  A NaN in column 0, whose reflector is
    then skipped, changes that column alone."""
    import torch
    clean = oracle.uniform((n, n), 1900 + n)

    def reduce(i, j, value):
        a = clean.copy()
        a[i, j] = value
        h, q = torch.from_numpy(np.ascontiguousarray(a.T)).cuda(), torch.empty(n, n, dtype=torch.float64).cuda()
        ctx.hessenberg_device(n, h.data_ptr(), n, q.data_ptr(), n)
        return h.cpu().numpy().T, q.cpu().numpy().T

    h0, q0 = reduce(0, 7, 0.25)
    h, q = reduce(0, 7, bad)
    np.testing.assert_array_equal(h[1:], h0[1:])
    np.testing.assert_array_equal(q, q0)
    h, _ = reduce(n // 2, 7, np.nan)
    assert np.isfinite(h[0]).all() and np.isnan(h[1:, 1:][np.triu_indices(n - 1, -1)]).all()
    h0, q0 = reduce(5, 0, 0.0)
    h, q = reduce(5, 0, np.nan)
    assert np.isfinite(h[:, 1:]).all() and np.linalg.norm(q.T @ q - np.eye(n)) < 1e-14 * n
