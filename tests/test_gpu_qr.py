"""GPU parity of the device-resident blocked Householder QR against the
oracle's restatement of the reference (HouseholderQR.factorizeBlocked and
buildQ): factor, tau and Q within rounding of the restatement, A = QR and Q
orthogonal to rounding, and the same bits on every run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(ctx, a, lda=None):
    import torch
    m, n = a.shape
    lda = lda or m
    at = torch.zeros((n, lda), dtype=torch.float64, device="cuda")  # column-major A: column j at row j of at
    at[:, :m] = torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    tau = torch.zeros(max(1, min(m, n)), dtype=torch.float64, device="cuda")
    ctx.qr_factor_device(m, n, at.data_ptr(), lda, tau.data_ptr())
    ctx.synchronize()
    return at, tau


def _q(ctx, at, tau, m, n, lda, qcols):
    import torch
    q = torch.zeros((qcols, m), dtype=torch.float64, device="cuda")
    ctx.qr_build_q_device(m, n, qcols, at.data_ptr(), lda, tau.data_ptr(), q.data_ptr(), m)
    ctx.synchronize()
    return q.cpu().numpy().T


@pytest.mark.parametrize("m,n,pad", [(96, 80, 0), (200, 150, 3), (130, 200, 0), (257, 64, 1), (300, 300, 0),
                                     (64, 64, 0), (1000, 190, 0)])
def test_qr_matches_restatement(ctx, oracle, m, n, pad):
    a = oracle.uniform((m, n), 31 * m + n)
    lda = m + pad
    at, tau = _factor(ctx, a, lda)
    f = at[:, :m].cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    k = min(m, n)
    np.testing.assert_allclose(tau.cpu().numpy()[:k], tau_ref, rtol=0, atol=1e-12)
    np.testing.assert_allclose(f, f_ref, rtol=0, atol=1e-11 * max(1.0, np.abs(f_ref).max()))
    q = _q(ctx, at, tau, m, n, lda, m)
    q_ref = oracle.householder_build_q(f_ref, tau_ref, m)
    np.testing.assert_allclose(q, q_ref, rtol=0, atol=1e-11)
    r = np.triu(f)
    assert np.linalg.norm(a - q @ r) <= 1e-13 * np.linalg.norm(a)
    assert np.linalg.norm(q.T @ q - np.eye(m)) <= 1e-12


def test_qr_thin_q_and_determinism(ctx, oracle):
    m, n = 500, 140
    a = oracle.uniform((m, n), 5)
    at1, tau1 = _factor(ctx, a)
    at2, tau2 = _factor(ctx, a)
    np.testing.assert_array_equal(at1.cpu().numpy(), at2.cpu().numpy())
    np.testing.assert_array_equal(tau1.cpu().numpy(), tau2.cpu().numpy())
    q = _q(ctx, at1, tau1, m, n, m, n)  # thin Q: m x n
    r = np.triu(at1[:, :m].cpu().numpy().T)[:n, :]
    assert np.linalg.norm(a - q @ r) <= 1e-13 * np.linalg.norm(a)


def test_qr_zero_column(ctx, oracle):
    a = oracle.uniform((90, 70), 9)
    a[:, 10] = 0.0
    at, tau = _factor(ctx, a)
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    assert tau.cpu().numpy()[10] == 0.0 and tau_ref[10] == 0.0
    np.testing.assert_allclose(at[:, :90].cpu().numpy().T, f_ref, rtol=0, atol=1e-11)


@pytest.mark.parametrize("m,n", [(60000, 70), (8000, 130)])
def test_qr_tall_panel(ctx, oracle, m, n):
    """Tall panels, against the restatement and R against the Gram matrix
    (R^T R = A^T A).  60000 x 70: the first panel's rows per CTA (406 x 64
    doubles, one CTA per SM) exceed the shared-memory slab and are factored in
    place, the second panel (6 columns) runs on one cluster.  8000 x 130: the
    first two panels' slabs do not fit a 16-CTA cluster (500 x 64 doubles) and
    run as a cooperative grid with slabs in shared memory, the third on a
    cluster."""
    a = oracle.uniform((m, n), 77)
    at, tau = _factor(ctx, a)
    f = at[:, :m].cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    np.testing.assert_allclose(tau.cpu().numpy()[:n], tau_ref, rtol=0, atol=1e-12)
    np.testing.assert_allclose(f, f_ref, rtol=0, atol=1e-11 * max(1.0, np.abs(f_ref).max()))
    r = np.triu(f[:n, :])
    g = a.T @ a
    assert np.abs(r.T @ r - g).max() <= 1e-12 * np.abs(g).max()


# stress/HouseholderQRTest.java:14-120 replayed through the device route: the
# same java.util.Random inputs, checks and tolerances
REF_QR_SEED, REF_QR_SIZES, REF_QR_TOL = 12345, [1, 2, 3, 5, 10, 20, 50, 100], 1e-12


@pytest.mark.parametrize("case", ["reconstruction", "orthogonality"])
def test_reference_qr_cases(ctx, oracle, case):
    seed = REF_QR_SEED + (0 if case == "reconstruction" else 1)
    for a, n in zip(oracle.qr_test_matrices(seed, [(n, n) for n in REF_QR_SIZES]), REF_QR_SIZES):
        at, tau = _factor(ctx, a)
        q = _q(ctx, at, tau, n, n, n, n)
        r = np.triu(at[:, :n].cpu().numpy().T)
        if case == "reconstruction":
            assert np.linalg.norm(q @ r - a) / np.linalg.norm(a) < REF_QR_TOL, n
        else:
            assert np.linalg.norm(q.T @ q - np.eye(n)) < REF_QR_TOL, n


def test_reference_thin_qr_case(ctx, oracle):
    (a,) = oracle.qr_test_matrices(REF_QR_SEED + 3, [(100, 40)])
    at, tau = _factor(ctx, a)
    q = _q(ctx, at, tau, 100, 40, 100, 40)
    r = np.triu(at[:, :100].cpu().numpy().T)[:40, :]
    assert np.linalg.norm(q @ r - a) / np.linalg.norm(a) < REF_QR_TOL
    assert np.linalg.norm(q.T @ q - np.eye(40)) < REF_QR_TOL


def _ref_matrix(a):
    import jlc_b200
    return jlc_b200.Matrix.wrap(np.ascontiguousarray(a).ravel(), *a.shape)


def _np(mat):
    return mat.to_numpy()


def test_reference_qr_test_file_through_mirror(ctx, oracle):
    """stress/HouseholderQRTest.java's four tests, written against the
    HouseholderQR mirror as the Java test is written against HouseholderQR."""
    from jlc_b200 import HouseholderQR
    for seed, case in ((REF_QR_SEED, "reconstruction"), (REF_QR_SEED + 1, "orthogonality"),
                       (REF_QR_SEED + 2, "upper")):
        for a, n in zip(oracle.qr_test_matrices(seed, [(n, n) for n in REF_QR_SIZES]), REF_QR_SIZES):
            qr = HouseholderQR.decompose(_ref_matrix(a), ctx=ctx)
            q, r = _np(qr.getQ()), _np(qr.getR())
            assert q.shape == (n, n) and r.shape == (n, n)
            if case == "reconstruction":
                assert np.linalg.norm(q @ r - a) / np.linalg.norm(a) < REF_QR_TOL, n
            elif case == "orthogonality":
                assert np.linalg.norm(q.T @ q - np.eye(n)) < REF_QR_TOL, n
            else:
                assert np.abs(np.tril(r, -1)).max(initial=0.0) < 1e-12, n
    (a,) = oracle.qr_test_matrices(REF_QR_SEED + 3, [(100, 40)])
    qr = HouseholderQR.decomposeThin(_ref_matrix(a), ctx=ctx)
    q, r = _np(qr.getQ()), _np(qr.getR())
    assert q.shape == (100, 40) and r.shape == (40, 40)
    assert np.linalg.norm(q @ r - a) / np.linalg.norm(a) < REF_QR_TOL
    assert np.linalg.norm(q.T @ q - np.eye(40)) < REF_QR_TOL


def test_mirror_shapes_and_factorize(ctx, oracle):
    from jlc_b200 import HouseholderQR
    a = oracle.uniform((70, 90), 4)           # wide: R is m x n, thin Q is m x m
    qr = HouseholderQR.decompose(_ref_matrix(a), ctx=ctx)
    assert _np(qr.getQ()).shape == (70, 70) and _np(qr.getR()).shape == (70, 90)
    assert np.linalg.norm(_np(qr.getQ()) @ _np(qr.getR()) - a) <= 1e-13 * np.linalg.norm(a)
    before = a.copy()
    HouseholderQR.factorize(_ref_matrix(a), ctx=ctx)  # factors a copy
    np.testing.assert_array_equal(a, before)


@pytest.mark.parametrize("m,n", [(2000, 130), (8000, 130), (60000, 70)])
def test_qr_extreme_column_scales(ctx, oracle, m, n):
    """Columns scaled by 2^900, 2^-900 and 1: products of two such entries
    overflow or underflow, so the panel must scale before it forms squares
    and dots, as the reference's normalised reflector does.  With power-of-two
    scales S, QR(A S) has QR(A)'s reflectors and tau and R S (exactly, on the
    restatement), so the device result is checked against the restatement of
    the unscaled A.  One shape per panel kernel: one cluster, a grid with
    slabs in shared memory, a grid in place."""
    a = oracle.uniform((m, n), 5 + m)
    s = np.array([2.0 ** 900 if j % 3 == 0 else (2.0 ** -900 if j % 3 == 1 else 1.0) for j in range(n)])
    at, tau = _factor(ctx, a * s)
    f = at[:, :m].cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    assert np.isfinite(f).all()
    np.testing.assert_allclose(tau.cpu().numpy()[:n], tau_ref, rtol=0, atol=1e-12)
    up = np.triu(np.ones((m, n), bool))
    tol = 1e-11 * max(1.0, np.abs(f_ref).max())
    np.testing.assert_allclose(np.where(up, f / s, 0.0), np.where(up, f_ref, 0.0), rtol=0, atol=tol)
    np.testing.assert_allclose(np.where(up, 0.0, f), np.where(up, 0.0, f_ref), rtol=0, atol=tol)


@pytest.mark.parametrize("m,n", [
    (64, 64), (127, 70), (128, 64), (129, 30),      # one CTA of up to four row slots, two CTAs
    (1024, 70), (1025, 70), (2049, 64), (2561, 70),  # 16 CTAs of 64, 65, 129 and 161 rows
    (4096, 37), (4097, 70), (4500, 130),            # the last size in registers; past it; both in one factorisation
])
def test_panel_kernel_edges(ctx, oracle, m, n):
    """The panel at the row counts where its cluster size, its rows per lane
    and its kernel change, and panels narrower than 64 columns, against the
    restatement (tolerances as for the other sizes)."""
    a = oracle.uniform((m, n), 7 * m + n)
    if n > 40:
        a[3:, 2] = 0.0      # a reflector whose tail vanishes after two steps, or nearly
        a[:, 20] = 0.0      # a zero column
    at, tau = _factor(ctx, a)
    f = at[:, :m].cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    np.testing.assert_allclose(tau.cpu().numpy()[:n], tau_ref, rtol=0, atol=1e-12)
    np.testing.assert_allclose(f, f_ref, rtol=0, atol=1e-11 * max(1.0, np.abs(f_ref).max()))


def test_panel_sign_flip_and_last_row(ctx, oracle):
    """A column that is zero below a negative diagonal entry (tau = 2, a sign
    flip) and a square panel, whose last column has no reflector."""
    a = np.triu(oracle.uniform((64, 64), 71))
    a[5, 5] = -0.75
    a[6, 6] = 0.5
    at, tau = _factor(ctx, a)
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    np.testing.assert_allclose(tau.cpu().numpy(), tau_ref, rtol=0, atol=1e-12)
    np.testing.assert_allclose(at[:, :64].cpu().numpy().T, f_ref, rtol=0, atol=1e-11)


@pytest.mark.parametrize("m,n,qcols", [
    (300, 200, 100), (300, 130, 300), (65, 64, 65), (200, 300, 150),   # fewer, more columns than reflectors
    (20000, 1000, 1000),   # more panels than one batch's workspace; panels above 4096 rows
])
def test_q_in_batches(ctx, m, n, qcols):
    """The first columns of Q, formed from panels whose V and T come in
    batches: orthonormal, and Q^T A is R.  Checked with torch in FP64; a
    backward stable Q leaves a small multiple of m u."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.rand(n, m, dtype=torch.float64, device="cuda", generator=g) * 2 - 1   # column-major m x n
    f, tau = a.clone(), torch.zeros(min(m, n), dtype=torch.float64, device="cuda")
    q = torch.zeros(qcols, m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.qr_factor_device(m, n, f.data_ptr(), m, tau.data_ptr())
    ctx.qr_build_q_device(m, n, qcols, f.data_ptr(), m, tau.data_ptr(), q.data_ptr(), m)
    tol = 1e-14 * max(m, n)
    assert float((q @ q.T - torch.eye(qcols, dtype=torch.float64, device="cuda")).norm()) < tol
    r = torch.triu(f.T[:min(m, n)])
    rows = min(qcols, min(m, n))
    assert float((q[:rows] @ a.T - r[:rows]).norm() / a.norm()) < tol


@pytest.mark.parametrize("m", [64, 100, 127, 200])
def test_last_columns_of_a_panel(ctx, oracle, m):
    """The last columns of a 64-column panel, where some warps have no column
    left, on one CTA and on a small cluster: the same bits on 200 runs, with
    columns whose scales differ by 2^1800, and every column as the restatement
    of the unscaled matrix has it."""
    import torch
    n = 64
    a = oracle.uniform((m, n), 90 + m)
    s = np.array([2.0 ** (900 if j % 2 else -900) for j in range(n)])
    at = torch.from_numpy(np.ascontiguousarray((a * s).T)).cuda()
    work, first = torch.empty_like(at), None
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    for _ in range(200):
        work.copy_(at)
        torch.cuda.synchronize()
        ctx.qr_factor_device(m, n, work.data_ptr(), m, tau.data_ptr())
        if first is None:
            first = work.clone()
        assert torch.equal(work, first)
    f = first.cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    np.testing.assert_allclose(tau.cpu().numpy(), tau_ref, rtol=0, atol=1e-12)
    up = np.triu(np.ones((m, n), bool))
    f = np.where(up, f / s, f)
    np.testing.assert_allclose(f, f_ref, rtol=0, atol=1e-11 * max(1.0, np.abs(f_ref).max()))


@pytest.mark.parametrize("m,n,i,j", [(60, 40, 5, 0), (60, 40, 5, 7), (60, 40, 7, 7), (300, 60, 200, 30), (300, 60, 0, 0)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_column_of_a_panel(ctx, oracle, m, n, i, j, bad):
    """A NaN or an infinity in column j of a one-panel matrix.  The columns
    before j are finished before it is reached: their reflectors and R's rows
    above j keep the bits they have with the column zeroed.  A NaN norm gives
    no reflector when the column's entry on the diagonal is a NaN too, and the
    columns after j are then those of the matrix without it."""
    a = oracle.uniform((m, n), 300 + m + j)
    a[0] = np.abs(a[0])      # a NaN below a positive diagonal entry leaves the column without a reflector
    zeroed, poisoned = a.copy(), a.copy()
    zeroed[:, j], poisoned[i, j] = 0.0, bad
    f, tau = (x.cpu().numpy() for x in _factor(ctx, poisoned))
    f0, tau0 = (x.cpu().numpy() for x in _factor(ctx, zeroed))
    f, f0 = f.T, f0.T
    assert np.isfinite(f0).all()
    np.testing.assert_array_equal(f[:, :j], f0[:, :j])          # finished columns
    np.testing.assert_array_equal(tau[:j], tau0[:j])
    np.testing.assert_array_equal(f[:j, j + 1:], f0[:j, j + 1:])  # finished rows
    if np.isnan(bad) and (i, j) != (0, 0):
        assert tau[j] == 0.0
        np.testing.assert_array_equal(f[:, j + 1:], f0[:, j + 1:])


def test_denormals_beside_normal_entries(ctx, oracle):
    """A column whose maximum is a normal number on one CTA while the rows of
    the others hold only denormals: they are part of the reflector.  A column
    of denormals alone has none, as in the restatement."""
    m, n = 300, 8
    a = oracle.uniform((m, n), 77) * 2.0 ** -1030
    a[3] = oracle.uniform((1, n), 78)[0] * 2.0 ** -1015
    at, tau = _factor(ctx, a)
    f = at[:, :m].cpu().numpy().T
    f_ref, tau_ref = oracle.householder_qr_blocked(a)
    # a denormal entry carries an absolute error of 2^-1075, 2^-60 of the columns' maxima
    np.testing.assert_allclose(tau.cpu().numpy()[0], tau_ref[0], rtol=0, atol=1e-12)
    np.testing.assert_allclose(f[1:, 0], f_ref[1:, 0], rtol=0, atol=1e-11)
    assert np.abs(f[4:, 0]).max() > 1e-6
    z = np.full((100, 1), 2.0 ** -1040)
    at, tau = _factor(ctx, z)
    assert tau.cpu().numpy()[0] == 0.0
    np.testing.assert_array_equal(at.cpu().numpy().T, z)


def test_q_with_little_room(ctx, oracle):
    """Where the workspace for all panels finds no room, Q is formed in smaller
    batches (the sums of V^T V may be cut differently: equal to rounding, a
    small multiple of m u); a factorisation, one panel at a time, reports the
    failure."""
    from jlc_b200 import JlcError
    import jlc_b200
    c2 = jlc_b200.Context(0)
    try:
        m, n = 700, 500
        a = oracle.uniform((m, n), 41)
        at, tau = _factor(ctx, a)
        q = _q(ctx, at, tau, m, n, m, n)
        c2.inject_fault(1)   # the next allocation
        assert np.abs(_q(c2, at, tau, m, n, m, n) - q).max() < 1e-14 * m
        c3 = jlc_b200.Context(0)
        c3.inject_fault(1)
        with pytest.raises(JlcError) as exc:
            _factor(c3, a)
        assert exc.value.code == -3
        c3.close()
    finally:
        c2.close()


def test_launch_count_of_tall_panels(ctx):
    """One panel of Q takes two launches for V, T and V T, and five above 4096
    rows, beside the same two GEMMs."""
    import torch
    counts = []
    for m in (4000, 4200):
        f, tau = torch.full((64, m), 0.01, dtype=torch.float64, device="cuda"), torch.ones(64, dtype=torch.float64).cuda()
        q = torch.zeros(64, m, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        before = ctx.launch_count()
        ctx.qr_build_q_device(m, 64, 64, f.data_ptr(), m, tau.data_ptr(), q.data_ptr(), m)
        counts.append(ctx.launch_count() - before)
    assert counts[1] - counts[0] == 3
