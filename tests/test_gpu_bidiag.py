"""GPU parity of the device Golub-Kahan bidiagonalisation (jlc_bidiag_device,
the Bidiagonalization / BidiagonalizationResult mirror).

The reference's tested class is Bidiagonalization
(decomposition/bidiagonal/Bidiagonalization.java:155-309).  Its own cases
(DecompositionTests.java:1231-1330) run here unchanged on their
java.util.Random inputs, with the same checks and tolerances; larger tall,
square and wide shapes are compared entry by entry with the oracle's
restatement (oracle.bidiagonalize): the device uses the reference's reflector
recipe, so B, U and V agree with it to rounding (the norms and dots are summed
in another order)."""
import numpy as np
import pytest

from oracle import oracle as O
from test_oracle_bidiag import reference_cases, validate

pytestmark = pytest.mark.gpu


def _device(a, ctx=None):
    from jlc_b200 import Bidiagonalization, Matrix
    m, n = a.shape
    r = Bidiagonalization().decompose(Matrix.wrap(np.ascontiguousarray(a).ravel().copy(), m, n), ctx=ctx)
    return r.getU().to_numpy(), r.getB().to_numpy(), r.getV().to_numpy(), r


@pytest.mark.parametrize("shape,seed", reference_cases())
def test_reference_cases_on_device(shape, seed):
    a = O.java_random_matrix(seed, *shape)
    u, b, v, r = _device(a)
    validate(a, u, b, v)
    assert r.residualNorm() < 1e-13
    uo, bo, vo = O.bidiagonalize(a)
    np.testing.assert_allclose(b, bo, rtol=0, atol=1e-13)
    np.testing.assert_allclose(u, uo, rtol=0, atol=1e-13)
    np.testing.assert_allclose(v, vo, rtol=0, atol=1e-13)


@pytest.mark.parametrize("m,n", [(97, 60), (256, 256), (600, 333), (640, 640), (300, 517), (4000, 64), (70, 1)])
def test_against_restatement(m, n):
    a = O.uniform((m, n), 2100 + m + n)
    u, b, v, r = _device(a)
    uo, bo, vo = O.bidiagonalize(a)
    scale = np.linalg.norm(a)
    tol = 1e-14 * max(m, n) * scale
    np.testing.assert_allclose(b, bo, rtol=0, atol=tol)
    np.testing.assert_allclose(u, uo, rtol=0, atol=1e-14 * max(m, n) * 10)
    np.testing.assert_allclose(v, vo, rtol=0, atol=1e-14 * max(m, n) * 10)
    assert np.linalg.norm(u.T @ u - np.eye(u.shape[0])) < 1e-12 * max(m, n)
    assert np.linalg.norm(v.T @ v - np.eye(v.shape[0])) < 1e-12 * max(m, n)
    assert r.residualNorm() < 1e-14 * max(m, n)


def test_skipped_reflectors_and_tiny_shapes():
    """A zero column (no column reflector at that step) and a zero row tail
    (no row reflector), 1 x 1, 2 x 2 and a single row."""
    a = O.uniform((50, 20), 2201)
    a[:, 0] = 0.0   # step 0: no column reflector ...
    a[0, :] = 0.0   # ... and no row reflector (row 0's tail is still zero)
    for x in (a, np.array([[-3.0]]), O.uniform((2, 2), 2202), np.array([[3.0, -4.0, 12.0]])):
        u, b, v, r = _device(x)
        uo, bo, vo = O.bidiagonalize(x)
        np.testing.assert_allclose(b, bo, rtol=0, atol=1e-13)
        np.testing.assert_allclose(u, uo, rtol=0, atol=1e-13)
        np.testing.assert_allclose(v, vo, rtol=0, atol=1e-13)


def test_device_entry_padded_lda_without_factors_is_reproducible(ctx):
    """The C entry on a column-major array with lda > m, U and V not asked for;
    two runs give the same bits (every reduction sums in a fixed order)."""
    import torch
    m, n, lda = 700, 450, 712
    a = O.uniform((m, n), 2301)
    buf = np.zeros((n, lda))
    buf[:, :m] = a.T
    outs = []
    for _ in range(2):
        at = torch.from_numpy(buf.copy()).cuda()
        d = torch.empty(n, dtype=torch.float64, device="cuda")
        e = torch.empty(n - 1, dtype=torch.float64, device="cuda")
        ctx.bidiag_device(m, n, at.data_ptr(), lda, d.data_ptr(), e.data_ptr(), None, m, None, n)
        outs.append((d.cpu().numpy(), e.cpu().numpy(), at.cpu().numpy()))
    np.testing.assert_array_equal(outs[0][0], outs[1][0])
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    np.testing.assert_array_equal(outs[0][2], outs[1][2])
    # the padding rows of each column are untouched
    np.testing.assert_array_equal(outs[0][2][:, m:], 0.0)
    _, bo, _ = O.bidiagonalize(a)
    tol = 1e-14 * m * np.linalg.norm(a)
    np.testing.assert_allclose(outs[0][0], np.diag(bo), rtol=0, atol=tol)
    np.testing.assert_allclose(outs[0][1], np.diag(bo, 1), rtol=0, atol=tol)


def test_rejects_bad_arguments(ctx):
    from jlc_b200 import IllegalArgumentException
    with pytest.raises(IllegalArgumentException):
        ctx.bidiag_device(3, 5, 8, 3, 8, 8, None, 3, None, 5)   # m < n
    with pytest.raises(IllegalArgumentException):
        ctx.bidiag_device(5, 3, 8, 4, 8, 8, None, 5, None, 3)   # lda < m


@pytest.mark.parametrize("m,n", [
    (1025, 1025),   # 16 rows per CTA, more than two columns per thread
    (1191, 520),    # 16 rows per CTA, the last CTA's slab partly past m
    (1600, 1537),   # more than three columns per thread
    (513, 513), (9, 2), (8, 8),   # one column past a thread each; two CTAs; one CTA
    (6000, 700),    # the slab does not fit in shared memory
    (2300, 2100),   # nor here; several column blocks per thread
])
def test_slab_and_column_block_edges(ctx, m, n):
    """A = U B V^T with U and V orthogonal, at the sizes where the kernel's slab
    placement and column blocks change, checked with torch in FP64.  A
    backward stable reduction leaves residuals of a small multiple of
    max(m, n) u."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(2400 + m + n)
    a = torch.rand(n, m, dtype=torch.float64, device="cuda", generator=g) * 2 - 1   # column-major m x n
    f, u, v = a.clone(), torch.empty(m, m, dtype=torch.float64, device="cuda"), \
        torch.empty(n, n, dtype=torch.float64, device="cuda")
    d = torch.empty(n, dtype=torch.float64, device="cuda")
    e = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.bidiag_device(m, n, f.data_ptr(), m, d.data_ptr(), e.data_ptr(), u.data_ptr(), m, v.data_ptr(), n)
    b = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    i = torch.arange(n, device="cuda")
    b[i, i] = d
    b[i[:-1], i[1:]] = e[:n - 1]
    u, v = u.T, v.T
    tol = 1e-14 * max(m, n)
    assert float((a.T - u @ b @ v.T).norm() / a.norm()) < tol
    assert float((u.T @ u - torch.eye(m, dtype=torch.float64, device="cuda")).norm()) < tol * m ** 0.5
    assert float((v.T @ v - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) < tol * n ** 0.5


@pytest.mark.parametrize("s", [900, -900])
def test_range_of_the_input(ctx, s):
    """Scaling A by 2^s scales d and e by 2^s exactly and leaves the reflectors
    as they are: every sum is formed from values scaled by a power of two."""
    import torch
    m, n = 150, 130
    a = O.uniform((n, m), 2501)
    outs = []
    for scale in (1.0, 2.0 ** s):
        at = torch.from_numpy(a * scale).cuda()
        u, v = torch.empty(m, m, dtype=torch.float64).cuda(), torch.empty(n, n, dtype=torch.float64).cuda()
        d, e = torch.empty(n, dtype=torch.float64).cuda(), torch.empty(n - 1, dtype=torch.float64).cuda()
        ctx.bidiag_device(m, n, at.data_ptr(), m, d.data_ptr(), e.data_ptr(), u.data_ptr(), m, v.data_ptr(), n)
        outs.append((d.cpu().numpy() / scale, e.cpu().numpy() / scale, u.cpu().numpy(), v.cpu().numpy()))
    for x, y in zip(*outs):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("m,n", [(60, 40), (300, 150), (4200, 70)])   # the last: V^T V over the whole grid
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_factors_of_a_matrix_with_a_non_finite_entry(ctx, m, n, bad):
    """The steps whose norms are not finite have no reflector.  U and V, formed
    from the others, are finite and orthogonal, V's first row and column the
    identity's."""
    import torch
    a = O.uniform((n, m), 2600 + m)
    a[7, 3] = bad
    f = torch.from_numpy(a).cuda()
    u, v = torch.empty(m, m, dtype=torch.float64).cuda(), torch.empty(n, n, dtype=torch.float64).cuda()
    d, e = torch.empty(n, dtype=torch.float64).cuda(), torch.empty(n - 1, dtype=torch.float64).cuda()
    ctx.bidiag_device(m, n, f.data_ptr(), m, d.data_ptr(), e.data_ptr(), u.data_ptr(), m, v.data_ptr(), n)
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert torch.equal(v[0], eye[0]) and torch.equal(v[:, 0], eye[:, 0])
    assert float((v.T @ v - eye).abs().max()) < 1e-14 * n
    assert float((u.T @ u - torch.eye(m, dtype=torch.float64, device="cuda")).abs().max()) < 1e-14 * m


@pytest.mark.parametrize("m,n", [(6000, 700), (2300, 2100), (20001, 301)])   # past shared memory
def test_in_place_where_the_copy_finds_no_room(m, n):
    """The reduction keeps its rows in a work array past shared memory.  Where
    that cannot be allocated they stay in the matrix: the same bits."""
    import jlc_b200
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.rand(n, m + 2, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    outs = []
    for full in (False, True):
        ctx = jlc_b200.Context(0)
        f, d, e = a.clone(), torch.zeros(n, dtype=torch.float64).cuda(), torch.zeros(n, dtype=torch.float64).cuda()
        v = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        if full:
            ctx.inject_fault(1)   # the next allocation
        ctx.bidiag_device(m, n, f.data_ptr(), m + 2, d.data_ptr(), e.data_ptr(), None, m, v.data_ptr(), n)
        outs.append((f, d, e, v))
        ctx.close()
    for x, y in zip(*outs):
        assert torch.equal(x, y)
    assert torch.equal(outs[0][0][:, m:], a[:, m:])   # the padding rows are untouched
