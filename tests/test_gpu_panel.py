"""The FP32 factorization at the edges of its inner blocking: 128-wide inner
blocks whatever block the caller names, a ragged last block in pieces of 64,
32 and 16, strips of 32 / 64 beside a block, and trailing updates on each side
of the tile forms' borders.  Bound as for the whole factorization elsewhere:
|got - want| <= 256 eps max(1, |want|) against the oracle's factors."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
FLT_EPS = float(np.finfo(np.float32).eps)


@pytest.mark.parametrize("n,bs,pad", [(16, 16, 0), (112, 16, 0), (144, 16, 4), (208, 16, 0), (224, 32, 0), (320, 64, 8),
                                      (384, 128, 0), (1088, 64, 0), (1280, 256, 0), (1536, 512, 4), (2304, 256, 0)])
def test_gefa_blocking_edges(ctx, dev, n, bs, pad):
    A, _, _, _ = oracle.gen_reference(n)
    store = np.full((n, n + pad), 7.0, np.float32)
    store[:, :n] = A
    d = dev.put(store)
    ctx.gefa(d.data_ptr(), n, n + pad, bs)
    got = dev.get(d)
    assert np.all(got[:, n:] == 7.0)  # the padding is not touched
    want = oracle.gefa_nopvt(A).astype(np.float64)
    err = np.abs(got[:, :n].astype(np.float64) - want) / np.maximum(1.0, np.abs(want))
    assert err.max() < 256 * FLT_EPS


@pytest.mark.parametrize("n", [496, 512, 528, 4080, 4096, 4240, 9216])
def test_gefa_block_of_the_order(ctx, dev, n):
    """Orders on each side of the inner block's borders, last blocks that are no multiple of it, a caller's block of
    16: max |L U - A| (the reference's storage: -1/u_kk on the diagonal, negated multipliers right of it, U^T below)
    within 4 n eps max|L| max|U| on 64 sampled rows, in FP64."""
    A, _, _, _ = oracle.gen_reference(n)
    d = dev.put(A)
    ctx.gefa(d.data_ptr(), n, n, 16)
    F = dev.get(d).astype(np.float64)
    M = np.triu(-F, 1) + np.eye(n)           # right of the diagonal: multipliers, unit diagonal
    U = np.tril(F, -1) + np.diag(-1.0 / np.diag(F))
    rows = np.unique(np.linspace(0, n - 1, 64).astype(int))
    err = np.abs(U[rows] @ M - A[rows]).max()
    assert err <= 4 * n * FLT_EPS * np.abs(U).max() * np.abs(M).max()


@pytest.mark.parametrize("prec,tol", [("bf16", 2e-3), ("fp8", 2e-2), ("f32_bf16x6", None)])
@pytest.mark.parametrize("n,pad", [(128, 0), (896, 0), (1152, 4), (1920, 0), (2176, 0), (4224, 0)])
def test_mixed_ragged_blocks(ctx, dev, prec, tol, n, pad):
    """Tensor-core schedules whose order is no multiple of their inner block (one short block, a last block of 128
    or 896): the bounds of the factors elsewhere (a few operand roundings; the emulated FP32 form 8 n eps)."""
    A, _, _ = oracle.gen_baseline(n, seed=42, margin=1.0)
    store = np.full((n, n + pad), 7.0, np.float32)
    store[:, :n] = A
    d = dev.put(store)
    ctx.gefa_prec(prec, d.data_ptr(), n, n + pad, 128)
    got = dev.get(d)
    assert np.all(got[:, n:] == 7.0)
    want = oracle.gefa_nopvt(A).astype(np.float64)
    rel = np.abs(got[:, :n].astype(np.float64) - want).max() / np.abs(want).max()
    assert rel < (tol or 8 * n * FLT_EPS)


@pytest.mark.parametrize("n,bs", [(1088, 64), (2096, 16), (1536, 128)])
def test_streamed_ragged_blocks(ctx, lp, n, bs):
    """Page-locked buffers (factored in row slabs while copied in) give the pageable path's bits."""
    A, b, _, _ = oracle.gen_reference(n)
    A1, b1 = A.copy(), b.copy()
    ctx.calculate(A1, b1, bs)
    pa, pb = lp.Pinned((n, n)), lp.Pinned((n,))
    pa.array[...], pb.array[...] = A, b
    ctx.calculate(pa.array, pb.array, bs)
    assert np.array_equal(pa.array, A1) and np.array_equal(pb.array, b1)


@pytest.mark.parametrize("n,nrhs", [(132, 1), (160, 2), (388, 1), (644, 3), (1156, 1)])
def test_pivoting_panel_edges(ctx, dev, torch_cuda, n, nrhs):
    """Panels whose last rows or columns do not fill a CTA's slice (its rows are held by fours), on matrices whose
    every step exchanges rows: the oracle's pivots, and solutions within 8 n eps max|x| of the FP64 ones (the matrix
    is a scaled permutation plus a perturbation of a third of its norm, so its condition is small)."""
    rng = np.random.default_rng(n)
    A = rng.uniform(-0.5, 0.5, (n, n)).astype(np.float32)
    A[np.arange(n), rng.permutation(n)] += np.float32(np.sqrt(n))
    B = rng.uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32)
    dA, dB = dev.put(A), dev.put(B)
    piv = torch_cuda.empty(n, dtype=torch_cuda.int32, device="cuda")
    ctx.gefa_pvt(dA.data_ptr(), n, n, piv.data_ptr())
    ctx.gesl_pvt(dA.data_ptr(), n, n, piv.data_ptr(), dB.data_ptr(), nrhs)
    ctx.sync()
    assert np.array_equal(piv.cpu().numpy(), oracle.gefa_pvt(A)[1])
    want = np.linalg.solve(A.T.astype(np.float64), B.T.astype(np.float64)).T
    assert np.abs(dev.get(dB) - want).max() <= 8 * n * FLT_EPS * np.abs(want).max()


@pytest.mark.parametrize("n,nrhs,pad", [(1, 1, 0), (31, 2, 1), (63, 1, 0), (64, 16, 0), (65, 17, 1), (200, 3, 0),
                                        (1000, 1, 0), (4801, 2, 3)])
def test_gesl_f64_edges(ctx, dev, n, nrhs, pad):
    """The FP64 substitution for orders that are no multiple of its 64 blocks, one to several groups of 16 right-hand
    sides, padded rows: against numpy's triangular products with the same bound as for the factored systems,
    1e3 n eps max(1, |x|)."""
    rng = np.random.default_rng(n)
    E = np.full((n, n + pad), 3.0)
    E[:, :n] = rng.uniform(-0.5, 0.5, (n, n))
    u = n / 4 * rng.uniform(0.99, 1.01, n) + 1.0
    E[:, :n] = np.tril(E[:, :n], -1) + np.triu(E[:, :n], 1) / u[:, None] - np.diag(1.0 / u)
    M = (np.eye(n) - np.triu(E[:, :n], 1)).T @ (np.tril(E[:, :n], -1) + np.diag(u)).T  # L U of the encoding
    want = rng.uniform(-1.0, 1.0, (nrhs, n))
    dE, dB = dev.put(E), dev.put(np.ascontiguousarray(want @ M.T))
    ctx.gesl_f64(dE.data_ptr(), n, n + pad, dB.data_ptr(), nrhs)
    ctx.sync()
    assert np.abs(dev.get(dB) - want).max() <= 1e3 * n * np.finfo(np.float64).eps


@pytest.mark.parametrize("sizes,pad", [([129, 160, 161, 255], 0), ([257, 384, 385, 530], 3), ([641, 1024], 0),
                                       ([31, 33, 64, 95, 127, 128], 1)])
def test_batch_tile_edges(ctx, dev, lp, sizes, pad):
    """Batched systems at the edges of the outer blocks (128), inner panels (32) and unknowns per thread, with rows
    that allow 16-byte copies and rows that do not, 1 to 16 right-hand sides: factors within 256 eps max(1, |want|)
    of the oracle's, solutions within 8 n eps max|x| of the FP64 ones (diagonally dominant: condition below 8)."""
    rhs = [1, 2, 5, 8, 9, 16]
    systems, mats, a_off, b_off = [], [], 0, 0
    for k, n in enumerate(sizes):
        lda = (n + 3) // 4 * 4 + pad
        systems.append(lp.LpSystem(n, rhs[k % 6], lda, n, a_off, b_off))
        mats.append(oracle.gen_reference(n)[0])
        a_off += (n * lda + 3) // 4 * 4
        b_off += rhs[k % 6] * n
    A, B = np.zeros(a_off, np.float32), np.random.default_rng(len(sizes)).uniform(-1, 1, b_off).astype(np.float32)
    for s, m in zip(systems, mats):
        A[s.a_off:s.a_off + s.n * s.lda].reshape(s.n, s.lda)[:, :s.n] = m
    dA, dB = dev.put(A), dev.put(B)
    ctx.batch_solve(systems, dA.data_ptr(), dB.data_ptr())
    gotA, gotB = dev.get(dA), dev.get(dB)
    for s, m in zip(systems, mats):
        f = gotA[s.a_off:s.a_off + s.n * s.lda].reshape(s.n, s.lda)[:, :s.n].astype(np.float64)
        want = oracle.gefa_nopvt(m).astype(np.float64)
        assert (np.abs(f - want) / np.maximum(1.0, np.abs(want))).max() < 256 * FLT_EPS, s.n
        b = B[s.b_off:s.b_off + s.nrhs * s.n].reshape(s.nrhs, s.n).astype(np.float64)
        x = np.linalg.solve(m.T.astype(np.float64), b.T).T
        got = gotB[s.b_off:s.b_off + s.nrhs * s.n].reshape(s.nrhs, s.n)
        assert np.abs(got - x).max() <= 8 * s.n * FLT_EPS * np.abs(x).max(), s.n


@pytest.mark.parametrize("n,nrhs", [(1, 1), (127, 5), (128, 8), (129, 9), (257, 3), (1000, 6), (4229, 8), (4229, 24)])
def test_gesl_rhs_forms(ctx, dev, n, nrhs):
    """The FP32 sweeps' forms for 1, 4, 8 and 16 right-hand sides on whole and ragged tiles, without and with chunk
    items (tile 33 on): |x - want| <= 8 n eps max|x| on encoded factors of a dominant matrix."""
    rng = np.random.default_rng(n + nrhs)
    lda = (n + 3) // 4 * 4
    u = n / 4 * rng.uniform(0.99, 1.01, n) + 1.0
    S = rng.uniform(-0.5, 0.5, (n, n))
    E = np.zeros((n, lda), np.float32)
    E[:, :n] = np.tril(S, -1) + np.triu(S, 1) / u[:, None] - np.diag(1.0 / u)
    want = rng.uniform(-1.0, 1.0, (nrhs, n))
    F = E[:, :n].astype(np.float64)
    y = want @ (np.tril(F, -1) - np.diag(1.0 / np.diag(F)))  # U x, U the transposed lower triangle
    B = y @ (np.eye(n) - np.triu(F, 1))                      # L y
    dE, dB = dev.put(E), dev.put(B.astype(np.float32))
    ctx.gesl(dE.data_ptr(), n, lda, dB.data_ptr(), nrhs)
    assert np.abs(dev.get(dB) - want).max() <= 8 * max(n, 16) * FLT_EPS
