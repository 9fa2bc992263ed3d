"""Calls at the limits of what the entry points accept: pivots over the whole
float range, matrices whose factors are exact numbers (so that nothing may be
lost to a reordering), pointers that are not aligned, and waits that run out."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
FLT_EPS = float(np.finfo(np.float32).eps)


@pytest.mark.parametrize("prec,n,bs", [("f32", 128, 16), ("f32", 256, 64), ("f32", 640, 128), ("bf16", 128, 128),
                                       ("fp8", 128, 128), ("f32_bf16x6", 128, 128)])
def test_reciprocal_pivots_over_the_float_range(ctx, dev, prec, n, bs):
    """A diagonal matrix is its own U: the factors hold -1/u_kk, correctly rounded (the quotient in double rounded to
    float), for pivots of every exponent whose reciprocal is finite, subnormal pivots and reciprocals among them."""
    rng = np.random.default_rng(n)
    u = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-127, 128, n)) * rng.choice([-1.0, 1.0], n)
    u[:8] = [1e38, -3e38, 5e-39, -1.1e-38, 2.0 ** 126, 2.0 ** 127, 2.0 ** -126, 2.0 ** -127]
    u = u.astype(np.float32)
    d = dev.put(np.diag(u))
    ctx.gefa_prec(prec, d.data_ptr(), n, n, bs)
    got = dev.get(d)
    want = (-1.0 / u.astype(np.float64)).astype(np.float32)
    assert np.all(np.isfinite(want)) and np.any(np.abs(want) < 2.0 ** -126)
    assert np.array_equal(np.diag(got), want)
    assert np.count_nonzero(got) == n


def test_solution_with_pivots_at_the_ends_of_the_range(ctx, dev):
    """A dominant matrix with a pivot of 1e38 and one of 5e-39 in a whole 128 block: the solution of a right-hand side
    M * ones within 8 n eps (the two rows' own rounding: subnormal numbers near 5e-39 carry 21 bits)."""
    n = 128
    rng = np.random.default_rng(5)
    S = rng.uniform(-0.5, 0.5, (n, n))
    S[np.arange(n), np.arange(n)] = np.abs(S).sum(1) + 1.0
    S[40, 40] = 1e38
    S[9, :], S[:, 9] = 0.0, 0.0
    S[9, 9] = 5e-39
    S = S.astype(np.float32)
    b = S.astype(np.float64).sum(0).astype(np.float32)
    dA, dB = dev.put(S), dev.put(b)
    ctx.gefa(dA.data_ptr(), n, n, 128)
    ctx.gesl(dA.data_ptr(), n, n, dB.data_ptr(), 1)
    assert np.abs(dev.get(dB) - 1.0).max() <= 8 * n * FLT_EPS


@pytest.mark.parametrize("n,kind", [(100, "dev"), (644, "dev"), (1156, "dev"), (644, "calculate")])
def test_pivot_wait_that_runs_out_reports_timeout(ctx, dev, lp, torch_cuda, n, kind):
    """A pivot step's wait that runs out (lp_ctx_test_stall) comes back as LP_E_TIMEOUT; nothing outside the matrix is
    written, ipvt holds rows of the matrix (stale entries in it, here the numbers of padding columns, are not used),
    and the next call gives the oracle's pivots."""
    rng = np.random.default_rng(n)
    A = rng.uniform(-0.5, 0.5, (n, n)).astype(np.float32)
    A[np.arange(n), rng.permutation(n)] += np.float32(np.sqrt(n))
    want = oracle.gefa_pvt(A)[1]
    ctx.test_stall(lp.LP_STALL_PIVOT)
    if kind == "calculate":
        with pytest.raises(lp.LpError) as e:
            ctx.calculate_pvt(A.copy(), A.sum(0))
        assert e.value.status == lp.LP_E_TIMEOUT
        assert np.array_equal(ctx.calculate_pvt(A.copy(), A.sum(0))[1], want)
        return
    pad = 64
    store = np.full((n + 2, n + pad), 7.0, np.float32)
    store[1:n + 1, :n] = A
    d = dev.put(store)
    piv = torch_cuda.full((n,), n + 1, dtype=torch_cuda.int32, device="cuda")
    piv += torch_cuda.arange(n, dtype=torch_cuda.int32, device="cuda") % (pad - 2)
    torch_cuda.cuda.synchronize()
    with pytest.raises(lp.LpError) as e:
        ctx.gefa_pvt(d.data_ptr() + 4 * (n + pad), n, n + pad, piv.data_ptr())
    assert e.value.status == lp.LP_E_TIMEOUT and "bounded wait" in str(e.value)
    got, p = dev.get(d), piv.cpu().numpy()
    assert np.all(got[0] == 7.0) and np.all(got[n + 1] == 7.0) and np.all(got[1:n + 1, n:] == 7.0)
    assert np.all((p >= np.arange(n)) & (p < n))
    d = dev.put(store)
    ctx.gefa_pvt(d.data_ptr() + 4 * (n + pad), n, n + pad, piv.data_ptr())
    ctx.sync()
    assert np.array_equal(piv.cpu().numpy(), want)


@pytest.mark.parametrize("off", [1, 2, 3])
@pytest.mark.parametrize("bs", [64, 128, 256, 512])
def test_lu_block_at_an_unaligned_address(ctx, dev, lp, bs, off):
    """lp_lu_block_dev takes blocks of up to 128 at any float's address (the exact factors), and refuses larger ones
    before anything is launched."""
    A = oracle.gen_reference(bs)[0]
    store = np.full(bs * bs + 8, 7.0, np.float32)
    store[off:off + bs * bs] = A.ravel()
    d = dev.put(store)
    if bs > 128:
        with pytest.raises(lp.LpError) as e:
            ctx.lu_block(d.data_ptr() + 4 * off, bs, bs)
        assert e.value.status == lp.LP_E_INVALID
        assert np.array_equal(dev.get(d), store)
        return
    ctx.lu_block(d.data_ptr() + 4 * off, bs, bs)
    store[off:off + bs * bs] = oracle.gefa_nopvt(A).ravel()
    assert np.array_equal(dev.get(d), store)


@pytest.mark.parametrize("api,n,nrhs", [("gesl_f64", 20, 1), ("gesl_f64", 200, 17), ("calculate", 256, 1), ("gmres", 256, 1)])
def test_fp64_substitution_wait_that_runs_out_reports_timeout(ctx, dev, lp, api, n, nrhs):
    """A barrier of the FP64 substitution that runs out (lp_ctx_test_stall) comes back as LP_E_TIMEOUT: from the calls
    that wait, and for lp_gesl_f64_dev from the next lp_ctx_sync, with NaN in the first group of 16 right-hand sides
    and the second group's solutions as they should be.  The next call succeeds."""
    A = oracle.gen_reference(n)[0]
    LU = oracle.gefa_nopvt(A.astype(np.float64))
    B = np.tile(A.astype(np.float64).sum(0), (nrhs, 1))

    def run():
        if api == "gesl_f64":
            dLU, dB = dev.put(LU), dev.put(B)
            ctx.gesl_f64(dLU.data_ptr(), n, n, dB.data_ptr(), nrhs)
            try:
                ctx.sync()
            finally:
                x = dB.cpu().numpy()
                assert np.all(np.abs(x[16:] - 1.0) < 1e-9)
                assert np.all(np.isnan(x[:16])) or np.all(np.abs(x - 1.0) < 1e-9)
            return x
        if api == "calculate":
            b = B[0].copy()
            ctx.calculate_f64(A.astype(np.float64), b, 128)
            return b
        dA, dLU, db = dev.put(A), dev.put(LU.astype(np.float32)), dev.put(B[0])
        dx = dev.empty(n, np.float64)
        ctx.gmres(dA.data_ptr(), n, dLU.data_ptr(), n, db.data_ptr(), dx.data_ptr(), tol=1e-12)
        return dev.get(dx)

    ctx.test_stall(lp.LP_STALL_GESL64)
    with pytest.raises(lp.LpError) as e:
        run()
    assert e.value.status == lp.LP_E_TIMEOUT and "bounded wait" in str(e.value)
    assert np.abs(run() - 1.0).max() < 1e-9


def whole_number_factors(n, w, e, seed):
    """(L, U) with small whole numbers: unit diagonals, -e throughout the strict triangles of the w-wide diagonal
    blocks, some +-1 outside them.  L U is a matrix of small whole numbers, and so is every intermediate value of the
    recurrences, which therefore give the factors exactly; the inverses of the blocks' triangles grow like (1 + e)^w."""
    rng = np.random.default_rng(seed)
    inside = (np.arange(n)[:, None] // w) == (np.arange(n)[None, :] // w)
    some = np.where(rng.random((n, n)) < 0.02, rng.choice([-1.0, 1.0], (n, n)), 0.0)
    F = np.where(inside, -float(e), some)
    return np.tril(F, -1) + np.eye(n), np.triu(F, 1) + np.eye(n)


def encoded(L, U):
    """The reference's storage (transposed, multipliers negated, -1/u_kk on the diagonal)."""
    return np.triu(-L.T, 1) + np.tril(U.T, -1) - np.diag(1.0 / np.diag(U))


@pytest.mark.parametrize("api,n,bs", [("gefa", 128, 16), ("gefa", 512, 128), ("gefa", 1280, 256), ("gefa", 720, 16),
                                      ("lu_block", 256, 256), ("lu_block", 512, 512), ("calculate", 1280, 64)])
def test_factors_of_whole_numbers_are_exact(ctx, dev, lp, api, n, bs):
    """Top and left lose nothing that the recurrences keep, whatever the condition of the diagonal blocks' triangles."""
    L, U = whole_number_factors(n, 32, 1, n)
    S = np.ascontiguousarray((L @ U).T).astype(np.float32)
    assert np.array_equal(S.astype(np.float64), (L @ U).T)
    if api == "calculate":
        pa, pb = lp.Pinned((n, n)), lp.Pinned((n,))
        pa.array[...], pb.array[...] = S, S.sum(0)
        ctx.calculate(pa.array, pb.array, bs)
        got = pa.array
    else:
        d = dev.put(S)
        if api == "gefa":
            ctx.gefa(d.data_ptr(), n, n, bs)
        else:
            ctx.lu_block(d.data_ptr(), n, bs)
        got = dev.get(d)
    assert np.array_equal(got, encoded(L, U).astype(np.float32))


@pytest.mark.parametrize("n,nrhs,pad", [(64, 1, 0), (100, 9, 1), (200, 2, 0), (1000, 17, 0)])
def test_fp64_solution_of_whole_numbers_is_exact(ctx, dev, n, nrhs, pad):
    """The FP64 substitution loses nothing that the recurrences keep: factors of whole numbers whose diagonal blocks'
    triangles have inverses up to 3^63, beyond what a double holds exactly."""
    L, U = whole_number_factors(n, 64, 2, n)
    want = np.random.default_rng(1).integers(-4, 5, (nrhs, n)).astype(np.float64)
    store = np.full((n, n + pad), 7.0)
    store[:, :n] = encoded(L, U)
    d, b = dev.put(store), dev.put(want @ U.T @ L.T)
    ctx.gesl_f64(d.data_ptr(), n, n + pad, b.data_ptr(), nrhs)
    assert np.array_equal(dev.get(b), want)


@pytest.mark.parametrize("kind,n,need_mb", [("f32", 9216, 38), ("calculate", 9216, 34), ("bf16", 4096, 114)])
def test_factors_do_not_depend_on_free_memory(lp, dev, torch_cuda, kind, n, need_mb):
    """The inner block follows from the order and the precision: with little memory left beside what it takes (its
    operands: need_mb), a context that has allocated nothing yet gives the bits of one with room.  With less than that,
    the call still succeeds, in the caller's block: the factors agree to the operands' rounding."""
    torch = torch_cuda
    bs, mb = 128, 1 << 20
    g = torch.Generator(device="cuda").manual_seed(n)
    S = torch.rand(n, n, generator=g, device="cuda").sub_(0.5)
    S.diagonal().copy_(S.abs().sum(1) + 1.0)
    torch.cuda.synchronize()
    host = lp.Pinned((n, n)) if kind == "calculate" else None

    def factors(c, M):
        if host is not None:
            host.array[...] = M.cpu().numpy()
            b = lp.Pinned((n,))
            b.array[...] = 1.0
            c.calculate(host.array, b.array, bs)
            return host.array.copy()
        c.gefa_prec(kind, M.data_ptr(), n, n, bs)
        c.sync()
        return M

    with lp.Context(0) as c:
        want = factors(c, S.clone())
    matrix_mb = n * n * 4 // mb + 4 if host is not None else 0  # lp_calculate's own copy
    for work, left_mb in zip((S.clone(), S.clone()), (2 * need_mb, need_mb // 2)):
        with lp.Context(0) as c:
            torch.cuda.empty_cache()
            hog = torch.empty(torch.cuda.mem_get_info()[0] - (left_mb + matrix_mb) * mb, dtype=torch.uint8, device="cuda")
            try:
                got = factors(c, work)
            finally:
                del hog
                torch.cuda.empty_cache()
        same = np.array_equal(got, want) if host is not None else torch.equal(got, want)
        if left_mb >= need_mb:
            assert same
        else:
            a, b = (torch.as_tensor(x).cuda().double() for x in (got, want))
            assert float((a - b).abs().max() / b.abs().max()) < (2e-3 if kind == "bf16" else 256 * FLT_EPS)


def test_stage_profile_of_the_fp32_schedule(ctx, dev):
    """Every stage of the factorization is booked, with its share of the work: top and left (one launch) each b^2 r
    flops per block step, all stages together the 2 n^3 / 3 of the factorization to its lower-order terms; a stage's
    time is at most the span of its launches, which parts running beside each other do not add to."""
    n = 2048
    d = dev.put(oracle.gen_baseline(n, seed=1, margin=1.0)[0])
    ctx.set_profiling(True)
    try:
        ctx.read_profile(reset=True)
        ctx.gefa(d.data_ptr(), n, n, 128)
        p = ctx.read_profile(reset=False)
        events = ctx.read_timeline()
        ctx.read_profile(reset=True)
    finally:
        ctx.set_profiling(False)
    assert p["left"]["s"] > 0.0 and p["top"]["s"] > 0.0
    assert p["left"]["flops"] == p["top"]["flops"] == sum(128.0 ** 2 * r for r in range(128, n, 128))
    total = sum(p[s]["flops"] for s in ("lu", "top", "left", "inner"))
    assert abs(total - 2 * n ** 3 / 3) < 0.01 * total
    for s in ("lu", "top", "left", "inner"):
        t = [(e[2], e[3]) for e in events if e[0] == s]
        assert len(t) == p[s]["calls"] and 0.0 < p[s]["s"] <= (max(b for _, b in t) - min(a for a, _ in t)) * (1 + 1e-6)
