"""The work that is timed: factorizations, solves and batches through the public entry points.

A program that uses this library keeps one Context (streams, workspaces), holds its matrices on
the GPU (or, for the host entry point, in page-locked memory) and calls factor and solve.  Matrices
are the LINPACK workload: entries uniform in [-0.5, 0.5), each storage row's diagonal its absolute
row sum + 1, right-hand side M * ones.  The pivoting path gets systems whose large entries are out of
order: uniform entries plus sqrt(n) at the places of a random permutation, so nearly every step exchanges
rows and the solution is still well determined in 32 bits.
Factorizations work in place, so a pass starts from the kept original, copied on the context's stream.
"""
import math

import numpy as np
import torch

from hpcc_fpga_b200 import lpcuda as lp

_CTX = None


def _ctx():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = lp.Context(0)
    return _CTX


def listed():
    return [
        # the smallest whole solve: a 512 x 512 system, where launches and the pivot chain are all there is
        {"name": "f32_n512", "kind": "lu", "precision": "f32", "n": 512, "bs": 128, "nrhs": 1},
        # an ordinary system, block 256 (the middle of the reference's range of blocks)
        {"name": "f32_n4096", "kind": "lu", "precision": "f32", "n": 4096, "bs": 256, "nrhs": 1},
        # the headline benchmark: n = 32768, block 512
        {"name": "f32_n32768", "kind": "lu", "precision": "f32", "n": 32768, "bs": 512, "nrhs": 1},
        # the same system in BF16 with FP64 refinement, the block that the benchmark takes there
        {"name": "bf16_n32768", "kind": "lu_ir", "precision": "bf16", "n": 32768, "bs": 1024, "nrhs": 1},
        # E4M3 with FP64 refinement on a middle-sized system, a few right-hand sides
        {"name": "fp8_n12288", "kind": "lu_ir", "precision": "fp8", "n": 12288, "bs": 512, "nrhs": 3},
        # FP32 emulated on the tensor cores
        {"name": "x6_n8192", "kind": "lu", "precision": "f32_bf16x6", "n": 8192, "bs": 512, "nrhs": 1},
        # the double build
        {"name": "f64_n6144", "kind": "lu_f64", "n": 6144, "bs": 256, "nrhs": 1},
        # partial pivoting on a size that is no multiple of the panel
        {"name": "pvt_n5000", "kind": "lu_pvt", "n": 5000, "nrhs": 1},
        # the batched workload: 4096 systems, n log-uniform in [32, 1024], 1 to 8 right-hand sides
        {"name": "batch_f32", "kind": "batch", "count": 4096, "lo": 32, "hi": 1024, "rhs_max": 8},
        # the refined batch
        {"name": "batch_bf16_ir", "kind": "batch_ir", "precision": "bf16", "count": 1000, "lo": 32, "hi": 700,
         "rhs_max": 4},
        # solves against resident factors: an odd order, several right-hand sides
        {"name": "solve_n10007_r8", "kind": "solve", "n": 10007, "nrhs": 8},
        # host buffers in, solution out: the copies belong to the call
        {"name": "host_bf16_n8192", "kind": "host", "precision": "bf16", "n": 8192, "bs": 512, "nrhs": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, bs, lo, hi):
    return max(1, int(round(_log(rng, lo, hi) / bs))) * bs


def draw(rng):
    kind = rng.choice(["lu", "lu", "lu_ir", "lu_ir", "lu_f64", "lu_pvt", "batch", "batch_ir", "solve", "host"])
    if kind == "lu":
        p = rng.choice(["f32", "f32", "f32_bf16x6"])
        bs = rng.choice([64, 128, 256, 512] if p == "f32" else [256, 512, 1024])
        return {"kind": kind, "precision": p, "n": _multiple(rng, bs, 512, 16384), "bs": bs, "nrhs": rng.randint(1, 4)}
    if kind == "lu_ir":
        bs = rng.choice([256, 512, 1024])
        return {"kind": kind, "precision": rng.choice(["bf16", "fp8"]), "n": _multiple(rng, bs, 2048, 32768), "bs": bs,
                "nrhs": rng.randint(1, 4)}
    if kind == "lu_f64":
        bs = rng.choice([64, 128, 256])
        return {"kind": kind, "n": _multiple(rng, bs, 512, 8192), "bs": bs, "nrhs": rng.randint(1, 4)}
    if kind == "lu_pvt":
        return {"kind": kind, "n": _multiple(rng, 4, 100, 8192), "nrhs": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 16, 4096), "lo": rng.randint(8, 100), "hi": _log(rng, 100, 1024),
                "rhs_max": rng.randint(1, 16)}
    if kind == "batch_ir":
        return {"kind": kind, "precision": rng.choice(["f32", "bf16"]), "count": _log(rng, 16, 1000),
                "lo": rng.randint(8, 100), "hi": _log(rng, 100, 1024), "rhs_max": rng.randint(1, 8)}
    if kind == "solve":
        return {"kind": kind, "n": _log(rng, 100, 32768), "nrhs": _log(rng, 1, 32)}
    bs = rng.choice([128, 256, 512])
    return {"kind": kind, "precision": rng.choice(["bf16", "fp8"]), "n": _multiple(rng, bs, 1024, 8192), "bs": bs,
            "nrhs": rng.randint(1, 2)}


# ---- inputs ---------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _dominant(S):
    """The diagonal of a square matrix set to its absolute row sums + 1 (of the other entries)."""
    S.diagonal().zero_()
    S.diagonal().copy_(S.abs().sum(1) + 1.0)
    return S


def _matrix(case, seed):
    """(S, right-hand sides) of one system: b = M * ones (M = S^T), more of them uniform."""
    n, g = case["n"], _gen(seed)
    dt = torch.float64 if case["kind"] == "lu_f64" else torch.float32
    S = torch.rand(n, n, generator=g, device="cuda", dtype=dt)
    S.sub_(0.5)
    if case["kind"] == "lu_pvt":
        S[torch.arange(n, device="cuda"), torch.randperm(n, generator=g, device="cuda")] += math.sqrt(n)
    else:
        _dominant(S)
    B = torch.rand(case["nrhs"], n, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0)
    B[0] = S.sum(0, dtype=torch.float64)
    return S, B


def _factors(case, seed):
    """Factors in the encoding, as those of a dominant matrix look: u_kk near n / 4."""
    n, g = case["n"], _gen(seed)
    lda = (n + 3) // 4 * 4
    E = torch.zeros(n, lda, device="cuda")
    S = torch.rand(n, n, generator=g, device="cuda").sub_(0.5)
    u = n / 4 * (1.0 + 0.02 * (torch.rand(n, generator=g, device="cuda") - 0.5)) + 1.0
    E[:, :n] = S.tril(-1) + S.triu(1) / u[:, None] - torch.diag(1.0 / u)
    B = torch.rand(case["nrhs"], n, generator=g, device="cuda").mul_(2.0).sub_(1.0)
    return E, B


def _batch(case, seed):
    """Packed systems: descriptors, the matrices and the right-hand sides; the sizes belong to the case."""
    sizes = np.random.default_rng([case["count"], case["lo"], case["hi"], case["rhs_max"]])
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    ns = np.clip(np.rint(np.exp(sizes.uniform(lo, hi, case["count"]))), case["lo"], case["hi"]).astype(int)
    rs = sizes.integers(1, case["rhs_max"] + 1, case["count"])
    systems, a_off, b_off = [], 0, 0
    for n, r in zip(ns.tolist(), rs.tolist()):
        ld = (n + 3) // 4 * 4
        systems.append(lp.LpSystem(n, r, ld, ld, a_off, b_off))
        a_off += n * ld
        b_off += r * ld
    g = _gen(seed)
    A = torch.rand(a_off, generator=g, device="cuda").sub_(0.5)
    B = torch.rand(b_off, generator=g, device="cuda").mul_(2.0).sub_(1.0)
    for s in systems:
        _dominant(A[s.a_off:s.a_off + s.n * s.lda].view(s.n, s.lda)[:, :s.n])
    return systems, A, B


def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    s = {"case": case, "ctx": ctx, "stream": torch.cuda.ExternalStream(ctx.stream)}
    if kind in ("batch", "batch_ir"):
        s["systems"], s["A0"], B = _batch(case, seed)
        s["B"] = B if kind == "batch" else B.double()
        s["A"], s["X"] = torch.empty_like(s["A0"]), torch.zeros_like(s["B"])
    elif kind == "solve":
        s["A"], s["B"] = _factors(case, seed)
        s["X"] = torch.empty_like(s["B"])
    elif kind == "host":
        S, B = _matrix(case, seed)
        s["pins"] = lp.Pinned(tuple(S.shape), np.float32), lp.Pinned(tuple(B.shape), np.float64)
        for pin, t in zip(s["pins"], (S, B)):
            pin.array[...] = t.cpu().numpy()
    else:
        s["A0"], B = _matrix(case, seed)
        s["B"] = B.float() if kind in ("lu", "lu_pvt") else B
        s["A"], s["X"] = torch.empty_like(s["A0"]), torch.empty_like(s["B"])
        if kind == "lu_pvt":
            s["ipvt"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------------------
def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, n, nrhs = case["kind"], case.get("n"), case.get("nrhs")
    if kind == "host":
        return ctx.solve_host(s["pins"][0].array, s["pins"][1].array, case["bs"], case["precision"], 50)[0]
    A, B, X = s["A"], s["B"], s["X"]
    with torch.cuda.stream(s["stream"]):  # the context's stream: in order with the calls below
        if kind != "solve":
            A.copy_(s["A0"], non_blocking=True)
        if kind not in ("lu_ir", "batch_ir"):
            X.copy_(B, non_blocking=True)
    if kind == "lu":
        ctx.gefa_prec(case["precision"], A.data_ptr(), n, n, case["bs"])
        ctx.gesl(A.data_ptr(), n, n, X.data_ptr(), nrhs)
    elif kind == "lu_ir":
        ctx.gefa_prec(case["precision"], A.data_ptr(), n, n, case["bs"])
        ctx.refine(s["A0"].data_ptr(), n, A.data_ptr(), n, B.data_ptr(), X.data_ptr(), nrhs)
    elif kind == "lu_f64":
        ctx.gefa_f64(A.data_ptr(), n, n, case["bs"])
        ctx.gesl_f64(A.data_ptr(), n, n, X.data_ptr(), nrhs)
    elif kind == "lu_pvt":
        ctx.gefa_pvt(A.data_ptr(), n, n, s["ipvt"].data_ptr())
        ctx.gesl_pvt(A.data_ptr(), n, n, s["ipvt"].data_ptr(), X.data_ptr(), nrhs)
        return {"factors": A, "pivots": s["ipvt"], "x": X}
    elif kind == "batch":
        ctx.batch_solve(s["systems"], A.data_ptr(), X.data_ptr())
    elif kind == "batch_ir":
        ctx.batch_solve_ir(s["systems"], A.data_ptr(), B.data_ptr(), X.data_ptr(), case["precision"])
    else:
        ctx.gesl(A.data_ptr(), n, A.shape[1], X.data_ptr(), nrhs)
        return X
    return {"factors": A, "x": X}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "batch_ir"):
        # sums over the log-uniform sizes: E[n^p] = (hi^p - lo^p) / (p ln(hi / lo))
        lo, hi, r = case["lo"], max(case["hi"], case["lo"] + 1), (1 + case["rhs_max"]) / 2
        e2, e3 = ((hi ** p - lo ** p) / (p * math.log(hi / lo)) for p in (2, 3))
        return {"bytes": case["count"] * 8.0 * e2, "flops": case["count"] * (2.0 * e3 / 3.0 + 2.0 * r * e2)}
    n, r = case["n"], case["nrhs"]
    solve = 2.0 * r * n * n
    if kind == "solve":
        return {"bytes": 4.0 * n * n + 8.0 * r * n, "flops": solve}
    e = 8.0 if kind == "lu_f64" else 4.0
    if kind == "host":
        return {"bytes": e * n * n + 16.0 * r * n, "flops": 2.0 * n ** 3 / 3.0 + solve}
    return {"bytes": 2.0 * e * n * n + 16.0 * r * n, "flops": 2.0 * n ** 3 / 3.0 + solve}


# ---- the same in 64 bits, by torch ----------------------------------------------------------
def _encoded(M):
    """LU of M without pivoting in the library's encoding (storage is M transposed)."""
    E = torch.linalg.lu_factor_ex(M, pivot=False)[0].t().contiguous()
    u = E.diagonal().clone()
    E -= 2.0 * E.triu(1)
    E.diagonal().copy_(-1.0 / u)
    return E


def _substituted(E, B):
    """Solutions (rows) for the right-hand sides B (rows) with encoded factors E, in 64 bits."""
    E = E.double()
    y = torch.linalg.solve_triangular(-E.triu(1).t(), B.double().t(), upper=False, unitriangular=True)
    U = E.tril(-1).t() + torch.diag(-1.0 / E.diagonal())
    return torch.linalg.solve_triangular(U, y, upper=True).t().contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "batch_ir"):
        systems, A, B = _batch(case, seed)
        X = B.double()
        if kind == "batch_ir":  # the padding of X is not written there
            X.zero_()
        A = A.double()
        for s in systems:
            a = A[s.a_off:s.a_off + s.n * s.lda].view(s.n, s.lda)[:, :s.n]
            b = B[s.b_off:s.b_off + s.nrhs * s.ldb].view(s.nrhs, s.ldb)[:, :s.n]
            a.copy_(_encoded(a.t()))
            X[s.b_off:s.b_off + s.nrhs * s.ldb].view(s.nrhs, s.ldb)[:, :s.n] = _substituted(a, b)
        return {"factors": A, "x": X}
    if kind == "solve":
        E, B = _factors(case, seed)
        return _substituted(E[:, :case["n"]], B)
    S, B = _matrix(case, seed)
    if kind in ("lu", "lu_pvt"):
        B = B.float()  # the path takes right-hand sides in 32 bits
    if kind == "lu_pvt":  # the multipliers stand in the order of their steps' exchanges: the solution is compared
        return {"factors": None, "pivots": None, "x": torch.linalg.solve(S.double().t(), B.double().t()).t().contiguous()}
    E = _encoded(S.double().t())
    x = _substituted(E, B)
    return x if kind == "host" else {"factors": E, "x": x}
