"""Performance cases of the TLR Cholesky library, through its public entry points.

Five kinds of work, each one that a program built on the library has it do:

``request``   one log-likelihood evaluation from parameters and observations to
              (status, loglik, logdet, x, band): ``tlr.serve_loglik``, what the serving
              loop and the maximum-likelihood fit call again and again.
``refactor``  restore a compressed covariance matrix, factor it and evaluate the
              log-likelihood: the step that ``bench.py`` times, plus the use of the factor.
``solve``     many right-hand sides with a factor that is kept (prediction at new sites).
``potrf``     Cholesky and inverse of one dense tile (the diagonal tiles, and callers
              that manage their own memory).
``gemm``      one dense tile product C = C - A B^T (the dense band's update).

Sizes, tile sizes, accuracies and rank caps are those of ``bench.py``'s workloads and of
the serving stream (``serving.sample_requests``); the nugget is the driver's default, 0.1.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from hicma_parsec_b200 import tlr

NUGGET = 0.1    # the reference driver's default


def listed():
    return [
        # the reference's own CTest problem (N 2700, tile 270): the smallest request, launches and latency
        dict(name="request-2d-2700", what="request", kind=2, n=2700, nb=270, maxrank=130, acc=1e-8, beta=0.1),
        # an ordinary request of the serving stream, 2D, tile 1350
        dict(name="request-2d-27000", what="request", kind=2, n=27000, nb=1350, maxrank=0, acc=1e-8, beta=0.1),
        # a large request of the stream: generation and factorization with the benchmark's tile and ranks
        dict(name="request-2d-97200", what="request", kind=2, n=97200, nb=2700, maxrank=150, acc=1e-8, beta=0.1),
        # the stream's rough 3D kernel: near tiles do not compress, a wide dense band
        dict(name="request-3d-exp-16000", what="request", kind=4, n=16000, nb=1000, maxrank=0, acc=1e-6, beta=0.1),
        # the stream's smooth 3D kernel, an odd tile size, high accuracy
        dict(name="request-3d-sqexp-19981", what="request", kind=3, n=19981, nb=1537, maxrank=0, acc=1e-8, beta=0.2),
        # the benchmark's workload at 60 x 60 tiles (its 100 x 100 would not fit three times)
        dict(name="refactor-2d-162000", what="refactor", kind=2, n=162000, nb=2700, maxrank=150, acc=1e-8, beta=0.1,
             mixed=False),
        # the benchmark's rough 3D kernel with ranks up to half the tile, at tile 1350 and the band given (the
        # driver's -b): stacked ranks of hundreds
        dict(name="refactor-3d-exp-8100", what="refactor", kind=4, n=8100, nb=1350, maxrank=675, acc=1e-8,
             beta=0.1, band=3, mixed=False),
        # the smooth 3D kernel with ranks up to half the tile, at tile 900
        dict(name="refactor-3d-sqexp-8100", what="refactor", kind=3, n=8100, nb=900, maxrank=450, acc=1e-8,
             beta=0.2, mixed=False),
        # the precision policy on the 2D workload
        dict(name="refactor-2d-mixed-54000", what="refactor", kind=2, n=54000, nb=2700, maxrank=150, acc=1e-8,
             beta=0.1, mixed=True),
        # 64 right-hand sides with a kept factor
        dict(name="solve-2d-40500x64", what="solve", kind=2, n=40500, nb=1350, maxrank=150, acc=1e-8, beta=0.1,
             nrhs=64),
        # one diagonal tile of the benchmark
        dict(name="potrf-2700", what="potrf", n=2700),
        # one dense band update of the benchmark
        dict(name="gemm-2700", what="gemm", m=2700, n=2700, k=2700),
    ]


def draw(rng):
    """One more case of the ranges above: tile sizes 270 to 2700 (any integer), 4 to 20
    tiles a side (2D up to N = 54,000, 3D up to 20,000), the stream's length scales and
    accuracies and rank caps, dense tiles of 200 to 4000."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["request", "request", "request", "refactor", "refactor", "solve", "potrf", "gemm"])
    if what == "potrf":
        return dict(what=what, n=log_int(200, 4000))
    if what == "gemm":
        return dict(what=what, m=log_int(200, 4000), n=log_int(200, 4000), k=log_int(200, 4000))
    kind = 2 if what == "solve" else rng.choice([2, 2, 3, 4])
    nb = log_int(270, 2700)
    nt = rng.randint(4, 20)
    nt = max(4, min(nt, (54000 if kind == 2 else 20000) // nb))
    case = dict(what=what, kind=kind, n=nt * nb, nb=nb, maxrank=0, acc=rng.choice([1e-6, 1e-8, 1e-9]),
                beta=round(rng.uniform(0.05, 0.3), 3))
    if what == "refactor":
        case["mixed"] = kind == 2 and rng.random() < 0.3
    if what == "solve":
        case["nrhs"] = log_int(1, 128)
    return case


def _cap(case):
    return case["maxrank"] or min(case["nb"] // 2 - 1, 200)


def _problem(case, seed):
    return tlr.Problem(kind=case["kind"], beta=case["beta"], noise=NUGGET, seed=seed)


def _generate(ctx, case, prob):
    """Generate, then widen the band over rejected tiles or by the band rule (serving.solve_request),
    or as the case gives it."""
    A = tlr.TLRMatrix(ctx, case["n"], case["nb"], _cap(case), 1)
    info = A.generate(prob, case["acc"])
    if case.get("band"):
        band = max([case["band"]] + [m - n + 1 for m, n in A.rejected_tiles()])
    elif info != 0:
        band = max(2, max(m - n for m, n in A.rejected_tiles()) + 1)
    else:
        band = tlr.parsec_band_size_auto_tuning(A.rank_map(), A.nt, A.nb)
    if band > 1:
        A.band_regenerate(prob, min(band, A.nt))
    return A


def prepare(case, seed):
    what, n = case["what"], case["n"]
    state = dict(case=case)
    if what == "gemm":
        g = torch.Generator(device="cuda").manual_seed(seed)
        m, k = case["m"], case["k"]
        # column-major operands: a torch tensor of shape (cols, rows)
        state["A"] = torch.randn(k, m, dtype=torch.float64, device="cuda", generator=g)
        state["B"] = torch.randn(k, n, dtype=torch.float64, device="cuda", generator=g)
        state["C0"] = torch.randn(n, m, dtype=torch.float64, device="cuda", generator=g)
        state["C"] = torch.empty_like(state["C0"])
        return state
    ctx = state["ctx"] = tlr.Context(0)
    if what == "potrf":
        state["A0"] = torch.from_numpy(_covariance_tile(n, seed)).cuda()
        state["A"] = torch.empty_like(state["A0"])
        state["X"] = torch.empty_like(state["A0"])
        state["info"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        return state
    rng = np.random.default_rng(seed)
    state["prob"] = _problem(case, seed)
    if what == "request":
        state["y"] = rng.standard_normal(n)
        return state
    A = _generate(ctx, case, state["prob"])
    if what == "solve":
        A.potrf(case["acc"])
        state["L"] = A
        state["B"] = np.asfortranarray(rng.standard_normal((case["nrhs"], n)).T)
        return state
    if case["mixed"]:
        ctx.set_precision(tlr.PREC_MIXED)
    state["A0"], state["y"] = A, rng.standard_normal(n)
    # the working copy is created at the generation band and adopts the source's
    state["A"] = tlr.TLRMatrix(ctx, n, case["nb"], _cap(case), 1)
    state["A"].copy_from(A)
    return state


def run(state):
    case = state["case"]
    what = case["what"]
    if what == "request":
        return tlr.serve_loglik(state["ctx"], state["prob"], case["n"], case["nb"], case["acc"], state["y"],
                                case["maxrank"])
    if what == "refactor":
        A = state["A"]
        A.copy_from(state["A0"])
        info = A.potrf(case["acc"])
        return (info, *A.loglik(state["y"]))
    if what == "solve":
        return state["L"].solve(state["B"])
    lib, stream = tlr.load_library(), torch.cuda.current_stream()
    if what == "potrf":
        n, A, X, info = case["n"], state["A"], state["X"], state["info"]
        A.copy_(state["A0"])
        info.zero_()
        stream.synchronize()    # the library works on the context's stream
        rc = lib.hicma_tlr_k_potrf(state["ctx"].h, n, A.data_ptr(), n, X.data_ptr(), info.data_ptr(), 0)
        if rc != 0:
            raise tlr.TLRError(rc, "hicma_tlr_k_potrf", tlr.last_error())
        return A, X, info
    m, n, k, C = case["m"], case["n"], case["k"], state["C"]
    C.copy_(state["C0"])
    rc = lib.hicma_tlr_k_dgemm(0, 1, m, n, k, -1.0, state["A"].data_ptr(), m, state["B"].data_ptr(), n, 1.0,
                               C.data_ptr(), m, ctypes.c_void_p(stream.cuda_stream))
    if rc != 0:
        raise tlr.TLRError(rc, "hicma_tlr_k_dgemm", tlr.last_error())
    return C


# Rank of a typical off-band tile by kernel, for the work estimate (bench.py's workloads and
# the stream, at e = 1e-8).
_RANK = {2: 22, 3: 90, 4: 250}


def work(case):
    """Bytes: the inputs read once and the outputs written once.  Operations: of the
    factorization's own algorithm at the typical rank (two thin QRs, products and the
    core of every update), or of the dense product."""
    what, n = case["what"], case["n"]
    if what == "gemm":
        m, k = case["m"], case["k"]
        return {"bytes": 8.0 * (m * k + k * n + 2 * m * n), "flops": 2.0 * m * n * k}
    if what == "potrf":
        return {"bytes": 8.0 * 2 * n * n, "flops": 2.0 * n ** 3 / 3}
    nb = case["nb"]
    nt = n // nb
    r = min(_RANK[case["kind"]], _cap(case), nb // 3)
    matrix = 8.0 * (nt * nb * nb / 2 + nt * (nt - 1) / 2 * 2 * nb * r)
    if what == "solve":
        q = case["nrhs"]
        return {"bytes": matrix + 16.0 * n * q, "flops": 4.0 * q * (nt * nb * nb / 2 + nt * (nt - 1) / 2 * 2 * nb * r)}
    pairs, triples = nt * (nt - 1) / 2, nt * (nt - 1) * (nt - 2) / 6
    flops = nt * nb ** 3 / 3 + pairs * (nb * nb * r + nb * nb * r + 2 * nb * r * r)
    flops += triples * (4 * nb * r * r + 2 * 2 * nb * (2 * r) ** 2 + 2 * 2 * nb * 2 * r * r + 20 * r ** 3)
    if what == "request":   # the covariance is sampled with about 2 r columns, twice
        flops += pairs * 8 * nb * nb * r
        return {"bytes": 16.0 * n + matrix, "flops": flops}
    return {"bytes": 2 * matrix + 16.0 * n, "flops": flops}


# ---------------------------------------------------------------- 64-bit values ----
def _mix(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _points(ndim, n, seed):
    """The problem's points as the library documents them: a jittered grid of the unit square
    or cube in Morton order, the first n kept."""
    side = round(n ** (1.0 / ndim))
    side += side ** ndim < n
    idx = np.arange(side ** ndim, dtype=np.uint64)
    with np.errstate(over="ignore"):
        base = _mix(np.array([seed], dtype=np.uint64))[0]
        code, xs, cell = np.zeros_like(idx), [], idx
        for a in range(ndim):
            z = _mix(base + idx * np.uint64(ndim) + np.uint64(a))
            u = (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
            x = (((cell % np.uint64(side)).astype(np.float64) + 0.1) + 0.8 * u) / side
            cell = cell // np.uint64(side)
            xs.append(x)
            q = np.clip(np.floor(x * 2097152.0), 0, 2097151).astype(np.uint64)
            for b in range(21):
                code |= ((q >> np.uint64(b)) & np.uint64(1)) << np.uint64(b * ndim + a)
    order = np.argsort(code, kind="stable")[:n]
    return np.stack([x[order] for x in xs])


def _covariance(kind, beta, pts):
    n = pts.shape[1]
    p = torch.from_numpy(pts).cuda()
    A = torch.empty(n, n, dtype=torch.float64, device="cuda")
    for i in range(0, n, 2048):
        d2 = sum((c[i:i + 2048, None] - c[None, :]) ** 2 for c in p)
        A[i:i + 2048] = torch.exp(-d2 / (2 * beta * beta)) if kind in (2, 3) else torch.exp(-torch.sqrt(d2) / beta)
    A.diagonal().add_(NUGGET)
    return A


def _covariance_tile(n, seed):
    """A diagonal tile of a 2D squared-exponential covariance (host, column-major = symmetric)."""
    p = _points(2, n, seed)
    d2 = (p[0][:, None] - p[0][None, :]) ** 2 + (p[1][:, None] - p[1][None, :]) ** 2
    A = np.exp(-d2 / (2 * 0.1 * 0.1))
    A[np.diag_indices(n)] += NUGGET
    return A


def exact(case, seed):
    what, n = case["what"], case["n"]
    if what == "gemm":
        state = prepare(case, seed)
        return state["C0"] - state["B"].T @ state["A"]
    if what == "potrf":
        L = torch.linalg.cholesky(torch.from_numpy(_covariance_tile(n, seed)).cuda())
        X = torch.linalg.solve_triangular(L, torch.eye(n, dtype=torch.float64, device="cuda"), upper=False)
        # the library's arrays are column-major
        return L.T.contiguous(), X.T.contiguous(), None
    if n > 60000:
        return None     # the dense matrix would not fit
    rng = np.random.default_rng(seed)
    rhs = rng.standard_normal((case["nrhs"], n)).T if what == "solve" else rng.standard_normal(n)[:, None]
    L = _covariance(case["kind"], case["beta"], _points(2 if case["kind"] == 2 else 3, n, seed))
    torch.linalg.cholesky(L, out=L)
    b = torch.from_numpy(np.ascontiguousarray(rhs)).cuda()
    x = torch.linalg.solve_triangular(L.mT, torch.linalg.solve_triangular(L, b, upper=False), upper=True)
    if what == "solve":
        return x
    logdet = float(2 * torch.log(L.diagonal()).sum())
    loglik = -0.5 * (float(b[:, 0] @ x[:, 0]) + logdet + n * math.log(2 * math.pi))
    return (None, loglik, logdet, x[:, 0].contiguous()) + ((None,) if what == "request" else ())
