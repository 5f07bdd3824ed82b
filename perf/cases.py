"""The work that programs give this library, as cases that can be timed one
by one through its public entry points (planc_b200.Context, Batch, CPLoss).

A case is a dict of plain values: `kind` names the entry point, `dims` the
mode sizes ("64x64x64"), `rank` the number of components, `precision` the
context's precision, and so on. A pass of an iterative case starts from the
program's initial factors, runs `iters` outer iterations with the relative
error of each, and reads the factors back, as a program that tries several
starts (or ranks of iterations) on one resident tensor does. Tensors are
nonnegative CP models with U[0, 1) factors plus Gaussian noise, clipped at 0.
"""
import numpy as np
import torch

import planc_b200
from planc_b200.autograd import CPLoss

DEV = "cuda:0"


def _dims(case):
    return tuple(int(d) for d in case["dims"].split("x"))


def listed():
    return [
        # A small FP64 tensor, twenty HALS iterations: the smallest whole call,
        # where launches and latency count.
        dict(name="hals_fp64_64cube", kind="ntf", dims="64x64x64", rank=8, algo="hals",
             precision="fp64", iters=20, dimtree=True, noise=0.01, sparse=0.0),
        # A small ragged 4-way FP64 tensor with an odd rank, multiplicative updates.
        dict(name="mu_fp64_4way_odd", kind="ntf", dims="61x47x33x29", rank=11, algo="mu",
             precision="fp64", iters=10, dimtree=True, noise=0.01, sparse=0.0),
        # FP64 at the size where the contractions dominate.
        dict(name="hals_fp64_512cube", kind="ntf", dims="512x512x512", rank=32, algo="hals",
             precision="fp64", iters=5, dimtree=True, noise=0.01, sparse=0.0),
        # The benchmark's tensor: 1024^3, rank 32, BF16 tensor-core MTTKRP.
        dict(name="hals_bf16_1024cube", kind="ntf", dims="1024x1024x1024", rank=32, algo="hals",
             precision="bf16", iters=5, dimtree=True, noise=0.01, sparse=0.0),
        # An ordinary measured tensor: no mode size or rank is round.
        dict(name="mu_bf16_odd", kind="ntf", dims="417x250x333", rank=20, algo="mu",
             precision="bf16", iters=5, dimtree=True, noise=0.01, sparse=0.0),
        # The large 4-way tensor with sparse factors, rank 64, ANLS/BPP.
        dict(name="bpp_bf16_192x4", kind="ntf", dims="192x192x192x192", rank=64, algo="anlsbpp",
             precision="bf16", iters=3, dimtree=True, noise=0.01, sparse=0.5),
        # The direct MTTKRP (the solver classes' own default) on split BF16, AO-ADMM.
        dict(name="admm_bf16x2_direct", kind="ntf", dims="300x260x220", rank=24, algo="aoadmm",
             precision="bf16x2", iters=5, dimtree=False, noise=0.01, sparse=0.0),
        # Nesterov with its extrapolation step (from the sixth iteration on), FP64.
        dict(name="nesterov_fp64", kind="ntf", dims="200x150x120", rank=16, algo="nesterov",
             precision="fp64", iters=8, dimtree=True, noise=0.01, sparse=0.0),
        # Many small tensors of uneven sizes and ranks factorised together.
        dict(name="batch256_hals_bf16", kind="batch", count=256, low=32, high=256, algo="hals",
             precision="bf16", iters=5, noise=0.01),
        # Forward and backward of the differentiable loss on torch leaves.
        dict(name="cploss_bf16_512cube", kind="cploss", dims="512x512x512", rank=32,
             precision="bf16", noise=0.05),
        # NMF of a large dense matrix, HALS.
        dict(name="nmf_hals_bf16_16384", kind="nmf", dims="16384x16384", rank=32, algo="hals",
             precision="bf16", iters=5, noise=0.01),
        # Nonnegative least squares on host arrays: one rank-50 mode's normal equations.
        dict(name="nnls_k50_3000rows", kind="nnls", rank=50, columns=3000),
    ]


def _log_int(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def _draw_dims(rng, n, low, high, most, least=1):
    while True:
        d = [min(high, max(low, _log_int(rng, low, high))) for _ in range(n)]
        if rng.random() < 0.3:  # powers of two are common, too
            d = [1 << int(round(np.log2(x))) for x in d]
        if least <= int(np.prod(d)) <= most and max(d) <= high:
            return "x".join(str(x) for x in d)


def draw(rng):
    kind = rng.choice(["ntf", "ntf", "ntf", "ntf", "ntf", "ntf", "batch", "cploss", "nmf", "nnls"])
    if kind == "ntf":
        algo = rng.choice(["hals", "hals", "mu", "anlsbpp", "aoadmm", "nesterov"])
        if algo == "nesterov":  # its inner loop's length depends on the data: the listed range
            return dict(kind=kind, dims=_draw_dims(rng, 3, 60, 300, 8_000_000, 300_000),
                        rank=rng.randint(6, 16), algo=algo, precision="fp64", iters=8,
                        dimtree=True, noise=0.01, sparse=0.0)
        precision = rng.choice(["fp64", "bf16", "bf16", "bf16x2"])
        four = rng.random() < 0.3
        most = 130_000_000 if precision == "fp64" else 600_000_000
        if four:
            dims = _draw_dims(rng, 4, 20 if precision == "fp64" else 32, 192, most)
        else:
            dims = _draw_dims(rng, 3, 48 if precision == "fp64" else 96, 1024, most)
        rank = rng.randint(4, min(64, min(int(d) for d in dims.split("x"))))
        return dict(kind=kind, dims=dims, rank=rank, algo=algo, precision=precision,
                    iters=rng.randint(3, 5), dimtree=rng.random() < 0.8, noise=0.01,
                    sparse=0.5 if algo == "anlsbpp" else 0.0)
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 8, 200), low=32, high=rng.randint(64, 256),
                    algo=rng.choice(["hals", "mu"]), precision="bf16", iters=rng.randint(3, 5),
                    noise=0.01)
    if kind == "cploss":
        return dict(kind=kind, dims=_draw_dims(rng, 3, 64, 640, 140_000_000),
                    rank=rng.randint(4, 48), precision=rng.choice(["bf16", "bf16", "bf16x2", "fp64"]),
                    noise=0.05)
    if kind == "nmf":
        return dict(kind=kind, dims=_draw_dims(rng, 2, 256, 16384, 200_000_000), rank=rng.randint(4, 48),
                    algo=rng.choice(["hals", "mu", "anlsbpp"]),
                    precision=rng.choice(["fp64", "bf16", "bf16"]), iters=rng.randint(3, 5), noise=0.01)
    return dict(kind=kind, rank=rng.randint(5, 64), columns=_log_int(rng, 100, 8000))


# ---------------------------------------------------------------- inputs


def _factors(dims, rank, rng, sparse=0.0):
    out = []
    for d in dims:
        a = rng.random((d, rank))
        if sparse > 0.0:
            a[rng.random(a.shape) < sparse] = 0.0
        out.append(a)
    return out


def _krp(fs):
    """Row-wise Kronecker product with the first factor's index fastest."""
    k = fs[0].clone()
    for f in fs[1:]:
        k = (f[:, None, :] * k[None, :, :]).reshape(-1, k.shape[1])
    return k


def _cp_data(A, noise, gen):
    """The CP model of host factors A + noise, clipped at 0: FP32, flat, mode 0 fastest."""
    G = np.ones((A[0].shape[1],) * 2)
    for a in A:
        G = G * (a.T @ a)
    sigma = noise * float(np.sqrt(G.sum() / np.prod([float(a.shape[0]) for a in A])))
    half = (len(A) + 1) // 2
    T = [torch.tensor(a, dtype=torch.float32, device=DEV) for a in A]
    X = _krp(T[half:]) @ _krp(T[:half]).T if len(A) > 2 else T[1] @ T[0].T
    X = X.reshape(-1)
    step = 1 << 27
    for a in range(0, X.numel(), step):
        part = X[a:a + step]
        part.add_(torch.randn(part.shape, generator=gen, device=DEV), alpha=sigma).clamp_(min=0.0)
    return X


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _tensor_inputs(case, seed):
    """(dims, data on the device, initial factors on the host)"""
    dims, rng = _dims(case), np.random.default_rng(seed)
    A = _factors(dims, case["rank"], rng, case.get("sparse", 0.0))
    F0 = _factors(dims, case["rank"], rng)
    X = _cp_data(A, case["noise"], _gen(seed))
    return dims, X.double() if case["precision"] == "fp64" else X, F0


def _batch_inputs(case, seed):
    # the sizes of a batch belong to the case and its data to the seed
    sizes = np.random.default_rng(case["count"] * 1000 + case["high"])
    rng, gen = np.random.default_rng(seed), _gen(seed)
    for _ in range(case["count"]):
        dims = tuple(int(d) for d in sizes.integers(case["low"], case["high"] + 1, size=3))
        rank = int(sizes.choice([4, 8, 16, 32]))
        yield dims, _cp_data(_factors(dims, rank, rng), case["noise"], gen), _factors(dims, rank, rng)


def _nnls_inputs(case, seed):
    # the normal equations of a mode of a sparse nonnegative model, away from its solution
    rng, n = np.random.default_rng(seed), case["rank"]
    G = np.ones((n, n))
    for a in _factors((4 * n, 4 * n), n, rng, 0.5):
        a = a / np.maximum(np.linalg.norm(a, axis=0), 1e-300)
        G = G * (a.T @ a)
    Xt = rng.random((n, case["columns"]))
    Xt[rng.random(Xt.shape) < 0.5] = 0.0
    return G, G @ Xt + 0.02 * rng.standard_normal(Xt.shape)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "nnls":
        G, B = _nnls_inputs(case, seed)
        return {"case": case, "ctx": planc_b200.Context(0, "fp64"), "G": G, "B": B}
    if kind == "batch":
        b = planc_b200.Batch(0, case["precision"], nstreams=64)
        starts = []
        for dims, X, F0 in _batch_inputs(case, seed):
            torch.cuda.current_stream().synchronize()
            b.add(X.data_ptr(), F0, dims=dims, dtype="f32")
            starts.append(F0)
        return {"case": case, "batch": b, "F0": starts}
    dims, X, F0 = _tensor_inputs(case, seed)
    torch.cuda.current_stream().synchronize()
    if kind == "cploss":
        loss = CPLoss(X, dims=dims, rank=case["rank"], precision=case["precision"])
        F = [torch.tensor(f, dtype=torch.float64, device=DEV, requires_grad=True) for f in F0]
        return {"case": case, "loss": loss, "F": F}
    ctx = planc_b200.Context(0, case["precision"])
    ctx.set_tensor(X.data_ptr(), dims=dims, dtype="f64" if X.dtype == torch.float64 else "f32")
    return {"case": case, "ctx": ctx, "F0": F0}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "nnls":
        X, passive, iters = state["ctx"].bpp_solve(state["G"], state["B"])
        return {"x": X, "passive": passive, "iters": iters}
    if kind == "batch":
        b = state["batch"]
        for i, F0 in enumerate(state["F0"]):
            b.set_factors(i, F0)
        errors = b.run(case["algo"], case["iters"])
        got = [b.get_factors(i) for i in range(len(state["F0"]))]
        return {"errors": errors, "factors": np.concatenate([f.ravel() for F, _ in got for f in F]),
                "lambda": np.concatenate([lam for _, lam in got])}
    if kind == "cploss":
        F = state["F"]
        for f in F:
            f.grad = None
        loss = state["loss"](*F)
        loss.backward()
        return {"loss": loss.detach(), "grads": [f.grad for f in F]}
    ctx = state["ctx"]
    if kind == "nmf":
        ctx.nmf_set_factors(*state["F0"])
        objective, rel = ctx.nmf_run(case["algo"], case["iters"])
        W, H = ctx.nmf_get_factors()
        return {"objective": objective, "rel": rel, "W": W, "H": H}
    ctx.set_factors(state["F0"])
    if case["algo"] in ("aoadmm", "nesterov"):
        ctx.reset_update_state()
    errors = ctx.run(case["algo"], case["iters"], dimtree=case["dimtree"])
    F, lam = ctx.get_factors()
    return {"errors": errors, "factors": F, "lambda": lam}


_ELEMENT = {"fp64": 8, "bf16": 2, "bf16x2": 4}


def _tensor_work(dims, rank, element, iters):
    # two sweeps over the resident tensor an iteration (the modes of one half
    # of the tree can share a partial contraction, the other half's needs the
    # first half's new factors), the factors in and out
    n = float(np.prod([float(d) for d in dims]))
    return iters * 2 * n * element + 2 * 8 * sum(dims) * rank, iters * 2 * 2 * n * rank


def work(case):
    kind = case["kind"]
    if kind == "nnls":
        n, c = case["rank"], case["columns"]
        # one Cholesky solve of about half of the indexes and one product a column
        return {"bytes": 8 * n * n + (2 * 8 + 4) * n * c + 4 * c,
                "flops": c * ((n / 2) ** 3 / 3 + 2 * (n / 2) ** 2 + 2 * n * n)}
    if kind == "batch":
        sizes = np.random.default_rng(case["count"] * 1000 + case["high"])
        total = np.zeros(2)
        for _ in range(case["count"]):
            dims = [int(d) for d in sizes.integers(case["low"], case["high"] + 1, size=3)]
            total += _tensor_work(dims, int(sizes.choice([4, 8, 16, 32])),
                                  _ELEMENT[case["precision"]], case["iters"])
        return {"bytes": float(total[0]), "flops": float(total[1])}
    b, f = _tensor_work(_dims(case), case["rank"], _ELEMENT[case["precision"]], case.get("iters", 1))
    return {"bytes": b, "flops": f}


# ------------------------------------------------- the same results in 64 bits


def _mttkrp(X, dims, F, n):
    """X: flat FP64; F: FP64 factors on the device."""
    half = (len(dims) + 1) // 2
    left = n < half
    mine = list(range(half)) if left else list(range(half, len(dims)))
    other = [m for m in range(len(dims)) if m not in mine]
    rows = int(np.prod([dims[m] for m in range(half)]))
    X2 = X.view(-1, rows)
    K = _krp([F[m] for m in other])
    P = X2.T @ K if left else X2 @ K
    k = K.shape[1]
    P = P.reshape([dims[m] for m in reversed(mine)] + [k])
    for m in reversed(mine):  # the slowest of mine is the first axis
        axis = 0 if m > n else P.dim() - 2
        if m == n:
            continue
        shape = [1] * P.dim()
        shape[axis], shape[-1] = dims[m], k
        P = (P * F[m].view(shape)).sum(axis)
    return P


def _normalize(f):
    lam = torch.linalg.vector_norm(f, dim=0)
    return f / torch.where(lam > 0, lam, torch.ones_like(lam)), lam


def _hals(H, M, G):
    H = H.clone()
    for i in range(H.shape[1]):
        H[:, i] = (H[:, i] + M[:, i] - H @ G[:, i]).clamp_(min=1e-17)
    return H


def _nnls(G, B, given=None):
    """Rows of the result: argmin over x >= 0 of x G x / 2 - b x, by block principal pivoting."""
    rows, n = B.shape
    passive = torch.zeros_like(B, dtype=torch.bool) if given is None else given
    best = torch.full((rows,), n + 1, device=B.device)
    tries = torch.full((rows,), 3, device=B.device)
    X, Y = torch.zeros_like(B), -B
    eye = torch.eye(n, dtype=B.dtype, device=B.device)
    for _ in range(5 * n + 1):
        wrong = ((Y < 0) & ~passive) | ((X < 0) & passive)
        bad = wrong.sum(1)
        open_ = bad > 0
        if not bool(open_.any()):
            break
        better = open_ & (bad < best)
        again = open_ & ~better & (tries >= 1)
        best = torch.where(better, bad, best)
        tries = torch.where(better, torch.full_like(tries, 3), tries - again.to(tries.dtype))
        last = torch.zeros_like(wrong)
        at = (wrong * torch.arange(1, n + 1, device=B.device)).argmax(1)
        last[torch.arange(rows, device=B.device), at] = True
        flip = torch.where((better | again)[:, None], wrong, last) & open_[:, None]
        passive = passive ^ flip
        r = torch.nonzero(open_).reshape(-1)
        for part in r.split(4096):
            p = passive[part].to(B.dtype)
            A = G[None] * p[:, :, None] * p[:, None, :] + eye[None] * (1 - p)[:, :, None]
            x = torch.linalg.solve(A, (B[part] * p)[:, :, None])[:, :, 0]
            y = x @ G - B[part]
            y = torch.where(passive[part], torch.zeros_like(y), y)
            X[part] = torch.where(x.abs() < 1e-12, torch.zeros_like(x), x)
            Y[part] = torch.where(y.abs() < 1e-12, torch.zeros_like(y), y)
    return X, passive


def _admm(H, U, M, G):
    k = G.shape[0]
    alpha = float(torch.trace(G)) / k
    alpha = alpha if alpha > 0 else 0.01
    L = torch.linalg.cholesky(G + alpha * torch.eye(k, dtype=G.dtype, device=G.device))
    for _ in range(5):
        old = H
        aux = torch.cholesky_solve((M + alpha * (H + U)).T, L).T
        H = (aux - U).clamp(min=0.0)
        U = U + H - aux
        r, s = torch.linalg.norm(H - aux), torch.linalg.norm(H - old)
        if r < 0.01 * torch.linalg.norm(H) and s < 0.01 * torch.linalg.norm(U):
            break
    return H, _normalize(U)[0]


def _nesterov(start, M, G):
    w = torch.linalg.eigvalsh(G)
    mu, L = float(w[0]), float(w[-1])
    q = L / mu
    lam = 10 * mu if q > 1e6 else mu if q > 1e3 else mu / 10
    Gm = G + lam * torch.eye(G.shape[0], dtype=G.dtype, device=G.device)
    q, inv = (mu + lam) / (L + lam), 1 / (L + lam)
    Mm = -lam * start - M
    H = Y = start
    alpha = 1.0
    for _ in range(20000):
        grad = Mm + Y @ Gm
        if float((grad * Y).abs().max()) <= 1e-2 and float(grad.min()) >= -1e-2:
            break
        new = (Y - inv * grad).clamp(min=0.0)
        b, c = alpha * alpha - q, -alpha * alpha
        nxt = (-b + (b * b - 4 * c) ** 0.5) / 2
        beta = alpha * (1 - alpha) / (nxt + alpha * alpha)
        Y, H, alpha = new + beta * (new - H), new, nxt
    return H


def _exact_ntf(case, X, dims, F0):
    N, algo = len(dims), case["algo"]
    F = [_normalize(torch.tensor(f, device=DEV))[0] for f in F0]
    lam = torch.ones(case["rank"], dtype=torch.float64, device=DEV)
    X = X.double()
    norm2 = (X @ X).clone()
    aux = [torch.zeros_like(f) for f in F]
    prox, prev = [torch.zeros_like(f) for f in F], [torch.zeros_like(f) for f in F]
    prox_lam = prev_lam = lam
    fails, exponent, errors = 0, 3, []

    def grams(skip=None):
        G = torch.ones(case["rank"], case["rank"], dtype=torch.float64, device=DEV)
        for m in range(N):
            if m != skip:
                G = G * (F[m].T @ F[m])
        return G

    def error(lam, M):
        inner = (M * F[N - 1]).sum(0) @ lam
        return torch.sqrt((norm2 - 2 * inner + lam @ grams() @ lam) / norm2)

    for it in range(case["iters"]):
        for n in range(N):
            G, M = grams(n), _mttkrp(X, dims, F, n)
            if algo == "hals":
                new = _hals(F[n], M, G)
            elif algo == "mu":
                new = F[n] * M / (F[n] @ G + 1e-6)
            elif algo == "anlsbpp":
                new = _nnls(G, M)[0]
            elif algo == "aoadmm":
                new, aux[n] = _admm(F[n], aux[n], M, G)
            else:
                if n == 0:
                    prev_lam = prox_lam
                prev[n] = prox[n]
                new = _nesterov(prox[n], M, G)
                prox[n], prox_lam = _normalize(new)
            F[n], lam = _normalize(new)
        e = error(lam, M)
        errors.append(e)
        if algo == "nesterov" and it > 5:  # extrapolate, keep what lowers the error
            kept, kept_lam = list(F), lam
            step, acc = (it + 1) ** (1.0 / exponent), []
            for n in range(N):
                cur, old = (lam * F[n], prev_lam * prev[n]) if n == N - 1 else (F[n], prev[n])
                a, acc_lam = _normalize((cur - old) * step + cur)
                acc.append(a)
            F[:] = acc
            if error(acc_lam, _mttkrp(X, dims, F, N - 1)) < e:
                prox, lam = list(F), acc_lam
                prox_lam = _normalize(F[N - 1])[1]
            else:
                F[:], lam = kept, prox_lam
                fails += 1
                if fails > 5:
                    fails, exponent = 0, exponent + 1
    return {"errors": torch.stack(errors), "factors": F, "lambda": lam}


def _exact_nmf(case, X, dims, F0):
    m, n = dims
    A = X.double().view(n, m)  # column-major A: its transpose
    norm2 = (X.double() @ X.double()).clone()
    W, H = (torch.tensor(f, device=DEV) for f in F0)

    def by_w(W, H):
        s = torch.linalg.vector_norm(W, dim=0)
        return W / s, H * s

    if case["algo"] == "hals":
        W, H = by_w(W, H)
    objective, rel = [], []
    for _ in range(case["iters"]):
        if case["algo"] == "anlsbpp":
            W = _nnls(H.T @ H, A.T @ H)[0]
            H = _nnls(W.T @ W, A @ W)[0]
        elif case["algo"] == "mu":
            H = H * (A @ W) / (H @ (W.T @ W) + 1e-17)
            W = W * (A.T @ H) / (W @ (H.T @ H) + 1e-17)
        else:
            H = _hals(H, A @ W, W.T @ W)
            AH, G = A.T @ H, H.T @ H
            W = W.clone()
            for x in range(W.shape[1]):
                w = (W[:, x] * G[x, x] + (AH[:, x] - W @ G[:, x])).clamp_(min=1e-17)
                W[:, x] = w / torch.linalg.vector_norm(w)
            W, H = by_w(W, H)
        fit = norm2 - 2 * (H * (A @ W)).sum() + ((W.T @ W) * (H.T @ H)).sum()
        objective.append(fit)
        rel.append(torch.sqrt(fit / norm2))
    if case["algo"] != "hals":
        W, H = by_w(W, H)
    return {"objective": torch.stack(objective), "rel": torch.stack(rel), "W": W, "H": H}


def exact(case, seed):
    kind = case["kind"]
    if kind == "nnls":
        G, B = (torch.tensor(a, device=DEV) for a in _nnls_inputs(case, seed))
        return {"x": _nnls(G, B.T.contiguous())[0].T.contiguous(), "passive": None, "iters": None}
    if kind == "batch":
        outs = []
        for dims, X, F0 in _batch_inputs(case, seed):
            one = dict(case, rank=F0[0].shape[1])
            outs.append(_exact_ntf(one, X, dims, F0))
        return {"errors": torch.stack([o["errors"] for o in outs]),
                "factors": torch.cat([f.reshape(-1) for o in outs for f in o["factors"]]),
                "lambda": torch.cat([o["lambda"] for o in outs])}
    dims, X, F0 = _tensor_inputs(case, seed)
    if kind == "cploss":
        F, X = [torch.tensor(f, device=DEV) for f in F0], X.double()
        M = [_mttkrp(X, dims, F, n) for n in range(len(F))]
        G = [f.T @ f for f in F]
        loss = 0.5 * (X @ X) - (M[0] * F[0]).sum() + 0.5 * torch.stack(G).prod(0).sum()
        grads = []
        for n, f in enumerate(F):
            rest = torch.stack([g for m, g in enumerate(G) if m != n]).prod(0)
            grads.append(f @ rest - M[n])
        return {"loss": loss, "grads": grads}
    return (_exact_nmf if kind == "nmf" else _exact_ntf)(case, X, dims, F0)
