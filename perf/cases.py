"""The work that users of this library have it do, as cases to be timed.

Every case is one call (or one loop of calls) of the public interface on
seeded synthetic data: low-rank-plus-noise matrices as in
24am_b200/workloads.py, and bag-of-words-like compressed matrices.  The
iteration counts are fixed (tolerance 0), so that a case is the same amount of
work whatever its inputs.  `kind` says which call:

  host        denseDataSolver on host arrays: upload, solve, result
  batch       a resident matrix's batch of starts, loaded, stepped, read back
  resident    a solve on a resident matrix (starts generated on the device)
  otf         the on-the-fly mode: finished starts replaced one by one
  components  a device matrix taken in, then several components by deflation
  group       many uneven problems run together
  serve       requests queued on a server of resident matrices
  sparse      a solve on a matrix kept compressed (column-centred)
"""
import importlib
import math

import numpy as np
import torch

am = importlib.import_module("24am_b200")


# --------------------------------------------------------------------- cases
def _solve(kind, m, n, k, form, s, iters, gamma=0.0, **more):
    return dict(kind=kind, m=m, n=n, k=k, form=form, s=s, iters=iters, gamma=gamma, **more)


def listed():
    return [
        # the smallest call: a few hundred features from host memory, 64 starts
        dict(_solve("host", 96, 640, 64, 0, 8, 20), name="host_small"),
        # an image data set's size (400 x 10304) stepped by a caller that reads
        # every start's loadings: a narrow batch of 64
        dict(_solve("batch", 400, 10304, 64, 0, 16, 20), name="batch_narrow"),
        # the same data in on-the-fly mode, 256 starts through 64 slots
        dict(_solve("otf", 400, 10304, 64, 1, 16, 10, total=256), name="on_the_fly"),
        # the main workload (2000 x 50000, 1024 starts), top-s with L2 variance
        dict(_solve("resident", 2000, 50000, 1024, 0, 16, 6), name="top_s_l2var"),
        # ... the L1 ball with L1 variance, by the default scan, at a wide support
        dict(_solve("resident", 2000, 50000, 1024, 3, 128, 6, exact_l1=False), name="l1_ball_l1var"),
        # ... an L1 penalty with L2 variance: supports of a hundred or so
        dict(_solve("resident", 2000, 50000, 1024, 6, 1, 6, gamma=0.05), name="l1_penalty_l2var"),
        # ... an L0 penalty that keeps most loadings: both products stay dense;
        # an odd shape
        dict(_solve("resident", 1501, 30011, 513, 5, 1, 6, gamma=0.1), name="l0_penalty_odd"),
        # the largest matrix and batch, mixed precision
        dict(_solve("resident", 8192, 65536, 4096, 0, 128, 8, mixed=True, lead=2), name="mixed_large"),
        # several components of a device matrix, exact L1 ball
        dict(_solve("components", 1000, 20000, 256, 2, 24, 6, count=3, exact_l1=True), name="components"),
        # uneven problems of all formulations in one group
        dict(kind="group", problems=16, m_lo=100, m_hi=5000, n_lo=1000, n_hi=60000, k_lo=32, k_hi=1024,
             s_lo=8, s_hi=256, iters=8, name="group_uneven"),
        # a server's queue: uneven requests on a few resident matrices
        dict(kind="serve", matrices=4, requests=16, m_lo=200, m_hi=3000, n_lo=2000, n_hi=40000, k_lo=32,
             k_hi=512, s_lo=8, s_hi=128, iters=8, name="serve_queue"),
        # a text corpus kept compressed: 100000 documents x 40000 terms
        dict(_solve("sparse", 100000, 40000, 512, 0, 32, 5, nnz=6000000), name="sparse_corpus"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "batch", "resident", "resident", "resident", "resident", "otf", "components",
                       "group", "serve", "sparse", "sparse"])
    if kind == "group":
        return dict(kind=kind, problems=rng.randint(4, 16), m_lo=100, m_hi=_log(rng, 500, 5000), n_lo=1000,
                    n_hi=_log(rng, 5000, 60000), k_lo=32, k_hi=_log(rng, 128, 1024), s_lo=8,
                    s_hi=rng.randint(16, 256), iters=rng.randint(4, 8))
    if kind == "serve":
        return dict(kind=kind, matrices=rng.randint(1, 4), requests=rng.randint(4, 16), m_lo=200,
                    m_hi=_log(rng, 400, 3000), n_lo=2000, n_hi=_log(rng, 4000, 40000), k_lo=32,
                    k_hi=_log(rng, 64, 512), s_lo=8, s_hi=rng.randint(16, 128), iters=rng.randint(4, 8))
    form = rng.randrange(8)
    # penalties from a few loadings kept to most of them
    lo, hi = {4: (0.02, 0.1), 5: (0.05, 0.2), 6: (0.04, 0.1), 7: (0.025, 0.1)}.get(form, (1.0, 1.0))
    gamma = math.exp(rng.uniform(math.log(lo), math.log(hi))) if form >= 4 else 0.0
    s = _log(rng, 4, 128)
    if kind == "sparse":
        n = _log(rng, 4000, 60000)
        return _solve(kind, _log(rng, 4000, 150000), n, _log(rng, 64, 512), rng.randrange(4), s,
                      rng.randint(3, 5), nnz=_log(rng, 300000, 6000000))
    if kind == "otf":
        form = rng.randrange(2)
        k = _log(rng, 16, 128)
        return _solve(kind, _log(rng, 50, 1000), _log(rng, 500, 12000), k, form, s, rng.randint(5, 10),
                      total=k * rng.randint(2, 4))
    if kind in ("host", "batch"):
        return _solve(kind, _log(rng, 64, 1000), _log(rng, 300, 12000), _log(rng, 16, 256), form, s,
                      rng.randint(5, 20), gamma=gamma, exact_l1=rng.random() < 0.5)
    if kind == "components":
        return _solve(kind, _log(rng, 100, 2000), _log(rng, 2000, 30000), _log(rng, 64, 512), rng.randrange(4), s,
                      rng.randint(4, 6), count=rng.randint(2, 3), exact_l1=rng.random() < 0.5)
    return _solve("resident", _log(rng, 100, 5000), _log(rng, 1000, 65536), _log(rng, 32, 2048), form, s,
                  rng.randint(4, 8), gamma=gamma, exact_l1=rng.random() < 0.5, mixed=rng.random() < 0.2, lead=2)


# -------------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _data(m, n, seed, noise=0.1):
    """(n, m) tensor, the m x n matrix column-major: 20 planted sparse
    components in noise, columns centred."""
    g = _generator(seed)
    r, nnz = 20, min(64, n)
    D = torch.randn((n, m), generator=g, device="cuda") * noise
    u = torch.randn((r, m), generator=g, device="cuda")
    u /= u.norm(dim=1, keepdim=True)
    idx = [torch.randperm(n, generator=g, device="cuda")[:nnz] for _ in range(r)]
    v = torch.randn((r, nnz), generator=g, device="cuda")
    v /= v.norm(dim=1, keepdim=True)
    sigma = 10.0 * 0.8 ** torch.arange(r, device="cuda")
    for i in range(r):  # in turn: the components' columns may overlap
        D.index_add_(0, idx[i], (sigma[i] * v[i])[:, None] * u[i][None, :])
    D -= D.mean(dim=1, keepdim=True)
    return D


def _gamma(D, form, c):
    if form < 4:
        return 0.0
    cols = torch.linalg.vector_norm(D, ord=1 if form in (5, 7) else 2, dim=1)
    return float(np.float32(c * float(cols.max())))


def _starts(n, k, seed):
    g = _generator(seed + 77)
    V = torch.rand((k, n), generator=g, device="cuda") * 2.0 - 1.0
    return V / V.norm(dim=1, keepdim=True)


def _settings(case, gamma, **kw):
    a = dict(formulation=case["form"], constraintParameter=min(case["s"], case["n"]), penaltyParameter=gamma,
             tolerance=0.0, maximumIterations=case["iters"], totalStartingPoints=case["k"],
             batchSize=case["k"], startMode=am.START_DEVICE_UNIFORM)
    if case.get("exact_l1"):
        a["l1Mode"] = am.L1_EXACT
    if case.get("mixed"):
        a.update(precision=am.PRECISION_MIXED, leadIterations=case["lead"])
    a.update(kw)
    return am.OptimizationSettings(**a)


def _uneven(case, seed):
    """The group's problems or the server's matrices: sizes spread over the
    logarithm of their ranges by the problem's place (the same for every seed,
    so that every seed is the same amount of work)."""
    count = case.get("problems") or case["matrices"]
    out = []
    for i in range(count):
        a, b = (i * 0.618034) % 1.0, (i * 0.754878 + 0.31) % 1.0
        m = int(case["m_lo"] * (case["m_hi"] / case["m_lo"]) ** a)
        n = int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** b)
        out.append((m, n, seed * 1000 + i))
    return out


def _requests(case):
    """(matrix, formulation, s, starts) of each problem or request."""
    count = case.get("problems") or case["requests"]
    out = []
    for i in range(count):
        c, d = (i * 0.569840 + 0.17) % 1.0, (i * 0.445042 + 0.53) % 1.0
        s = int(round(case["s_lo"] + (case["s_hi"] - case["s_lo"]) * c))
        k = int(round(case["k_lo"] + (case["k_hi"] - case["k_lo"]) * d))
        out.append((i % case.get("matrices", count), (i * 3 + 1) % 8, s, k))
    return out


def _uneven_settings(case, form, s, k, n, gammas):
    return am.OptimizationSettings(formulation=form, constraintParameter=min(s, n),
                                   penaltyParameter=gammas[form], tolerance=0.0,
                                   maximumIterations=case["iters"], totalStartingPoints=k, batchSize=k,
                                   startMode=am.START_DEVICE_UNIFORM)


def _gammas(D):
    return [0.0] * 4 + [_gamma(D, f, 0.1 if f in (4, 6) else 0.025) for f in range(4, 8)]


def _corpus(case, seed):
    """CSC arrays (rows ascending within a column) and column means: terms with
    Zipf-like popularity, documents uniform, counts-like values."""
    m, n, nnz = case["m"], case["n"], case["nnz"]
    g = _generator(seed)
    p = 1.0 / (np.arange(n) + 10.0) ** 1.1
    cdf = torch.from_numpy(np.cumsum(p / p.sum())).cuda()
    u = torch.rand(nnz, generator=g, device="cuda", dtype=torch.float64)
    col = torch.searchsorted(cdf, u).clamp_(max=n - 1)
    row = torch.randint(0, m, (nnz,), generator=g, device="cuda")
    key = torch.unique(col * m + row)
    col, row = key // m, key % m
    # values in steps of 1/1024, so that the means are the same in any order
    val = 1024 - (1024.0 * torch.log1p(-torch.rand(key.numel(), generator=g, device="cuda"))).long()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(col, minlength=n), 0)
    mean = torch.zeros(n, dtype=torch.int64, device="cuda").index_add_(0, col, val).double() / (1024.0 * m)
    return (val.double() / 1024.0).float(), row.int(), ptr.int(), col, mean.float()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sparse":
        val, row, ptr, _, mean = (t.cpu().numpy() for t in _corpus(case, seed))
        solver = am.Solver(0)
        M = am.Matrix.from_csc(solver, val, row, ptr, case["m"], case["n"], means=mean, keep_sparse=True)
        return dict(case=case, solver=solver, matrix=M, settings=_settings(case, 0.0))
    if kind in ("group", "serve"):
        server = am.Server(0, 60 << 30) if kind == "serve" else None
        solver = am.Solver(0) if kind == "group" else None
        mats, gam = [], []
        for m, n, sd in _uneven(case, seed):
            D = _data(m, n, sd)
            torch.cuda.synchronize()
            gam.append(_gammas(D))
            mats.append(server.add_matrix(on_device_ptr=D.data_ptr(), m=m, n=n) if server else
                        am.Matrix(solver, None, on_device_ptr=D.data_ptr(), m=m, n=n))
            del D
        shapes = [(m, n) for m, n, _ in _uneven(case, seed)]
        todo = [(mats[i], _uneven_settings(case, f, s, k, shapes[i][1], gam[i]))
                for i, f, s, k in _requests(case)]
        return dict(case=case, server=server, solver=solver, mats=mats, todo=todo)
    m, n, k = case["m"], case["n"], case["k"]
    D = _data(m, n, seed)
    gamma = _gamma(D, case["form"], case["gamma"])
    torch.cuda.synchronize()
    solver = am.Solver(0)
    if kind == "host":
        return dict(case=case, solver=solver, B=np.asfortranarray(D.cpu().numpy().T),
                    V=np.asfortranarray(_starts(n, k, seed).cpu().numpy().T),
                    settings=_settings(case, gamma, startMode=am.START_INJECTED))
    if kind == "components":
        return dict(case=case, solver=solver, D=D, settings=_settings(case, gamma))
    M = am.Matrix(solver, None, on_device_ptr=D.data_ptr(), m=m, n=n)
    if kind == "batch":
        st = _settings(case, gamma, startMode=am.START_INJECTED)
        V = _starts(n, k, seed).contiguous()
        torch.cuda.synchronize()
        return dict(case=case, solver=solver, matrix=M, V=V, batch=M.batch(st, k))
    if kind == "otf":
        V = np.asfortranarray(_starts(n, case["total"], seed).cpu().numpy().T)
        return dict(case=case, solver=solver, matrix=M, V=V,
                    settings=_settings(case, gamma, startMode=am.START_INJECTED, useOTF=True,
                                       totalStartingPoints=case["total"]))
    return dict(case=case, solver=solver, matrix=M, settings=_settings(case, gamma))


# ---------------------------------------------------------------------- runs
def _signed(x):
    """A loading is defined up to its sign: the largest entry is made positive."""
    return -x if x[np.argmax(np.abs(x))] < 0 else x


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host":
        x, f, st = state["solver"].solve(state["B"], state["settings"], start_points=state["V"])
        return dict(x=_signed(x), objective=f, variance=np.float32(st.explainedVariance))
    if kind == "batch":
        b = state["batch"]
        b.load(device_ptr=state["V"].data_ptr())
        b.iterate(0, case["iters"], sync=False)
        V, val, _, _ = b.read()
        return dict(V=V, objective=val)
    if kind == "components":
        D = state["D"]
        M = am.Matrix(state["solver"], None, on_device_ptr=D.data_ptr(), m=case["m"], n=case["n"])
        X, f, st = M.components(state["settings"], case["count"])
        M.close()
        return dict(x=[_signed(X[:, i]) for i in range(case["count"])], objective=[float(v) for v in f],
                    variance=np.array([s.explained_variance for s in st], np.float32))
    if kind == "group":
        with am.Group(state["solver"], capacity=len(state["todo"])) as g:
            ids = [g.add(M, st) for M, st in state["todo"]]
            g.run()
            out = [g.result(i) for i in ids]
        return [dict(x=_signed(x), objective=float(s.fval), variance=np.float32(s.explained_variance))
                for x, s in out]
    if kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(mid, st) for mid, st in state["todo"]]
        out = [srv.wait(t) for t in tickets]
        return [dict(x=_signed(x), objective=float(s.fval), variance=np.float32(s.explained_variance))
                for x, s in out]
    x, f, st = state["matrix"].solve(state["settings"], start_points=state.get("V"))
    return dict(x=_signed(x), objective=f, variance=np.float32(st.explained_variance))


# ---------------------------------------------------------------------- work
def _iterations(m, n, k, form, s, iters, products_nnz=None):
    """Operations of `iters` steps of k starts: both products on the first
    (dense) step, then V = B^T Z whole and Z = B V over the kept loadings (s of
    them for the constraints; the penalties keep what they keep, counted as the
    one entry in 32 up to which a gather is the cheaper form)."""
    whole = 2.0 * (m * n if products_nnz is None else products_nnz) * k
    kept = s if form < 4 else n / 32
    part = min(whole, 2.0 * m * kept * k) if products_nnz is None else whole * min(1.0, 32.0 * kept / n)
    return whole * (iters + 1) + part * (iters - 1)


def work(case):
    kind, iters = case["kind"], case["iters"]
    if kind in ("group", "serve"):
        shapes = [(m, n) for m, n, _ in _uneven(case, 0)]
        flops, data = 0.0, float(sum(4 * m * n for m, n in shapes))
        for i, f, s, k in _requests(case):
            m, n = shapes[i]
            flops += _iterations(m, n, k, f, s, iters)
            data += 4.0 * n
        return dict(bytes=data, flops=flops)
    m, n, k, f, s = case["m"], case["n"], case["k"], case["form"], case["s"]
    if kind == "sparse":
        return dict(bytes=8.0 * case["nnz"] + 4.0 * (m + 2 * n),
                    flops=_iterations(m, n, k, f, s, iters, products_nnz=case["nnz"]))
    if kind == "otf":
        rounds = case["total"] // k
        return dict(bytes=4.0 * (m * n + n * case["total"] + n),
                    flops=rounds * _iterations(m, n, k, f, s, iters))
    count = case.get("count", 1)
    starts = {"host": n * k, "batch": 2 * n * k}.get(kind, 0)
    return dict(bytes=4.0 * (m * n * (2 * count - 1) + starts + n * count),
                flops=count * _iterations(m, n, k, f, s, iters))


# ------------------------------------------------------------- in 64 bits
def _device_starts(n, k):
    """The library's device starts: U[-1, 1) from the top 24 bits of the
    splitmix64 mixer of (start << 32 | row), unit columns.  n x k."""
    M64 = (1 << 64) - 1

    def wrap(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    def shr(x, b):
        return (x >> b) & ((1 << (64 - b)) - 1)

    key = (torch.arange(k, device="cuda", dtype=torch.int64) << 32)[None, :]
    x = key | torch.arange(n, device="cuda", dtype=torch.int64)[:, None]
    x = x + wrap(0x9E3779B97F4A7C15 & M64)
    x = (x ^ shr(x, 30)) * wrap(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * wrap(0x94D049BB133111EB)
    x = x ^ shr(x, 31)
    V = shr(x, 40).double() * (2.0 / 16777216.0) - 1.0
    return V / torch.linalg.vector_norm(V, dim=0, keepdim=True)


def _l1_ball(V, s):
    """The level w with ||(|v| - w)_+||_1 / ||(|v| - w)_+||_2 = sqrt(s), per column."""
    a, _ = torch.sort(V.abs(), dim=0, descending=True)
    n = a.shape[0]
    t = torch.arange(1, n + 1, device=a.device, dtype=a.dtype)[:, None]
    S1, S2 = torch.cumsum(a, 0), torch.cumsum(a * a, 0)
    lo = torch.cat([a[1:], torch.zeros_like(a[:1])])
    num, den = S1 - t * lo, (S2 - 2.0 * lo * S1 + t * lo * lo).clamp_(min=1e-300)
    hit = num * num >= s * den
    at = torch.where(hit.any(0), hit.int().argmax(0), torch.full((a.shape[1],), n - 1, device=a.device))[None, :]
    t1, s1, s2 = (at + 1).to(a.dtype), S1.gather(0, at), S2.gather(0, at)
    qa, qb, qc = t1 * (t1 - s), 2.0 * s1 * (s - t1), s1 * s1 - s * s2
    w = (-qb - torch.sqrt((qb * qb - 4.0 * qa * qc).clamp_(min=0.0))) / (2.0 * qa)
    w = torch.where(qa == 0.0, -qc / qb, w)
    w = torch.minimum(torch.maximum(w, lo.gather(0, at)), a.gather(0, at))
    return torch.where(hit.any(0)[None, :], w, torch.zeros_like(w))


def _step(mul, tmul, V, form, s, gamma, exact_l1=False):
    """One iteration in 64 bits: (new loadings, objectives)."""
    Z = mul(V)
    l1var = form in (1, 3, 5, 7)
    norm = Z.abs().sum(0) if l1var else torch.linalg.vector_norm(Z, dim=0)
    if l1var:
        Z = torch.sign(Z)
    elif form >= 4:
        Z = Z / norm
    V = tmul(Z)
    if form < 4:
        if form < 2:
            level = torch.topk(V.abs(), s, dim=0).values[-1:]
            V = torch.where(V.abs() >= level, V, torch.zeros_like(V))
        else:
            w = _l1_ball(V, s)
            V = torch.sign(V) * (V.abs() - w).clamp_(min=0.0)
        return V / torch.linalg.vector_norm(V, dim=0, keepdim=True), norm
    if form >= 6:
        d = (V.abs() - gamma).clamp_(min=0.0)
        return torch.sign(V) * d, torch.sqrt((d * d).sum(0))
    d = (V * V - gamma).clamp_(min=0.0)
    return torch.where(d > 0.0, V, torch.zeros_like(V)), d.sum(0)


def _best(mul, V, f):
    """The first largest objective's loading, normalised and signed."""
    i = int(torch.argmax(torch.where(torch.isnan(f), torch.full_like(f, -1.0), f)))
    x = V[:, i] / torch.linalg.vector_norm(V[:, i])
    return dict(x=_signed(x.cpu().numpy()), objective=float(f[i]),
                variance=np.float64(float((mul(x[:, None]) ** 2).sum())))


def _exact_solve(B, n, k, form, s, iters, gamma, exact_l1, V=None):
    """B: the n x m transpose in 64 bits."""
    def mul(X):
        return B.t() @ X

    def tmul(Z):
        return B @ Z

    V = _device_starts(n, k) if V is None else V
    for _ in range(iters):
        V, f = _step(mul, tmul, V, form, s, gamma, exact_l1)
    return V, f, mul


def _no_value(form, exact_l1):
    # the default L1-ball scan stops at its first rank or not by the last bit of
    # the largest |v|: it has no value of its own in 64 bits
    return form in (2, 3) and not exact_l1


def exact(case, seed):
    kind = case["kind"]
    if kind == "sparse":
        if _no_value(case["form"], False):
            return None
        val, row, ptr, col, mean = _corpus(case, seed)
        m, n = case["m"], case["n"]
        C = torch.sparse_csr_tensor(ptr.long(), row.long(), val.double(), size=(n, m))  # B^T by columns
        order = torch.argsort(row.long() * n + col)
        rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
        rp[1:] = torch.cumsum(torch.bincount(row.long(), minlength=m), 0)
        R = torch.sparse_csr_tensor(rp, col[order], val[order].double(), size=(m, n))
        mu = mean.double()[:, None]

        def mul(X):
            return R @ X - (mu * X).sum(0, keepdim=True)

        def tmul(Z):
            return C @ Z - mu * Z.sum(0, keepdim=True)

        V = _device_starts(n, case["k"])
        for _ in range(case["iters"]):
            V, f = _step(mul, tmul, V, case["form"], min(case["s"], n), 0.0)
        return _best(mul, V, f)
    if kind in ("group", "serve"):
        shapes = _uneven(case, seed)
        out = []
        for i, f, s, k in _requests(case):
            m, n, sd = shapes[i]
            if _no_value(f, False):
                out.append(None)
                continue
            D = _data(m, n, sd)
            g = _gammas(D)[f]
            V, fv, mul = _exact_solve(D.double(), n, k, f, min(s, n), case["iters"], g, False)
            out.append(_best(mul, V, fv))
        return out
    m, n, k, form = case["m"], case["n"], case["k"], case["form"]
    if case.get("mixed") or kind == "otf" or _no_value(form, case.get("exact_l1")):
        # mixed precision keeps 11 bits of each operand by the caller's choice;
        # on the fly, starts finish in an order of their own
        return None
    D = _data(m, n, seed)
    gamma, s = _gamma(D, form, case["gamma"]), min(case["s"], n)
    B = D.double()
    del D
    if kind in ("host", "batch"):
        V, f, mul = _exact_solve(B, n, k, form, s, case["iters"], gamma, True, _starts(n, k, seed).double().t())
        return _best(mul, V, f) if kind == "host" else dict(V=V.cpu().numpy(), objective=f.cpu().numpy())
    if kind == "components":
        got = []
        for _ in range(case["count"]):
            V, f, mul = _exact_solve(B, n, k, form, s, case["iters"], gamma, True)
            got.append(_best(mul, V, f))
            x = torch.from_numpy(got[-1]["x"]).cuda()
            B = B - x[:, None] * (B.t() @ x)[None, :]
        return dict(x=[g["x"] for g in got], objective=[g["objective"] for g in got],
                    variance=np.array([g["variance"] for g in got]))
    V, f, mul = _exact_solve(B, n, k, form, s, case["iters"], gamma, True)
    return _best(mul, V, f)
