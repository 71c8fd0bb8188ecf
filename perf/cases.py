"""The work that is measured: calls through the package's public entry points, as a
program that searches for formulas makes them.

Such a program draws batches of expressions (``sample``) and converts them between the
notations (``convert``), evaluates them with or without gradients (``eval``, ``multi``),
fits their constants (``fit``), and keeps a learned warm start in step (``warm``).  The
sizes are those of the package's workloads, tests and benchmark (``workloads.py``: tapes of
up to 64 nodes, mean length about 20 for evaluation and uniform lengths for fits, N = 512 to
1024 points; the README problem: N = 100, M = 32), scaled down to a single interactive call
and up to a whole search batch, with odd sizes in between.

``listed()`` is the fixed set, ``draw()`` gives further cases of the same ranges,
``prepare()`` the inputs on the GPU, ``run()`` one pass, ``work()`` the bytes and operations
it cannot do without, and ``exact()`` its outputs in 64 bits by plain torch.
"""
from __future__ import annotations

import numpy as np
import torch

import cudasymbolicregression_gb300 as sr
from cudasymbolicregression_gb300 import tapes, warmstart, workloads

DEV = "cuda"
ADD, SUB, MUL, DIV, SIN, COS, EXP, LOG, LEARNABLE, VAR = 40, 41, 42, 43, 10, 11, 12, 13, 1, 50

# Closures (forward + adjoint passes) an average problem of each fit workload takes, and
# the operations one closure takes at one point (workloads.FWD_FLOPS + ADJ_FLOPS of its
# average tape), for work().
CLOSURES = {"readme": 110, "ragged": 90, "backtracking": 80}
FLOPS_PER_POINT = {"readme": 50, "ragged": 200}


def listed():
    return [
        # one interactive look at a population: a hundred README expressions, values only
        dict(name="eval_small", kind="eval", tapes="readme", B=100, M=32, N=100, n_x=1, grad="", dtype="f32"),
        # an ordinary gradient step of a program of its own (torch optimiser): odd sizes,
        # gradients for the constants and the inputs
        dict(name="eval_step_odd", kind="eval", tapes="general", B=1003, M=50, N=777, n_x=3, grad="CX", dtype="f32"),
        # a large batch of the evaluation workload, forward and adjoint
        dict(name="eval_step_large", kind="eval", tapes="general", B=16384, M=64, N=1024, n_x=4, grad="C", dtype="f32"),
        # the same in double precision, for a final check or refinement of a shortlist
        dict(name="eval_step_f64", kind="eval", tapes="general", B=512, M=64, N=1000, n_x=2, grad="CX", dtype="f64"),
        # several constant sets per expression at once (multi-start), with gradients
        dict(name="multi_step", kind="multi", tapes="general", B=1000, M=32, N=256, n_x=2, K=8),
        # fits: a handful of README expressions, a README population, the ragged batch of a
        # search round, and an odd-sized one with the backtracking line search
        dict(name="fit_small", kind="fit", tapes="readme", B=32, M=32, N=100, max_iter=100, search="strong_wolfe"),
        dict(name="fit_readme", kind="fit", tapes="readme", B=8192, M=32, N=100, max_iter=100, search="strong_wolfe"),
        dict(name="fit_ragged", kind="fit", tapes="ragged", B=16384, M=64, N=512, max_iter=200, search="strong_wolfe"),
        dict(name="fit_backtracking", kind="fit", tapes="ragged", B=2999, M=40, N=257, max_iter=100,
             search="backtracking"),
        # candidates of a search round from the grammar object
        dict(name="sample", kind="sample", B=262144, L=64),
        # a stored population through the notations
        dict(name="convert", kind="convert", B=50001, L=48),
        # a round of the online warm start: screened starts, then one training step
        dict(name="warm_round", kind="warm", B=2048, M=64, N=512),
    ]


def _log(rng, lo, hi):
    """Log-uniform whole number in [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval64", "multi", "readme", "ragged", "backtracking", "sample", "convert",
                       "warm"])
    if kind == "eval":
        grad = rng.choice(["", "C", "CX"])
        N = _log(rng, 30, 2000)
        M = rng.randint(16, 64)
        B = min(_log(rng, 30, 16384), 16384 * 1024 * 64 // (N * M))
        family = rng.choice(["readme", "general"]) if grad == "" and B <= 2000 else "general"
        return dict(kind="eval", tapes=family, B=B, M=M, N=N, n_x=1 if family == "readme" else rng.randint(1, 4),
                    grad=grad, dtype="f32")
    if kind == "eval64":
        return dict(kind="eval", tapes="general", B=_log(rng, 30, 1500), M=rng.randint(16, 64), N=_log(rng, 50, 1100),
                    n_x=rng.randint(1, 4), grad=rng.choice(["C", "CX"]), dtype="f64")
    if kind == "multi":
        return dict(kind="multi", tapes="general", B=_log(rng, 50, 2000), M=rng.randint(16, 48),
                    N=_log(rng, 50, 600), n_x=rng.randint(1, 4), K=rng.randint(2, 12))
    if kind == "readme":
        return dict(kind="fit", tapes="readme", B=_log(rng, 16, 8192), M=32, N=_log(rng, 40, 300),
                    max_iter=rng.choice([50, 100, 200]), search="strong_wolfe")
    if kind == "ragged":
        return dict(kind="fit", tapes="ragged", B=_log(rng, 100, 16384), M=rng.randint(24, 64), N=_log(rng, 60, 512),
                    max_iter=rng.choice([50, 100, 200]), search="strong_wolfe")
    if kind == "backtracking":
        return dict(kind="fit", tapes="ragged", B=_log(rng, 100, 8000), M=rng.randint(24, 64), N=_log(rng, 60, 512),
                    max_iter=rng.choice([50, 100]), search="backtracking")
    if kind == "sample":
        return dict(kind="sample", B=_log(rng, 1000, 1000000), L=rng.randint(24, 100))
    if kind == "convert":
        return dict(kind="convert", B=_log(rng, 1000, 200000), L=rng.randint(24, 64))
    return dict(kind="warm", B=_log(rng, 256, 8192), M=rng.randint(24, 64), N=_log(rng, 64, 1024))


# ---- plain torch interpreter (inputs' targets, screening, and the 64-bit outputs) --------

def _steps(ops):
    """Per node position: (code, rows of the batch with that code), as numpy."""
    for k in range(ops.shape[1]):
        col = ops[:, k]
        yield k, [(int(c), np.where(col == c)[0]) for c in np.unique(col) if c != 0]


def _forward(X, ops, ch, C):
    """(M, B, N) node values of tapes ops/ch (numpy) at X (N, n_x), constants C (B, M), in
    X's precision; NaN in the padding."""
    B, M = ops.shape
    vals = torch.full((M, B, X.shape[0]), float("nan"), dtype=X.dtype, device=X.device)
    dev = X.device
    for k, groups in _steps(ops):
        for code, rows in groups:
            r = torch.as_tensor(rows, device=dev)
            if code >= VAR:
                vals[k, r] = X[:, code - VAR]
                continue
            if code == LEARNABLE:
                vals[k, r] = C[r, k].unsqueeze(1).expand(-1, X.shape[0])
                continue
            a = vals[torch.as_tensor(ch[rows, k, 0], device=dev), r]
            if code >= ADD:
                b = vals[torch.as_tensor(ch[rows, k, 1], device=dev), r]
                v = {ADD: lambda: a + b, SUB: lambda: a - b, MUL: lambda: a * b,
                     DIV: lambda: torch.where(b == 0, torch.full_like(a, float("nan")), a / b)}[code]()
            else:
                v = {SIN: lambda: a.sin(), COS: lambda: a.cos(), EXP: lambda: a.exp(),
                     LOG: lambda: torch.where(a <= 0, torch.full_like(a, float("nan")), a.log())}[code]()
            vals[k, r] = v
    return vals


def _adjoint(vals, ops, ch, G):
    """(M, B, N) adjoints of every node for the output gradient G (M, B, N); a zero adjoint
    propagates nothing."""
    adj = G.clone()
    dev = vals.device
    for k, groups in reversed(list(_steps(ops))):
        for code, rows in groups:
            if code >= VAR or code == LEARNABLE:
                continue
            r = torch.as_tensor(rows, device=dev)
            c0 = torch.as_tensor(ch[rows, k, 0], device=dev)
            g, a = adj[k, r], vals[c0, r]
            o1 = c1 = None
            if code >= ADD:
                c1 = torch.as_tensor(ch[rows, k, 1], device=dev)
                b = vals[c1, r]
                o0, o1 = {ADD: lambda: (g, g), SUB: lambda: (g, -g), MUL: lambda: (g * b, g * a),
                          DIV: lambda: (g / b, -(g * a) / (b * b))}[code]()
            else:
                o0 = {SIN: lambda: g * a.cos(), COS: lambda: -g * a.sin(), EXP: lambda: g * vals[k, r],
                      LOG: lambda: g / a}[code]()
            zero = torch.zeros_like(g)
            adj[c0, r] += torch.where(g == 0, zero, o0)
            if o1 is not None:
                adj[c1, r] += torch.where(g == 0, zero, o1)
    return adj


def _chunks(B, M, N, limit=1 << 27):
    step = max(1, limit // max(1, M * N))
    return [(s, min(B, s + step)) for s in range(0, B, step)]


def _zero_denominator(ops, ch, X, C):
    """(B,) tapes with a denominator at or next to 0 at a point of X (numpy in and out)."""
    bad = np.zeros(ops.shape[0], bool)
    Xt = torch.as_tensor(np.asarray(X, np.float32), device=DEV)
    for s, e in _chunks(ops.shape[0], ops.shape[1], X.shape[0]):
        o, c = ops[s:e], ch[s:e]
        vals = _forward(Xt, o, c, torch.as_tensor(np.asarray(C[s:e], np.float32), device=DEV))
        b, k = np.where(o == DIV)
        den = vals[torch.as_tensor(c[b, k, 1], device=DEV), torch.as_tensor(b, device=DEV)]
        bad[s:e][b[(den.abs() < 1e-30).any(1).cpu().numpy()]] = True
    return bad


# ---- inputs ---------------------------------------------------------------------------

def _tape_batch(case, seed, X, C):
    """(ops, ch) of the case's tape family as numpy arrays."""
    B, M, n_x = case["B"], case["M"], X.shape[1]
    if case["tapes"] == "readme":
        wl = workloads.readme_fit(B=B, N=2, M=M, seed=seed)
        return wl.ops, wl.ch
    rng = np.random.default_rng([seed, 5])
    if case["tapes"] == "general":  # every point is screened: a gradient through a/0 is an error
        tb = tapes.generate(B, M, seed=seed + 1, mean_length=20.0, n_vars=n_x, p_const_leaf=0.2, X_screen=X,
                            C_screen=C, screen_fn=_zero_denominator)
    else:  # tapes to be fitted: lengths U[3, M], up to 8 constants
        Xs = X[rng.choice(X.shape[0], size=min(X.shape[0], 32), replace=False)]
        tb = tapes.generate(B, M, seed=seed + 1, lengths=rng.integers(3, M + 1, size=B),
                            const_counts=rng.integers(0, 9, size=B), n_vars=n_x, X_screen=Xs, C_screen=C,
                            no_exp_in_denominator=True, screen_fn=_zero_denominator)
    return tb.ops, tb.ch


def _eval_inputs(case, seed):
    """numpy X, ops, ch, C (B, M) or (B, M, K), the root positions, and the (B,) mask of the
    tapes that are finite and moderate at every point (no node above 100, no denominator or
    argument of a logarithm within 0.01 of 0): the ones a program lets into its loss, as a
    few exploding gradients would drown the others."""
    rng = np.random.default_rng([seed, 3])
    B, M, N = case["B"], case["M"], case["N"]
    dt = np.float64 if case.get("dtype") == "f64" else np.float32
    X = (2.0 * rng.standard_normal((N, 1)) if case["tapes"] == "readme" else
         rng.uniform(-3, 3, (N, case["n_x"]))).astype(dt)
    K = case.get("K", 1)
    C = rng.standard_normal((B, M, K)).astype(dt)
    ops, ch = _tape_batch(case, seed, X, C[:, :, 0])
    fine = np.ones(B, bool)
    if case.get("grad", "C"):
        Xt = torch.as_tensor(X.astype(np.float32), device=DEV)
        for s, e in _chunks(B, M, N):
            pad = torch.as_tensor((ops[s:e] == 0).T.copy(), device=DEV).unsqueeze(2)
            near = np.zeros(ops[s:e].shape, bool)  # nodes that must keep away from 0
            for code, child in ((DIV, 1), (LOG, 0)):
                b, k = np.where(ops[s:e] == code)
                near[b, ch[s:e][b, k, child]] = True
            far = torch.as_tensor(~near.T, device=DEV).unsqueeze(2)
            for j in range(K):
                v = _forward(Xt, ops[s:e], ch[s:e], torch.as_tensor(C[s:e, :, j].astype(np.float32), device=DEV))
                ok = ((v.abs() < 100) & ((v.abs() > 0.01) | far)) | pad
                fine[s:e] &= ok.all(2).all(0).cpu().numpy()
    root = np.maximum((ops != 0).sum(1) - 1, 0)
    return X, ops, ch, C, root, fine


def _root_gradient(case, seed, root, fine, dtype):
    """(B, M, N[, K]) gradient of a mean squared error: nonzero on the root rows of the fine
    tapes only."""
    B, M, N, K = case["B"], case["M"], case["N"], case.get("K", 0)
    shape = (B, M, N, K) if K else (B, M, N)
    g = torch.Generator(device=DEV).manual_seed(seed + 9)
    G = torch.zeros(shape, dtype=dtype, device=DEV)
    r = torch.randn((B,) + shape[2:], generator=g, device=DEV, dtype=torch.float32).to(dtype) * (2.0 / N)
    mask = torch.as_tensor(fine, device=DEV).view((B,) + (1,) * (len(shape) - 2))
    G[torch.arange(B, device=DEV), torch.as_tensor(root, device=DEV)] = r * mask
    return G


def _fit_inputs(case, seed):
    rng = np.random.default_rng([seed, 4])
    B, M, N = case["B"], case["M"], case["N"]
    C = rng.standard_normal((B, M)).astype(np.float32)
    if case["tapes"] == "readme":  # one target row for every expression
        X = (2.0 * rng.standard_normal((N, 1))).astype(np.float32)
        ops, ch = _tape_batch(case, seed, X, C)
        Y = np.tile((2.5 * np.cos(X[:, 0]) - 1.5).astype(np.float32), (B, 1))
        return X, Y, ops, ch, C
    X = rng.uniform(-3, 3, (N, 2)).astype(np.float32)
    ops, ch = _tape_batch(case, seed, X, C)
    Xt = torch.as_tensor(X, device=DEV)
    # targets: hidden expressions of the same family plus noise, where finite and moderate
    Y = torch.zeros((B, N), device=DEV)
    todo = np.arange(B)
    for attempt in range(6):
        hid = tapes.generate(todo.size, M, seed=seed + 100 + attempt, lengths=rng.integers(3, M + 1, size=todo.size),
                             const_counts=rng.integers(0, 9, size=todo.size), n_vars=2)
        hc = rng.standard_normal((todo.size, M)).astype(np.float32)
        left = []
        for s, e in _chunks(todo.size, M, N):
            v = _forward(Xt, hid.ops[s:e], hid.ch[s:e], torch.as_tensor(hc[s:e], device=DEV))
            r = torch.as_tensor((hid.ops[s:e] != 0).sum(1) - 1, device=DEV)
            y = v[r, torch.arange(e - s, device=DEV)]
            ok = (y.abs() < 1e4).all(1)
            idx = torch.as_tensor(todo[s:e], device=DEV)
            Y[idx[ok]] = y[ok]
            left.append(todo[s:e][~ok.cpu().numpy()])
        todo = np.concatenate(left)
        if todo.size == 0:
            break
    g = torch.Generator(device=DEV).manual_seed(seed + 8)
    return X, Y + 0.01 * torch.randn((B, N), generator=g, device=DEV), ops, ch, C


def _warm_inputs(case, seed):
    X, Y, ops, ch, C = _fit_inputs(dict(case, tapes="ragged"), seed)
    rng = np.random.default_rng([seed, 6])
    n = (ops == LEARNABLE).sum(1)
    mask = (np.arange(8)[None, :] < n[:, None]).astype(np.float32)
    return X, Y, ops, ch, C, (rng.standard_normal((case["B"], 8)) * mask).astype(np.float32), mask


def _cuda(a):
    return a if isinstance(a, torch.Tensor) else torch.as_tensor(a, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": int(seed)}
    if kind in ("eval", "multi"):
        X, ops, ch, C, root, fine = _eval_inputs(case, seed)
        grad = case.get("grad", "C")
        s.update(X=_cuda(X), ops=_cuda(ops), ch=_cuda(ch), C=_cuda(C if kind == "multi" else C[:, :, 0].copy()))
        if grad:
            s["G"] = _root_gradient(case, seed, root, fine, s["X"].dtype)
            s["C"].requires_grad_(True)
            s["X"].requires_grad_("X" in grad)
    elif kind == "fit":
        for name, a in zip(("X", "Y", "ops", "ch", "C"), _fit_inputs(case, seed)):
            s[name] = _cuda(a)
    elif kind == "warm":
        for name, a in zip(("X", "Y", "ops", "ch", "C", "target", "mask"), _warm_inputs(case, seed)):
            s[name] = _cuda(a)
        s["net"] = warmstart.WarmStartMLP(DEV, seed=seed % 1000, n_vars=2)
    else:
        s["pcfg"] = sr.ProbabilisticContextFreeGrammar(workloads.SEARCH_GRAMMAR, "E", case["L"], 3, torch.device(DEV))
        if kind == "convert":
            torch.manual_seed(seed)
            s["infix"] = s["pcfg"].sample_infix(case["B"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("eval", "multi"):
        fn = sr.evaluation.evaluate if kind == "eval" else sr.evaluation.evaluate_multiple
        grad = case.get("grad", "C")
        if not grad:
            with torch.no_grad():
                return {"cache": fn(s["X"], s["ops"], s["ch"], s["C"])}
        cache = fn(s["X"], s["ops"], s["ch"], s["C"])
        grads = torch.autograd.grad(cache, [s["C"], s["X"]] if "X" in grad else [s["C"]], s["G"])
        return {"cache": cache.detach(), "grads": list(grads)}
    if kind == "fit":
        if case["tapes"] == "readme":
            C, Y = sr.optimize(s["X"], s["Y"], s["ops"], s["ch"], s["C"], max_iter=case["max_iter"],
                               line_search_fn=case["search"])
            return {"C": C, "Y": Y}
        r = sr.optimize_ex(s["X"], s["Y"], s["ops"], s["ch"], s["C"], max_iter=case["max_iter"],
                           line_search_fn=case["search"], raise_errors=False)
        return {"C": r.C, "Y": r.Y, "iters": r.iters, "loss": r.loss, "evals": r.evals}
    if kind == "sample":
        torch.manual_seed(s["seed"])  # a reproducible search seeds its draws
        ops, ch = s["pcfg"].sample(case["B"])
        return {"ops": ops, "ch": ch}
    if kind == "convert":
        p = s["pcfg"]
        post = p.infix_to_postfix(s["infix"])
        pre = p.infix_to_prefix(s["infix"])
        return {"postfix": post, "children": p.get_postfix_children(post),
                "infix": p.postfix_to_infix(post, 2 * case["L"]), "prefix": pre,
                "from_prefix": p.prefix_to_postfix(pre)}
    net = s["net"]
    C = warmstart.gated_warm_start(net, s["X"], s["Y"], s["ops"], s["ch"], s["C"])
    loss = net.train_batch(s["ops"], s["X"], s["Y"], s["target"], s["mask"], lr=1e-3, weight_decay=1e-4)
    return {"C": C, "loss": loss, "w": dict(net.w), "b": dict(net.b)}


def work(case):
    kind, B = case["kind"], case["B"]
    M, N = case.get("M", 0), case.get("N", 0)
    if kind in ("eval", "multi"):
        K, e = case.get("K", 1), 8 if case.get("dtype") == "f64" else 4
        grad = case.get("grad", "C")
        ops = 10.0 * min(20, M) / 2  # operations of the average tape at one point, forward
        b = 24.0 * B * M + e * (N * case["n_x"] + B * M * K + B * M * N * K)
        if grad:
            b += e * (B * M * N * K + B * M * K + (N * case["n_x"] if "X" in grad else 0))
        return {"bytes": b, "flops": (3.0 if grad else 1.0) * ops * B * N * K}
    if kind == "fit":
        clos = CLOSURES["backtracking" if case["search"] == "backtracking" else case["tapes"]] * case["max_iter"] / (
            200.0 if case["tapes"] == "ragged" and case["search"] == "strong_wolfe" else 100.0)
        per = FLOPS_PER_POINT[case["tapes"]] * (M / 64.0 if case["tapes"] == "ragged" else 1.0)
        return {"bytes": 24.0 * B * M + 8.0 * B * M + 8.0 * B * N, "flops": clos * per * B * N}
    if kind == "sample":
        return {"bytes": 24.0 * B * case["L"], "flops": 0.0}
    if kind == "convert":
        return {"bytes": 8.0 * B * case["L"] * (1 + 1 + 2 + 2 + 1 + 1), "flops": 0.0}
    w = 64 * 64 + 256 * 128 + 2 * 256 * 256 + 64 * 256
    # one forward for the starts, forward + backward for the step; the screening of two starts
    return {"bytes": 4.0 * B * N + 32.0 * B * M + 12.0 * B * M + 24.0 * w,
            "flops": 8.0 * B * w + 2 * 65.0 * M / 64.0 * B * N + 4.0 * 60 * B * N}


# ---- 64-bit outputs -------------------------------------------------------------------

def _exact_eval(case, seed):
    X, ops, ch, C, root, fine = _eval_inputs(case, seed)
    K, multi = case.get("K", 1), case["kind"] == "multi"
    B, M, N, n_x = case["B"], case["M"], case["N"], X.shape[1]
    grad = case.get("grad", "C")
    Xt = torch.as_tensor(X.astype(np.float64), device=DEV)
    Ct = torch.as_tensor(C.astype(np.float64), device=DEV)
    big = 3.4028235e38 if case.get("dtype") != "f64" else float("inf")
    cache = torch.empty((B, M, N, K), dtype=torch.float64, device=DEV)
    gC = torch.zeros((B, M, K), dtype=torch.float64, device=DEV)
    gX = torch.zeros((N, n_x), dtype=torch.float64, device=DEV)
    G = _root_gradient(case, seed, root, fine, torch.float64 if case.get("dtype") == "f64" else torch.float32) \
        if grad else None
    is_c = torch.as_tensor(ops == LEARNABLE, device=DEV)
    for s, e in _chunks(B, M, N, 1 << 26):
        for j in range(K):
            v = _forward(Xt, ops[s:e], ch[s:e], Ct[s:e, :, j])
            c = v.permute(1, 0, 2)
            # values beyond the working precision's range are infinite there
            cache[s:e, :, :, j] = torch.where(c.abs() > big, torch.sign(c) * float("inf"), c)
            if grad:
                g = (G[s:e, :, :, j] if multi else G[s:e]).double().permute(1, 0, 2)
                adj = _adjoint(v, ops[s:e], ch[s:e], g)
                gC[s:e, :, j] = torch.where(is_c[s:e], adj.sum(2).T, torch.zeros((), dtype=torch.float64, device=DEV))
                for x in range(n_x):
                    rows, pos = np.where(ops[s:e] == VAR + x)
                    gX[:, x] += adj[torch.as_tensor(pos, device=DEV), torch.as_tensor(rows, device=DEV)].sum(0)
    if not multi:
        cache, gC = cache[..., 0], gC[..., 0]
    if not grad:
        return {"cache": cache}
    return {"cache": cache, "grads": [gC, gX] if "X" in grad else [gC]}


def _exact_step(case, seed):
    """The training step of the warm start in 64 bits without any rounding between layers."""
    X, Y, ops, ch, C, target, mask = (_cuda(a) for a in _warm_inputs(case, seed))
    net = warmstart.WarmStartMLP(DEV, seed=seed % 1000, n_vars=2)  # only its initial values are used
    w = {k: v.double() for k, v in net.w.items()}
    b = {k: v.double() for k, v in net.b.items()}
    X, Y, target, mask = X.double(), Y.double(), target.double(), mask.double()
    B = ops.shape[0]
    hist = torch.zeros((B, 64), dtype=torch.float64, device=DEV)
    tok = torch.where((ops >= 0) & (ops < 64), ops, torch.full_like(ops, 63))
    hist.scatter_add_(1, tok, (ops != 0).double())
    hist /= (ops != 0).sum(1, keepdim=True).clamp(min=1)
    phi = 2.0 ** 0.5 * torch.cos(X @ net.omega.double().T + net.beta.double())
    mu = Y.mean(1, keepdim=True)
    d = Y - mu
    sd = (d * d).mean(1).sqrt()
    z = d / sd.unsqueeze(1)
    f = torch.cat([torch.asinh(mu), (sd + 1e-3).log().unsqueeze(1), (z ** 3).mean(1, keepdim=True).clamp(-50, 50),
                   torch.asinh((z ** 4).mean(1, keepdim=True) - 3.0), z @ phi / Y.shape[1]], 1)
    f = torch.where(torch.isfinite(f), f, torch.zeros_like(f))
    x0 = torch.cat([hist @ w["E"].T, f, torch.zeros_like(f)], 1)
    h, acts = x0, [x0]
    for n in ("W1", "W2", "W3"):
        h = (h @ w[n].T + b[n]).clamp(min=0)
        acts.append(h)
    out = (h @ w["W4"].T + b["W4"])[:, :8]
    diff = (out - target) * (mask > 0)
    loss = (mask * diff * diff).sum(1)
    dz = torch.zeros((B, 64), dtype=torch.float64, device=DEV)
    dz[:, :8] = 2.0 * mask * diff / B
    gw = {}
    for i, n in ((3, "W4"), (2, "W3"), (1, "W2"), (0, "W1")):
        gw[n] = dz.T @ acts[i]
        dz = dz @ w[n]
        if i:
            dz = dz * (acts[i] > 0)
    gw["E"] = dz[:, :64].T @ hist
    for n in w:  # the first Adam step: m / (1 - beta1) = g, v / (1 - beta2) = g^2
        w[n] = w[n] - 1e-3 * (gw[n] / (gw[n].abs() + 1e-8) + 1e-4 * w[n])
    # the biases start at 0, so their first step is the sign of a gradient that bf16 rounding
    # may flip: no value in 64 bits to hold them to
    return {"C": None, "loss": loss, "w": w, "b": {n: None for n in b}}


def exact(case, seed):
    if case["kind"] in ("eval", "multi"):
        return _exact_eval(case, seed)
    if case["kind"] == "warm":
        return _exact_step(case, seed)
    return None  # whole numbers, or the end of an iteration that rounding steers
