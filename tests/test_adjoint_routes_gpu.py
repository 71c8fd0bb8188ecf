"""The adjoint's kernels, each at batches that reach it: the sweep over stack rows, its general
sweeps, and the staged kernel for tapes out of stack order, large batches, few points and calls
without a cache.  grad_C bit for bit against the oracle's order of sums; grad_X exactly, on
whole numbers whose sums float32 holds."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _tapes(form, rng, B, M, nx):
    """Short tapes of + - * neg (at most one *), as (ops, ch)."""
    ops = np.zeros((B, M), np.int64)
    ch = np.full((B, M, 2), -1, np.int64)
    for b in range(B):
        if form == "comb":  # leaves under neg first: more results wait than the row table holds
            n = int(rng.integers(1, (M + 1) // 3 + 1))
            for i in range(n):
                ops[b, 2 * i], ops[b, 2 * i + 1] = (1 if rng.random() < 0.5 else 50 + rng.integers(nx)), 27
                ch[b, 2 * i + 1, 0] = 2 * i
            top = 2 * n - 1
            for i in range(n - 1):
                k = 2 * n + i
                ops[b, k], ch[b, k], top = rng.choice((40, 41)), (2 * (n - 2 - i) + 1, top), k
            continue
        stack, times = [], 0
        L = int(rng.integers(1, M + 1))
        for k in range(L):
            u = rng.random()
            if form == "dag" and k and u > 0.4:  # any earlier nodes, the same one twice among them
                ops[b, k] = rng.choice((27, 40, 41))
                ch[b, k, 0] = rng.integers(k)
                if ops[b, k] != 27:
                    ch[b, k, 1] = ch[b, k, 0] if u > 0.9 else rng.integers(k)
            elif form != "dag" and len(stack) > 1 and u > 0.5:
                ops[b, k] = 42 if times == 0 and u > 0.9 else rng.choice((40, 41))
                times += ops[b, k] == 42
                ch[b, k, 1], ch[b, k, 0] = stack.pop(), stack.pop()
                stack.append(k)
            elif form != "dag" and stack and u > 0.4:
                ops[b, k], ch[b, k, 0] = 27, stack.pop()
                stack.append(k)
            else:
                ops[b, k] = 1 if rng.random() < 0.4 else 50 + rng.integers(nx)
                stack.append(k)
    return ops, ch


@pytest.mark.parametrize("form,M", [("stack", 9), ("dag", 9), ("comb", 47)])
@pytest.mark.parametrize("B,N,K", [(40, 65, 1), (40, 300, 1), (40, 64, 1), (33, 64, 4), (33, 65, 5), (6000, 65, 1),
                                   (6000, 130, 2), (29200, 65, 1), (29200, 1, 1)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_every_route(form, M, B, N, K, dtype):
    from cudasymbolicregression_gb300 import _lib
    from cudasymbolicregression_gb300.tape import compile_tapes
    if B * M * N * K > 1 << 27:
        B //= 8
    rng = np.random.default_rng([B, M, N, K])
    nx = 3
    few = min(B, 400)  # the batch repeats these
    ops, ch = (np.resize(a, (B,) + a.shape[1:]) for a in _tapes(form, rng, few, M, nx))
    X = rng.integers(-2, 3, (N, nx)).astype(dtype)
    C = rng.integers(-2, 3, (B, M, K)).astype(dtype)
    gout = rng.integers(-1, 2, (B, M, N, K)).astype(dtype)
    gout[ops == 0] = 0
    d = {k: torch.as_tensor(v).cuda() for k, v in dict(X=X, C=C, g=gout, ops=ops, ch=ch).items()}
    tp = compile_tapes(d["ops"], d["ch"], nx)
    L, p, st = _lib.lib(), _lib.ptr, _lib.stream_ptr(d["X"].device)
    sfx = "f32" if dtype == np.float32 else "f64"
    cache = torch.empty_like(d["g"])
    _lib.check(getattr(L, "sr_eval_forward_multi_" + sfx)(
        p(d["X"]), N, nx, p(tp.desc), p(tp.meta), p(tp.order), B, M, tp.max_len, p(d["C"]), *d["C"].stride(), K,
        p(cache), st), "forward")
    want_x, want_c = np.zeros((N, nx)), []
    for k in range(K):
        g = np.ascontiguousarray(gout[..., k])
        gc, gx, err = oracle.eval_bwd(X.astype(np.float64), ops, ch, C[..., k].astype(np.float64), g.astype(np.float64),
                                      dtype=np.float64)
        assert err == 0 and np.abs(gx).max() < 1 << 24 and np.abs(gc).max() < 1 << 24
        want_x += gx
        want_c.append(gc)
    for c in (cache, None):
        gC, gX = torch.full_like(d["C"], 7.0), torch.zeros_like(d["X"])
        status = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        _lib.check(getattr(L, "sr_eval_backward_multi_" + sfx)(
            p(d["X"]), N, nx, p(tp.desc), p(tp.meta), p(tp.order), B, M, tp.max_len, p(d["C"]), *d["C"].stride(), K,
            p(c), p(d["g"]), p(gC), p(gX), p(status), st), "backward")
        assert int(status) == 0
        # every sum is a whole number that the type holds, so its order does not matter
        np.testing.assert_array_equal(gC.cpu().numpy(), np.stack(want_c, -1))
        np.testing.assert_array_equal(gX.cpu().numpy(), want_x)


@pytest.mark.parametrize("B,N", [(40, 129), (1300, 65), (1300, 160), (29200, 65)])
@pytest.mark.parametrize("form,M", [("dag", 12), ("comb", 62), ("stack", 12)])
def test_constant_gradients_bit_identical_on_every_route(form, M, B, N):
    """Values with rounding: the sums have the oracle's order whichever kernel takes a tape."""
    import cudasymbolicregression_gb300 as sr
    if B * M * N > 1 << 27:
        B //= 8
    rng = np.random.default_rng([B, N, M])
    ops, ch = (np.resize(a, (B,) + a.shape[1:]) for a in _tapes(form, rng, min(B, 300), M, 2))
    X = rng.uniform(-1, 1, (N, 2)).astype(np.float32)
    C = rng.uniform(-1, 1, (B, M)).astype(np.float32)
    gout = rng.uniform(-1, 1, (B, M, N)).astype(np.float32)
    gout[ops == 0] = 0
    Ct = torch.as_tensor(C).cuda().requires_grad_(True)
    out = sr.evaluation.evaluate(torch.as_tensor(X).cuda(), torch.as_tensor(ops).cuda(), torch.as_tensor(ch).cuda(), Ct)
    out.backward(torch.as_tensor(gout).cuda())
    want, err = oracle.eval_gc_kernel_order(X, ops, ch, C, gout)
    assert err == 0
    np.testing.assert_array_equal(Ct.grad.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("dtype,L,cached", [(np.float32, 785, True), (np.float32, 784, False), (np.float32, 1300, True),
                                            (np.float64, 417, False), (np.float64, 417, True)])
@pytest.mark.parametrize("N", [3, 70])
@pytest.mark.parametrize("n_x", [1, 16])
def test_longest_tapes_that_the_tables_hold(dtype, L, cached, N, n_x):
    """Chains as long as the tables of the kernels hold, grad_X of up to 16 variables included."""
    from cudasymbolicregression_gb300 import _lib
    from cudasymbolicregression_gb300.tape import compile_tapes
    ops, ch = np.full((3, L), 27, np.int64), np.full((3, L, 2), -1, np.int64)
    ops[:, :3], ch[:, 2] = (50 + n_x - 1, 1, 42), (0, 1)
    ch[:, 3:, 0] = np.arange(2, L - 1)
    rng = np.random.default_rng(L + N)
    X, C = rng.integers(-2, 3, (N, n_x)).astype(dtype), rng.integers(-2, 3, (3, L)).astype(dtype)
    gout = rng.integers(-1, 2, (3, L, N)).astype(dtype)
    d = {k: torch.as_tensor(v).cuda() for k, v in dict(X=X, C=C, g=gout, ops=ops, ch=ch).items()}
    tp = compile_tapes(d["ops"], d["ch"], n_x)
    lib, p, st = _lib.lib(), _lib.ptr, _lib.stream_ptr(d["X"].device)
    sfx = "f32" if dtype == np.float32 else "f64"
    cache, gC, gX = torch.empty_like(d["g"]), torch.empty_like(d["C"]), torch.zeros_like(d["X"])
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = (p(d["X"]), N, n_x, p(tp.desc), p(tp.meta), p(tp.order), 3, L, tp.max_len, p(d["C"]), L, 1)
    _lib.check(getattr(lib, "sr_eval_forward_" + sfx)(*args, p(cache), st), "forward")
    _lib.check(getattr(lib, "sr_eval_backward_" + sfx)(*args, p(cache) if cached else None, p(d["g"]), p(gC), p(gX),
                                                     p(status), st), "backward")
    want_c, want_x, err = oracle.eval_bwd(X, ops, ch, C, gout, dtype=np.float64)
    assert err == 0 and int(status) == 0
    np.testing.assert_array_equal(gC.cpu().numpy(), want_c)
    np.testing.assert_array_equal(gX.cpu().numpy(), want_x)
