"""The evaluation kernels' table layouts at their edges, bit for bit against the oracle.

Tapes whose child table is that of an evaluation stack hold one 16-byte-wide row per
waiting operator result; tapes that share or skip subtrees, need more rows than the table
has or use more variables than it holds take one row per node.  Both have to give the
oracle's cache and constant gradient bit for bit, at point counts around a lane pack (4
points) and a pass (128), and with constant sets taken in one pass (K = 3) or one by one
(K = 65).
"""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

UNARY, BINARY = (10, 11, 14, 27), (40, 41, 42)  # sin cos square neg; + - *


def _bits_equal(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    u = np.uint32 if a.dtype == np.float32 else np.uint64
    return np.array_equal(na, nb) and np.array_equal(a.view(u)[~na], b.view(u)[~nb])


def _tapes(form, rng, B, nx, unary):
    """(ops, ch) of one form of child table."""
    from cudasymbolicregression_gb300 import tapes
    if form == "stack":
        tb = tapes.generate(B, 64, seed=int(rng.integers(1 << 30)), lengths=rng.integers(1, 65, size=B), n_vars=nx,
                            unary=unary, binary=BINARY, p_const_leaf=0.4)
        return tb.ops, tb.ch
    M = 64
    ops = np.zeros((B, M), np.int64)
    ch = np.full((B, M, 2), -1, np.int64)
    for b in range(B):
        if form == "comb":  # u(x) u(x) ... + + +: up to 21 operator results wait at once
            n = int(rng.integers(1, 22))
            for i in range(n):
                ops[b, 2 * i] = 1 if rng.random() < 0.5 else 50 + rng.integers(nx)
                ops[b, 2 * i + 1] = rng.choice(unary)
                ch[b, 2 * i + 1, 0] = 2 * i
            top = 2 * n - 1
            for i in range(n - 1):
                k = 2 * n + i
                ops[b, k] = rng.choice(BINARY)
                ch[b, k] = (2 * (n - 2 - i) + 1, top)
                top = k
        else:  # "dag": any earlier nodes as children, so shared and unused subtrees
            L = int(rng.integers(2, M + 1))
            for k in range(L):
                r = rng.random()
                if k == 0 or r < 0.35:
                    ops[b, k] = 1 if rng.random() < 0.4 else 50 + rng.integers(nx)
                elif r < 0.6:
                    ops[b, k] = rng.choice(unary)
                    ch[b, k, 0] = rng.integers(k)
                else:
                    ops[b, k] = rng.choice(BINARY)
                    ch[b, k] = rng.integers(k, size=2)
    return ops, ch


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("form,nx", [("stack", 3), ("stack", 17), ("comb", 2), ("dag", 2)])
@pytest.mark.parametrize("B,N,K", [(37, 1, 1), (37, 31, 1), (20, 128, 1), (20, 129, 1), (5, 1000, 1), (300, 260, 1),
                                   (12, 33, 3), (6, 128, 8), (3, 7, 65)])
def test_table_layouts_bit_identical(dtype, form, nx, B, N, K):
    import cudasymbolicregression_gb300 as sr
    rng = np.random.default_rng([B, N, K, nx])
    # float64 sin and cos are CUDA's, not the oracle's: exact operators only
    ops, ch = _tapes(form, rng, B, nx, UNARY if dtype == np.float32 else (14, 27))
    X = rng.uniform(-1, 1, (N, nx)).astype(dtype)
    C = rng.uniform(-1, 1, ops.shape + (K,)).astype(dtype)
    single = K == 1
    fn = sr.evaluation.evaluate if single else sr.evaluation.evaluate_multiple
    Ct = torch.as_tensor(C[..., 0].copy() if single else C).cuda().requires_grad_(True)
    out = fn(torch.as_tensor(X).cuda(), torch.as_tensor(ops).cuda(), torch.as_tensor(ch).cuda(), Ct)
    got = out.detach().cpu().numpy().reshape(ops.shape + (N, K))
    for k in sorted({0, K // 2, K - 1}):
        want = oracle.eval_fwd(X, ops, ch, C[..., k], dtype=dtype, kernel_math=dtype == np.float32)
        assert _bits_equal(np.ascontiguousarray(got[..., k]), want), f"set {k}"
    if dtype != np.float32:
        return  # the oracle states the adjoint's summation order in float32
    gout = rng.uniform(-1, 1, got.shape).astype(dtype)
    gout[np.isnan(got)] = 0.0
    out.backward(torch.as_tensor(gout.reshape(out.shape)).cuda())
    gc = Ct.grad.cpu().numpy().reshape(ops.shape + (K,))
    for k in sorted({0, K // 2, K - 1}):
        want, err = oracle.eval_gc_kernel_order(X, ops, ch, C[..., k], np.ascontiguousarray(gout[..., k]))
        assert err == 0
        assert _bits_equal(np.ascontiguousarray(gc[..., k]), want), f"set {k}"
