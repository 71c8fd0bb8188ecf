"""The fit kernel's row assignment and two-chunk passes at their edges, bit for bit.

Values that the reverse sweep does not read share rows with its adjoints, and a warp with
a second chunk works on two chunks at once unless a constant has several parents (its
sums then need one chunk's terms before the next chunk's).  Tapes that share and skip
subtrees, at point counts around one and two chunks per warp, must give the oracle's fit.
"""
import numpy as np
import pytest
import torch

import oracle
from test_fit_exact_gpu import assert_bit_identical, cuda

pytestmark = pytest.mark.gpu


def _dags(rng, B, M, nx, share_constants):
    """Tapes whose operators take any earlier operators and variables (shared and unused
    subtrees); a constant gets one parent unless share_constants."""
    ops = np.zeros((B, M), np.int64)
    ch = np.full((B, M, 2), -1, np.int64)
    for b in range(B):
        L = int(rng.integers(1, M + 1))
        free = []  # constants without a parent yet
        for k in range(L):
            r = rng.random()
            if k == 0 or (r < 0.4 and k < L - 1):
                ops[b, k] = 1 if rng.random() < 0.4 else 50 + rng.integers(nx)
                if ops[b, k] == 1:
                    free.append(k)
                continue
            pool = [i for i in range(k) if share_constants or ops[b, i] != 1 or i in free]
            if not pool:
                ops[b, k] = 50
                continue
            unary = rng.random() < 0.4
            ops[b, k] = rng.choice((10, 12, 14, 27) if unary else (40, 41, 42))
            for j in range(1 if unary else 2):
                c = int(pool[rng.integers(len(pool))])
                if j == 1 and not share_constants and ops[b, c] == 1 and c == ch[b, k, 0]:
                    c = int(next((i for i in pool if ops[b, i] != 1), -1))
                    if c < 0:
                        ops[b, k], ch[b, k, 1] = 27, -1
                        break
                ch[b, k, j] = c
                if c in free:
                    free.remove(c)
    return ops, ch


@pytest.mark.parametrize("share_constants", [False, True])
@pytest.mark.parametrize("N,W", [(32, 1), (33, 1), (64, 1), (65, 1), (100, 2), (129, 2), (250, 4)])
def test_shared_subtrees_bit_identical(N, W, share_constants):
    import cudasymbolicregression_gb300 as sr
    rng = np.random.default_rng([N, W, share_constants])
    B, M = 96, 20
    ops, ch = _dags(rng, B, M, 2, share_constants)
    X = rng.uniform(-1, 1, (N, 2)).astype(np.float32)
    Y = rng.uniform(-1, 1, (B, N)).astype(np.float32)
    C = rng.uniform(-1, 1, (B, M)).astype(np.float32)
    o = oracle.optimize(X, Y, ops, ch, C, max_iter=40, dot_mode=2, warps=W, points_per_lane=1)
    r = sr.optimize_ex(cuda(X), cuda(Y), cuda(ops), cuda(ch), cuda(C), max_iter=40, warps_per_block=W,
                       points_per_lane=1, raise_errors=False)
    assert_bit_identical(r, o, f"N={N} W={W} shared={share_constants}")
    losses = sr.optimization.screen_starts(cuda(X), cuda(Y), cuda(ops), cuda(ch), cuda(C)[None])[:, 0].cpu().numpy()
    first = oracle.optimize(X, Y, ops, ch, C, max_iter=0, dot_mode=2, warps=W, points_per_lane=1)["loss"]
    fine = np.isfinite(first)
    np.testing.assert_allclose(losses[fine], first[fine], rtol=1e-6)


@pytest.mark.parametrize("L", [741, 743, 781])
def test_longest_tapes_that_the_tables_hold(L):
    """Chains of operators, whose tables take the most shared memory: up to 781 nodes fit."""
    import cudasymbolicregression_gb300 as sr
    from parity import fit_bits_differ, oracle_fit_like
    rng = np.random.default_rng(L)
    B, N = 3, 40
    ops = np.zeros((B, L), np.int64)
    ch = np.full((B, L, 2), -1, np.int64)
    ops[:, :3], ch[:, 2] = (50, 1, 40), (0, 1)
    ops[:, 3:] = rng.choice((10, 11, 27), size=(B, L - 3))
    ch[:, 3:, 0] = np.arange(2, L - 1)
    X = rng.uniform(-1, 1, (N, 1)).astype(np.float32)
    Y = rng.uniform(-1, 1, (B, N)).astype(np.float32)
    C = rng.uniform(-1, 1, (B, L)).astype(np.float32)
    r = sr.optimize_ex(cuda(X), cuda(Y), cuda(ops), cuda(ch), cuda(C), max_iter=3, raise_errors=False)
    assert not fit_bits_differ(r, oracle_fit_like(r, X, Y, ops, ch, C, max_iter=3)).any()
