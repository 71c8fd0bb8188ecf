"""The forward's rows and the NaN padding where their forms change, bit for bit against the
oracle: more variables than rows (by number, packed, a row per leaf), tapes whose operators fill
the row table at four, two or one value per lane, few points, and padding ranges around one bulk
copy."""
import numpy as np
import pytest
import torch

import oracle
from test_eval_paths_gpu import _bits_equal, _tapes

pytestmark = pytest.mark.gpu


def _check(ops, ch, X, C, dtype):
    import cudasymbolicregression_gb300 as sr
    K = C.shape[2] if C.ndim == 3 else 0
    fn = sr.evaluation.evaluate_multiple if K else sr.evaluation.evaluate
    out = fn(*(torch.as_tensor(a).cuda() for a in (X, ops, ch, C))).cpu().numpy()
    for k in range(max(K, 1)):
        want = oracle.eval_fwd(X, ops, ch, C[..., k] if K else C, dtype=dtype, kernel_math=dtype == np.float32)
        assert _bits_equal(np.ascontiguousarray(out[..., k]) if K else out, want), f"set {k}"


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nx", [16, 17, 40, 200])
@pytest.mark.parametrize("N,K", [(31, 0), (64, 0), (65, 0), (300, 0), (20, 3), (50, 3)])
def test_variables_of_a_tape(nx, N, K, dtype):
    rng = np.random.default_rng([nx, N, K])
    unary = (10, 27) if dtype == np.float32 else (14, 27)
    parts = [_tapes(form, rng, 24, nx, unary) for form in ("stack", "dag")]
    ops, ch = (np.concatenate(a) for a in zip(*parts))
    ops[ops == 1] = 50 + rng.integers(0, nx, int((ops == 1).sum()))  # variables only: up to 32 distinct
    X = rng.uniform(-1, 1, (N, nx)).astype(dtype)
    C = rng.uniform(-1, 1, ops.shape + ((K,) if K else ())).astype(dtype)
    _check(ops, ch, X, C, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N", [32, 33, 64, 65, 200])
@pytest.mark.parametrize("n_ops", [1, 12, 13, 16, 17, 24, 26, 27, 32, 33, 63])
def test_operators_out_of_stack_order(n_ops, N, dtype):
    """Each operator takes the one before it and an earlier node, so every one needs a row."""
    rng = np.random.default_rng([n_ops, N])
    B, M = 5, 64
    ops, ch = np.zeros((B, M), np.int64), np.full((B, M, 2), -1, np.int64)
    ops[:, 0] = 50
    for k in range(1, n_ops + 1):
        ops[:, k] = rng.choice((40, 41), B)
        ch[:, k, 0], ch[:, k, 1] = k - 1, rng.integers(0, k, B)
    X = rng.uniform(-1, 1, (N, 1)).astype(dtype)
    _check(ops, ch, X, np.zeros((B, M), dtype), dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("B,M,N", [(1, 3, 1), (33, 5, 3), (5000, 9, 7), (700, 17, 60), (160, 9, 128), (5000, 9, 129),
                                   (40, 9, 1001)])
def test_padding_ranges(B, M, N, dtype):
    from cudasymbolicregression_gb300 import tapes
    rng = np.random.default_rng([B, M, N])
    tb = tapes.generate(B, M, seed=B, lengths=rng.integers(1, M + 1, B), n_vars=2, unary=(27,), binary=(40, 41))
    X = rng.uniform(-1, 1, (N, 2)).astype(dtype)
    _check(tb.ops, tb.ch, X, rng.uniform(-1, 1, (B, M)).astype(dtype), dtype)
