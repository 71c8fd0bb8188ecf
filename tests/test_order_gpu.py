"""The work order and the error-word summary against numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column", [0, 1])
@pytest.mark.parametrize("B,M", [(1, 1), (31, 3), (1023, 64), (1024, 64), (1025, 64), (5000, 4095), (70001, 48)])
def test_tape_order_lists_every_tape_by_falling_length(B, M, column):
    from cudasymbolicregression_gb300 import _lib
    rng = np.random.default_rng([B, M, column])
    meta = np.zeros((B, 4), np.int32)
    meta[:, column] = rng.integers(0, M + 1 - column, size=B)
    m = torch.as_tensor(meta).cuda()
    order = torch.full((B,), -1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().sr_tape_order(_lib.ptr(m), B, M, column, _lib.ptr(order), _lib.stream_ptr(m.device)), "order")
    o = order.cpu().numpy()
    assert np.array_equal(np.sort(o), np.arange(B))
    assert (np.diff(meta[o, column]) <= 0).all()


@pytest.mark.parametrize("n", [0, 1, 255, 2048, 2049, 300001])
def test_any_nonzero(n):
    from cudasymbolicregression_gb300 import _lib
    w = torch.zeros(n, dtype=torch.int64, device="cuda")
    assert not _lib.any_nonzero(w)
    for i in {0, n // 2, n - 1} if n else ():
        w[i] = 1 << 40
        assert _lib.any_nonzero(w)
        w[i] = 0


@pytest.mark.parametrize("M", [1, 33, 64])
@pytest.mark.parametrize("B", [1, 8, 9, 9728, 9729, 30001])
def test_compile_summary_is_the_maximum_over_tapes(B, M):
    """Batches below, at and above the tapes that the grid's warps take at once; the longest
    tape first, last or in between."""
    from cudasymbolicregression_gb300 import tape, tapes
    tb = tapes.generate(B, M, seed=B + M, mean_length=min(5, M), n_vars=2, p_const_leaf=0.5)
    ops = tb.ops.copy()
    for at in {0, B // 2, B - 1}:
        rows = ops.copy()
        rows[at] = 1  # constants only: the root is the last of them
        want = ((rows != 0) * np.arange(1, M + 1)).max(), (rows != 0).sum(1).max(), (rows == 1).sum(1).max()
        ch = tb.ch.copy()
        ch[at] = -1
        c = tape.compile_tapes(torch.as_tensor(rows).cuda(), torch.as_tensor(ch).cuda(), 2)
        assert (c.max_len, c.max_root, c.max_consts) == want


@pytest.mark.parametrize("B,M", [(8192, 64), (8193, 64), (65535, 1), (65536, 4095), (262145, 64), (1000003, 33)])
def test_tape_order_over_the_shares_of_a_cluster(B, M):
    test_tape_order_lists_every_tape_by_falling_length(B, M, 0)
