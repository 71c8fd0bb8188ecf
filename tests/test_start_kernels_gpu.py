"""Placing predicted constants and picking starts, against torch indexing."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,M", [(1, 1), (7, 31), (8, 32), (9, 33), (300, 70)])
def test_place_and_pick(B, M):
    from cudasymbolicregression_gb300 import _lib
    rng = np.random.default_rng([B, M])
    L, st = _lib.lib(), _lib.stream_ptr(torch.device("cuda"))
    ops = torch.as_tensor(rng.choice([0, 1, 1, 40, 50], size=(B, M))).cuda()
    C = torch.as_tensor(rng.standard_normal((B, M)).astype(np.float32)).cuda()
    pred = torch.as_tensor((20 * rng.standard_normal((B, 8))).astype(np.float32)).cuda()
    pred[0, 0] = float("nan")
    want = C.clone()
    is_c = ops == 1
    rank = torch.cumsum(is_c.to(torch.int32), 1) - 1
    sel = is_c & (rank < 8)
    rows = torch.arange(B, device="cuda").unsqueeze(1).expand_as(ops)
    want[sel] = pred.clamp(-10, 10)[rows[sel], rank[sel].long()]
    for o, c in ((ops, C), (ops.t().contiguous().t(), C.t().contiguous().t())):  # both memory orders
        out = torch.empty_like(c)
        _lib.check(L.sr_mlp_place_constants(_lib.ptr(o), B, M, *o.stride(), _lib.ptr(pred), 8, 8, 10.0, _lib.ptr(c),
                                            _lib.ptr(out), *c.stride(), st), "place")
        assert torch.equal(torch.nan_to_num(out, nan=99.0), torch.nan_to_num(want, nan=99.0))
    for K in (1, 2, 5):
        sets = torch.as_tensor(rng.standard_normal((K, B, M)).astype(np.float32)).cuda()
        loss = torch.as_tensor(rng.choice([1.0, 2.0, np.inf, -np.inf, np.nan], size=(B, K)).astype(np.float32)).cuda()
        clean = torch.where(torch.isfinite(loss), loss, torch.full_like(loss, float("inf"))).cpu().numpy()
        best = torch.as_tensor(clean.argmin(1)).cuda()  # numpy: the first of equal ones
        out = torch.empty((B, M), device="cuda")
        _lib.check(L.sr_mlp_pick_start(_lib.ptr(loss), _lib.ptr(sets), K, B, M, _lib.ptr(out), st), "pick")
        assert torch.equal(out, sets[best, torch.arange(B, device="cuda")])


def test_starts_carry_a_tangent():
    """Forward-mode differentiation goes through the chosen start: the tangent of the chosen
    candidate, zero where a prediction took the constant's place."""
    import torch.autograd.forward_ad as fw

    from cudasymbolicregression_gb300 import tapes, warmstart
    rng = np.random.default_rng(3)
    B, M, N = 40, 24, 60
    tb = tapes.generate(B, M, seed=3, mean_length=10, n_vars=2, unary=(10, 11), binary=(40, 41, 42), p_const_leaf=0.5)
    ops, ch = torch.as_tensor(tb.ops).cuda(), torch.as_tensor(tb.ch).cuda()
    X = torch.as_tensor(rng.uniform(-1, 1, (N, 2)).astype(np.float32)).cuda()
    Y = torch.as_tensor(rng.uniform(-1, 1, (B, N)).astype(np.float32)).cuda()
    C = torch.as_tensor(rng.standard_normal((B, M)).astype(np.float32)).cuda()
    net = warmstart.WarmStartMLP(seed=1)
    plain = warmstart.warm_start_constants(net, X, Y, ops, C)
    with fw.dual_level():
        t = torch.as_tensor(rng.standard_normal((B, M)).astype(np.float32)).cuda()
        out = fw.unpack_dual(warmstart.warm_start_constants(net, X, Y, ops, fw.make_dual(C, t)))
        rank = torch.cumsum((ops == 1).int(), 1) - 1
        assert torch.equal(out.primal, plain)
        assert torch.equal(out.tangent, torch.where((ops == 1) & (rank < 8), torch.zeros_like(t), t))
        sets, ts = torch.stack([C, plain]), torch.stack([t, -t])
        out = fw.unpack_dual(warmstart.screened_start(X, Y, ops, ch, fw.make_dual(sets, ts)))
        chosen = warmstart.screened_start(X, Y, ops, ch, sets)
        assert torch.equal(out.primal, chosen)
        first = (chosen == C).all(1, keepdim=True)
        assert torch.equal(out.tangent, torch.where(first, t, -t))
