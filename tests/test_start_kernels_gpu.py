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
