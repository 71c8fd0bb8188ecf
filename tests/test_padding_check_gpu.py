"""The adjoint's check of the padding rows: one nonzero gradient anywhere in them raises error 201.

A range of padding starts and ends off 16-byte boundaries (odd point counts, odd tape lengths) and
is read in copies of 8192 bytes through a ring of four (the sweep's batches) or by strided 16-byte
loads (the staged kernel's), so the nonzero is put at the first and last element, around the
boundaries and into the middle, with constant sets and on both sides of the size from which
the check runs beside the adjoint."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# more than five copies of 8192 bytes; one copy; less than a boundary; few points (staged)
SHAPES = [(40, 24, 777, 0), (40, 24, 778, 0), (700, 12, 257, 0), (12, 24, 300, 5), (30, 6, 65, 0), (30, 24, 3, 0),
          (3, 9, 1, 0), (1500, 20, 130, 0), (29500, 4, 66, 0)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("B,M,N,K", SHAPES)
def test_any_nonzero_padding_gradient_is_found(B, M, N, K, dtype):
    import cudasymbolicregression_gb300 as sr
    g = torch.Generator().manual_seed(B + N)
    lengths = torch.randint(1, M, (B,), generator=g)
    ops = torch.zeros(B, M, dtype=torch.int64)
    ch = -torch.ones(B, M, 2, dtype=torch.int64)
    k = torch.arange(M)
    ops[:, 0] = 50
    chain = (k > 0) & (k < lengths[:, None])
    ops[chain] = 27  # a chain of neg
    ch[..., 0] = torch.where(chain, (k - 1).expand(B, M), ch[..., 0])
    X = torch.linspace(-1, 1, N, dtype=dtype).reshape(N, 1).cuda()
    C = torch.zeros((B, M, K) if K else (B, M), dtype=dtype).cuda().requires_grad_(True)
    fn = sr.evaluation.evaluate_multiple if K else sr.evaluation.evaluate
    y = fn(X, ops.cuda(), ch.cuda(), C)
    gout = torch.zeros_like(y)
    width = N * max(K, 1)  # elements of a row
    flat = gout.view(B, M * width)

    def backward():
        return torch.autograd.grad(y, C, gout, retain_graph=True)

    def fails(b, at, value):
        flat[b, at] = value
        try:
            with pytest.raises(RuntimeError, match="NO_OP"):
                backward()
        finally:
            flat[b, at] = 0

    flat[:, -1] = -0.0  # no gradient
    backward()
    flat[:, -1] = 0
    least = 2.0 ** -149 if dtype == torch.float32 else 2.0 ** -1074  # one bit, in a double's lower word
    per = 8192 // gout.element_size()
    for b in {0, B // 2, B - 1}:
        lo, hi = int(lengths[b]) * width, M * width
        mis = (-(b * M * width + lo)) % (16 // gout.element_size())  # elements before the boundary
        places = {lo, lo + 1, lo + mis - 1, lo + mis, hi - 1, hi - 2, (lo + hi) // 2}
        places |= {lo + mis + i * per + d for i in (1, 4, 5) for d in (-1, 0)}
        for i, at in enumerate(sorted(p for p in places if lo <= p < hi)):
            fails(b, at, (1.0, least, float("nan"), float("inf"))[i % 4])
        if lo < hi:
            fails(b, hi - 1, least)
    backward()
