"""The kernels that work on rows of one byte per token, against the oracle and against the
kernels that take the same rows with wider tokens (longer rows, larger ids): every word and
every error code, failed rows included, at row lengths around a word of four tokens and at
batch sizes around a CTA's 128 rows."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _call(fn, x, n_vars, width=None, last=()):
    from cudasymbolicregression_gb300 import _lib
    xd = torch.tensor(x).cuda()
    B, M = x.shape
    out = torch.full((B, M if width is None else width) + last, 77, dtype=torch.int64, device="cuda")
    err = torch.full((B,), 77, dtype=torch.int64, device="cuda")
    args = [_lib.ptr(xd), B, M, n_vars, _lib.ptr(out)] + ([width] if width is not None else [])
    assert getattr(_lib.lib(), fn)(*args, _lib.ptr(err), _lib.stream_ptr(xd.device)) == 0
    return out.cpu().numpy(), err.cpu().numpy()


def _postfix(B, M, seed):
    """Postfix rows of up to M tokens, a third of them damaged, some empty."""
    rng = np.random.default_rng(seed)
    rows = np.zeros((B, M), np.int64)
    for b in range(B):
        n, depth, left = 0, 0, int(rng.integers(0, M + 1))
        while n + max(depth - 1, 0) < left or (depth > 1 and n < M):
            close = n + depth > left or n + depth >= M
            u = rng.random()
            if depth >= 2 and (close or u < 0.35):
                rows[b, n] = rng.integers(40, 45)
                depth -= 1
            elif depth >= 1 and not close and u < 0.6:
                rows[b, n] = rng.integers(10, 32)
            elif not close or depth == 0:
                rows[b, n] = rng.choice([1, 2, 7, 50, 51])
                depth += 1
            else:
                break
            n += 1
    bad = np.nonzero(rng.random(B) < 0.33)[0]
    rows[bad, rng.integers(0, M, bad.size)] = rng.choice([0, 10, 14, 40, 50, 2, -3, 60, 52, 2 ** 40], size=bad.size)
    return rows


SHAPES = [(1, 1), (127, 2), (128, 3), (129, 4), (500, 5), (1000, 31), (257, 64), (300, 127), (200, 128)]


@pytest.mark.parametrize("B,M", SHAPES)
def test_reorder_equals_wide_tokens(B, M):
    for fn, x in (("sr_postfix_to_prefix", _postfix(B, M, B + M)),
                  ("sr_prefix_to_postfix", _postfix(B, M, B + M)[:, ::-1].copy()),
                  ("sr_prefix_to_postfix", _call("sr_postfix_to_prefix", _postfix(B, M, M), 2)[0])):
        x[x >= 60] = -1  # out of range with either number of variables
        got, err = _call(fn, x, 10)
        ref, ref_err = _call(fn, x, 2000)
        np.testing.assert_array_equal(err, ref_err)
        np.testing.assert_array_equal(got, ref)
        want, want_err = oracle.reorder(x, 10, fn == "sr_prefix_to_postfix")
        np.testing.assert_array_equal(err, want_err)
        np.testing.assert_array_equal(got[err == 0], want[err == 0])


@pytest.mark.parametrize("B,M", SHAPES)
@pytest.mark.parametrize("width", [0, 1, 33, 500])
def test_infix_equals_wide_tokens(B, M, width):
    x = _postfix(B, M, 3 * B + M)
    x[x >= 60] = -1
    got, err = _call("sr_postfix_to_infix", x, 10, width)
    ref, ref_err = _call("sr_postfix_to_infix", x, 2000, width)
    np.testing.assert_array_equal(err, ref_err)
    np.testing.assert_array_equal(np.where(got >= 60, got + 1990, got), ref)
    want, want_err = oracle.to_infix(x, 10, width)
    np.testing.assert_array_equal(err, want_err)
    np.testing.assert_array_equal(got[err == 0], want[err == 0])


@pytest.mark.parametrize("B,M", SHAPES)
@pytest.mark.parametrize("n_vars", [2, 400])
def test_children_equal_long_rows(B, M, n_vars):
    """The same rows padded to 160 tokens go to the kernel for long rows; the table at an
    address that is no multiple of 16 bytes is written with single stores."""
    from cudasymbolicregression_gb300 import _lib
    x = _postfix(B, M, 5 * B + M)
    got, err = _call("sr_postfix_children", x, n_vars, last=(2,))
    ref, ref_err = _call("sr_postfix_children", np.pad(x, ((0, 0), (0, 160 - M))), n_vars, last=(2,))
    np.testing.assert_array_equal(err, ref_err)
    np.testing.assert_array_equal(got, ref[:, :M])
    xd = torch.tensor(x).cuda()
    flat = torch.full((2 * B * M + 2,), 77, dtype=torch.int64, device="cuda")
    e = torch.empty(B, dtype=torch.int64, device="cuda")
    assert _lib.lib().sr_postfix_children(_lib.ptr(xd), B, M, n_vars, flat.data_ptr() + 8, _lib.ptr(e),
                                          _lib.stream_ptr(xd.device)) == 0
    np.testing.assert_array_equal(flat[1:-1].cpu().numpy().reshape(B, M, 2), got)
    assert flat[0] == 77 and flat[-1] == 77


@pytest.mark.parametrize("B,M", SHAPES)
@pytest.mark.parametrize("n_vars", [2, 202, 203])
def test_parsers_match_oracle(B, M, n_vars):
    """202 variables are the most whose token ids fit a byte row."""
    rng = np.random.default_rng(7 * B + M)
    lp, rp = 50 + n_vars, 51 + n_vars
    x = rng.choice([lp, rp, lp, 10, 14, 40, 42, 44, 50, 51, 1, lp - 1], size=(B, M)).astype(np.int64)
    post = _postfix(B, M, B)
    good, e = oracle.to_infix(np.where(post >= 52, 50, np.maximum(post, 0)), n_vars, M)
    x[::2] = good[::2]
    x[np.arange(M) >= rng.integers(0, M + 1, (B, 1))] = 0
    bad = np.nonzero(rng.random(B) < 0.1)[0]
    x[bad, rng.integers(0, M, bad.size)] = rng.choice([-1, rp + 1, 0, 2 ** 33 + 50, 50], size=bad.size)
    for fn, prefix in (("sr_infix_to_postfix", False), ("sr_infix_to_prefix", True)):
        got, err = _call(fn, x, n_vars)
        want, want_err = oracle.infix_parse(x, n_vars, prefix)
        np.testing.assert_array_equal(err, want_err)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("B,length", [(1, 1), (63, 3), (129, 9), (5000, 20), (100000, 128)])
@pytest.mark.parametrize("offset,n_symbols", [(0, 8), (250, 8), (251, 8), (3000, 8), (0, 300), (0, 2000)])
def test_sampler_symbol_and_table_sizes(B, length, offset, n_symbols):
    """Rules of no, one, two, six and nine symbols; terminals moved up to the last id that
    fits a byte, past it and past the symbols that have rules; more symbols than a byte
    holds."""
    from cudasymbolicregression_gb300 import _lib
    E, V = 1, 2
    rules = {E: [[V], [E, 3, E], [4, E], [], [5, V, 3, V, 3, V], [5] * 8 + [V], [7]], V: [[6], [7], [5, V]]}
    probs = {E: [0.4, 0.6, 0.7, 0.75, 0.85, 0.9, 0.99], V: [0.5, 0.8, 1.0]}
    nt, cum, rp, rc = [0], [], [0], []
    for s in range(n_symbols):
        for r, c in zip(rules.get(s, []), probs.get(s, [])):
            rc += [v if v <= V else v + (offset if v == 5 else 0) for v in r]
            rp.append(len(rc))
            cum.append(c)
        nt.append(len(cum))
    tables = [np.array(nt, np.int32), np.array(cum, np.float32), np.array(rp, np.int32), np.array(rc, np.int32)]
    d = [torch.tensor(a).cuda() for a in tables]
    out = torch.full((B, length), 77, dtype=torch.int64, device="cuda")
    err = torch.full((B,), 77, dtype=torch.int64, device="cuda")
    assert _lib.lib().sr_pcfg_sample_infix(*(_lib.ptr(a) for a in d), n_symbols, E, B, length, 5, 99, _lib.ptr(out),
                                           _lib.ptr(err), _lib.stream_ptr(out.device)) == 0
    want, want_err = oracle.pcfg_sample(tables, E, B, length, 5, 99)
    np.testing.assert_array_equal(err.cpu().numpy(), want_err)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_calls_of_several_threads_keep_their_shared_memory():
    """Threads whose calls need different amounts of shared memory launch the same kernels at
    the same time: no launch is refused, and every row is right."""
    import threading

    from cudasymbolicregression_gb300 import _lib
    L = _lib.lib()
    sizes = [(128, 384), (128, 200), (100, 300), (128, 300)]
    rows = [_postfix(300, M, i) for i, (M, _) in enumerate(sizes)]
    want = [_call("sr_postfix_to_infix", x, 2, width) + _call("sr_postfix_children", x, 2, last=(2,))
            for x, (_, width) in zip(rows, sizes)]
    failed = []

    def work(x, width, want):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            xd = torch.tensor(x).cuda()
            B, M = x.shape
            out, ch = torch.empty((B, width), dtype=torch.int64).cuda(), torch.empty((B, M, 2), dtype=torch.int64).cuda()
            err, err_ch = (torch.empty(B, dtype=torch.int64).cuda() for _ in range(2))
            st = _lib.stream_ptr(xd.device)
            for _ in range(3000):
                if L.sr_postfix_to_infix(_lib.ptr(xd), B, M, 2, _lib.ptr(out), width, _lib.ptr(err), st) or \
                        L.sr_postfix_children(_lib.ptr(xd), B, M, 2, _lib.ptr(ch), _lib.ptr(err_ch), st):
                    failed.append(L.sr_last_error())
                    return
            stream.synchronize()
            got = [t.cpu().numpy() for t in (out, err, ch, err_ch)]
            if not all(np.array_equal(a, b) for a, b in zip(got, want)):
                failed.append("rows differ")

    threads = [threading.Thread(target=work, args=(x, w, e)) for x, (_, w), e in zip(rows, sizes, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("rules,symbols,top", [(209, 260, 255), (400, 500, 120), (3, 3000, 255), (209, 260, 256), (400, 600, 5000)])
@pytest.mark.parametrize("B,length", [(1, 1), (65, 9), (3000, 64), (40000, 128)])
def test_sampler_tables_larger_than_its_copy(rules, symbols, top, B, length):
    """Grammars whose tables stay in global memory: more rules, or more symbols on their right-hand
    sides, than the copy holds, with ids that fit a byte and ids that do not."""
    from cudasymbolicregression_gb300 import _lib
    rng = np.random.default_rng([rules, symbols, top])
    per = symbols // rules
    E = 1
    rc, rp = [], [0]
    for r in range(rules):
        rc += [E if r % 5 == 0 and i % 2 == 0 and i < 3 else int(rng.integers(2, top + 1)) for i in range(max(1, per))]
        rp.append(len(rc))
    rc[-1] = top
    n_symbols = min(256, top + 1)
    nt = np.zeros(n_symbols + 1, np.int32)
    nt[E + 1:] = rules
    cum = ((np.arange(rules) + 1) / rules).astype(np.float32)
    tables = [nt, cum, np.array(rp, np.int32), np.array(rc, np.int32)]
    d = [torch.tensor(a).cuda() for a in tables]
    out = torch.full((B, length), 77, dtype=torch.int64, device="cuda")
    err = torch.full((B,), 77, dtype=torch.int64, device="cuda")
    assert _lib.lib().sr_pcfg_sample_infix(*(_lib.ptr(a) for a in d), n_symbols, E, B, length, 5, 99, _lib.ptr(out),
                                           _lib.ptr(err), _lib.stream_ptr(out.device)) == 0
    want, want_err = oracle.pcfg_sample(tables, E, B, length, 5, 99)
    np.testing.assert_array_equal(err.cpu().numpy(), want_err)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
