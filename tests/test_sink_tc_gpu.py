"""Attention with a sink in long steps, the kernel of sequences that bring many tokens: edges of its tiles (128 queries, 64 keys) over unequal sequences,
offsets, windows with kept tokens, chunks, biases, gates and head sizes against the kernel of shorter ones, to the bit, and against 64 bits; rows of the
last page that hold no numbers."""
import math

import pytest
import torch

gpu = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def test_which_steps_it_takes():
    takes, each, n = K().sink_tc_takes, K().SINK_TC_TOKENS, K().SINK_TC_ALL
    assert takes(n, 1, 4, 2, 64, 64, 64) and not takes(n - 1, 1, 4, 2, 64, 64, 64) and not takes(50 * each - 1, 50, 4, 2, 64, 64, 64)
    assert takes(50 * each, 50, 8, 1, 128, 16, 256) and not takes(n, 1, 4, 4, 64, 64, 64) and not takes(n, 1, 6, 2, 64, 64, 64)
    assert not takes(n, 1, 4, 2, 64, 80, 64) and not takes(n, 1, 4, 2, 64, 64, 32) and not takes(n, 1, 4, 2, 144, 64, 64)


def test_steps_measured_on_both_sides_of_the_rule():
    """(tokens, sequences, heads, whether it is the faster kernel)"""
    for N, n, nh, there in [(2048, 1, 32, True), (2048, 1, 8, True), (4096, 1, 2, True), (1024, 8, 32, True), (1024, 1, 32, True), (1024, 4, 32, True), (1536, 16, 32, True),
                            (1536, 16, 16, True), (4096, 32, 8, True), (1024, 8, 48, False), (1200, 4, 32, False), (1024, 8, 16, False), (1536, 16, 8, False), (1536, 16, 2, False),
                            (4096, 32, 2, False), (2048, 32, 32, False), (512, 1, 32, False), (256, 1, 128, False)]:
        assert K().sink_tc_takes(N, n, nh, nh // 2, 64, 64, 64) == there, (N, n, nh)


def case(lens, starts, nh, nkv, dk, dv, page, seed, v_in_k=False, tail=None):
    g = torch.Generator().manual_seed(seed)
    total = [a + n for a, n in zip(starts, lens)]
    pages = [-(-t // page) for t in total]
    keys = [torch.randn(t, nkv, dk, generator=g).to(BF) for t in total]
    values = [k[..., :dv] if v_in_k else torch.randn(k.shape[0], nkv, dv, generator=g).to(BF) for k in keys]
    order = torch.randperm(sum(pages), generator=g)
    row = dk if v_in_k else dk + dv
    pool = torch.zeros(sum(pages), nkv * page * row, dtype=BF)
    if tail is not None:
        pool.fill_(tail)
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32)
    for b, t in enumerate(total):
        for i in range(pages[b]):
            at = int(order[sum(pages[:b]) + i])
            table[b, i] = at
            n = min(page, t - i * page)
            pool[at, :nkv * page * dk].view(nkv, page, dk)[:, :n] = keys[b][i * page:i * page + n].transpose(0, 1)
            if not v_in_k:
                pool[at, nkv * page * dk:].view(nkv, page, dv)[:, :n] = values[b][i * page:i * page + n].transpose(0, 1)
    q = torch.randn(sum(lens), nh, dk, generator=g).to(BF)
    return q, keys, values, pool, table


def run(q, pool, table, lens, starts, nh, nkv, dk, dv, page, *, all_heads=False, **kw):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)     # noqa: E731
    N = sum(lens)
    out = torch.zeros(N, nh * dv, dtype=BF, device=DEV)
    full = torch.zeros(N, nh, nkv, dv, device=DEV) if all_heads else None
    kw = {k: tuple(x.to(DEV) for x in v) if isinstance(v, tuple) else v.to(DEV) if torch.is_tensor(v) else v for k, v in kw.items()}
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    got = K().attention_sink_prefill(q.reshape(N, -1).to(DEV), pool.to(DEV), page, table.to(DEV), i32(cu), i32(starts), out, len(lens), nh, nkv, dk, dv,
                                     dk ** -0.5, out_all=full, **kw)
    return got.cpu()


def exact(q, keys, values, lens, starts, nh, nkv, dv, *, softcap=0.0, window=0, keep_first=0, chunk=0, sinks=None, gate=None, gate_wide=False,
          distance_bias=None, distance_table=None, all_heads=False, **_):
    outs, at = [], 0
    for b, n in enumerate(lens):
        p = torch.arange(starts[b], starts[b] + n)[:, None]
        t = torch.arange(keys[b].shape[0])[None]
        seen = t <= p
        if chunk:
            seen &= t >= p - p % chunk
        elif window:
            seen &= (t > p - window) | (t < keep_first)
        rows = []
        for h in range(nh):
            g = h // (nh // nkv)
            s = q[at:at + n, h].double() @ keys[b][:, g].double().T * q.shape[-1] ** -0.5
            if softcap:
                s = softcap * torch.tanh(s / softcap)
            d = (p - t).clamp(min=0)
            if distance_table is not None:
                s = s + distance_table[h].double()[d.clamp(max=distance_table.shape[1] - 1)]
            if distance_bias is not None:
                s = s - distance_bias[0][h].double() * torch.log1p(distance_bias[1][h].double() * d)
            s = s.masked_fill(~seen, -math.inf)
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            w = torch.softmax(s, -1)[:, :keys[b].shape[0]]
            o = torch.stack([w @ values[b][:, v].double() for v in (range(nkv) if all_heads else [g])], 1)
            if gate is not None:
                z = gate[at:at + n].double()
                o = o * torch.sigmoid(z.view(n, nh, -1)[:, h])[:, None]
            rows.append(o if all_heads else o[:, 0])
        outs.append(torch.stack(rows, 1))
        at += n
    return torch.cat(outs)


FORMS = [dict(), dict(softcap=30.0, window=100, keep_first=70, sinks=True, gate="head"), dict(chunk=150, split_weights=True),
         dict(softcap=50.0, sinks=True, table=241, split_weights=True), dict(table=2500, split_weights=True), dict(softcap=20.0, table=1, window=300),
         dict(window=37, keep_first=200, sinks=True, split_weights=True, all_heads=True), dict(bias=True, window=500, v_in_k=True, gate="element", sinks=True),
         dict(bias=True, split_weights=True, chunk=64), dict(window=64, keep_first=1)]


@gpu
@pytest.mark.parametrize("form", range(len(FORMS)))
@pytest.mark.parametrize("lens,starts,nh,nkv,dk,dv,page", [([1, 127, 128, 129, 500], [0, 5, 100, 0, 77], 4, 2, 64, 64, 64), ([257, 640], [63, 1], 4, 1, 80, 64, 128),
                                                           ([300], [641], 2, 1, 16, 16, 64), ([190, 260], [0, 0], 4, 2, 128, 48, 256)])
def test_against_64_bits_and_the_other_kernel(form, lens, starts, nh, nkv, dk, dv, page, monkeypatch):
    kw = dict(FORMS[form])
    g = torch.Generator().manual_seed(form)
    N, v_in_k = sum(lens), kw.pop("v_in_k", False)
    if kw.get("sinks"):
        kw["sinks"] = torch.randn(nh, generator=g)
    if "gate" in kw:
        kw["gate_wide"] = kw["gate"] == "element"
        kw["gate"] = torch.randn(N, nh * dv if kw["gate_wide"] else nh, generator=g)
    if "table" in kw:
        kw["distance_table"] = torch.randn(nh, kw.pop("table"), generator=g)
    if kw.pop("bias", False):
        kw["distance_bias"] = (torch.rand(nh, generator=g), torch.rand(nh, generator=g))
    q, keys, values, pool, table = case(lens, starts, nh, nkv, dk, dv, page, form, v_in_k)
    if v_in_k:
        kw["values_in_keys"] = True
    with monkeypatch.context() as m:
        m.setattr(K(), "SINK_TC_TOKENS", 1)
        m.setattr(K(), "SINK_TC_ALL", 1)
        assert K().sink_tc_takes(N, len(lens), nh, nkv, dk, dv, page)
        got = run(q, pool, table, lens, starts, nh, nkv, dk, dv, page, **kw)
        m.setattr(K(), "SINK_TC_TOKENS", 1 << 30)
        other = run(q, pool, table, lens, starts, nh, nkv, dk, dv, page, **kw)
    assert torch.equal(got, other)
    want = exact(q, keys, values, lens, starts, nh, nkv, dv, **kw)
    # the result's rounding to bfloat16, and the weights', which with values of up to 5 moves a row's average by at most 2^-9 of 5 (2^-17 where they are split)
    tol = 2 ** -13 if kw.get("split_weights") else 5 * 2 ** -9
    assert bool(((got.double().view(want.shape) - want).abs() <= 2 ** -8 * want.abs() + tol).all())


@gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_after_the_last_token_hold_anything(bad, monkeypatch):
    lens, starts, nh, nkv, dk, dv, page = [131, 300], [0, 10], 4, 2, 64, 32, 128
    monkeypatch.setattr(K(), "SINK_TC_TOKENS", 1)
    monkeypatch.setattr(K(), "SINK_TC_ALL", 1)
    outs = [run(*[x for i, x in enumerate(case(lens, starts, nh, nkv, dk, dv, page, 1, tail=tail)) if i in (0, 3, 4)], lens, starts, nh, nkv, dk, dv, page)
            for tail in (0.0, bad)]
    assert torch.equal(*outs) and outs[0].isfinite().all()


@gpu
def test_sinks_of_any_size(monkeypatch):
    lens, starts, nh, nkv, dk, dv, page = [200], [0], 4, 2, 64, 64, 64
    q, _, _, pool, table = case(lens, starts, nh, nkv, dk, dv, page, 2)
    sinks = torch.tensor([float("-inf"), -2e38, 60.0, 2e38])
    outs = []
    monkeypatch.setattr(K(), "SINK_TC_ALL", 1)
    for n in (1, 1 << 30):
        monkeypatch.setattr(K(), "SINK_TC_TOKENS", n)
        outs.append(run(q, pool, table, lens, starts, nh, nkv, dk, dv, page, sinks=sinks))
    assert torch.equal(*outs)


@gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("form", [dict(), dict(window=100, keep_first=70), dict(window=37), dict(window=300, keep_first=64, split_weights=True), dict(chunk=150),
                                  dict(softcap=20.0, chunk=64, all_heads=True)])
@pytest.mark.parametrize("lens,starts,dk,dv,page", [([700], [0], 64, 64, 64), ([130, 400], [301, 45], 80, 48, 128), ([520], [250], 128, 64, 64)])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(bad, form, lens, starts, dk, dv, page, monkeypatch):
    """Values before and behind the edges of blocks, tiles, windows, kept tokens and chunks, each in a channel of its own of one kv head."""
    monkeypatch.setattr(K(), "SINK_TC_TOKENS", 1)
    monkeypatch.setattr(K(), "SINK_TC_ALL", 1)
    nh, nkv, kw = 4, 2, dict(form)
    q, _, _, pool, table = case(lens, starts, nh, nkv, dk, dv, page, 7)
    window, keep, chunk = kw.get("window", 0), kw.get("keep_first", 0), kw.get("chunk", 0)
    assert K().sink_tc_takes(sum(lens), len(lens), nh, nkv, dk, dv, page)
    spots, row0 = [], 0
    for b, (n, s) in enumerate(zip(lens, starts)):
        at = [s + p for p in (-60, -1, 0, 3, 63, 64, 70, 127, 128, 129, 255, n - 70, n - 1)] + [5, 63, 64, 69, 70, 149, 150, 199]
        spots += [(p, b, s, row0, n) for p in sorted(set(at)) if 0 <= p < s + n]
        row0 += n
    N = sum(lens)
    for round0 in range(0, len(spots), dv):
        some = spots[round0:round0 + dv]
        pools = []
        for value in (bad, 0.0):
            pools.append(pool.clone())
            for c, (p, b, *_) in enumerate(some):
                pools[-1][int(table[b, p // page]), nkv * page * dk + ((c % nkv) * page + p % page) * dv + c] = value
        got, want = (run(q, x, table, lens, starts, nh, nkv, dk, dv, page, **kw) for x in pools)
        sees = torch.zeros(N, nh, nkv, dv, dtype=torch.bool)
        for c, (p, b, s, r0, n) in enumerate(some):
            pos = torch.arange(s, s + n)
            see = pos >= p
            if chunk:
                see &= p >= pos - pos % chunk
            elif window:
                see &= (p > pos - window) | (p < keep)
            for h in range(nh):
                sees[r0:r0 + n, h, c % nkv, c] = see
        if kw.get("all_heads"):
            got, want = got.view(N, nh, nkv, dv), want.view(N, nh, nkv, dv)
        else:
            got, want = got.view(N, nh, dv), want.view(N, nh, dv)
            sees = torch.stack([sees[:, h, h // (nh // nkv)] for h in range(nh)], 1)
        assert torch.equal(got[~sees], want[~sees]) and bool(want.isfinite().all()) and not bool(got[sees].isfinite().any())
    K().check_device_errors()
