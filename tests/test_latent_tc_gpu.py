"""Attention over a compressed cache in long steps, the kernel of sequences that bring or see many rows: edges of its tiles (128 queries, 64
keys) over unequal sequences, offsets, windows, sinks and gates against 64 bits; a sink far above every key; values that are not finite."""
import pytest
import torch

from test_latent_prefill_gpu import DEV, attend, exact, inputs, rows_seen

gpu = pytest.mark.gpu


def takes(lens, starts, window, rot=32):
    from mivi_v4_b200.ops import kernels as K
    return K.latent_tc_takes(sum(lens), rows_seen(lens, starts, window), len(lens), 64, rot, 64, 0.1)


def test_which_steps_it_takes():
    assert takes([200], [0], 0) and not takes([199], [0], 0) and takes([199], [201], 0) and not takes([199, 199], [201, 200], 0)
    assert not takes([199], [500], 100) and takes([200], [500], 100, rot=64) and not takes([200], [500], 100, rot=16)


def test_steps_measured_on_both_sides_of_the_rule():
    """(sequences, tokens of each, earlier ones, heads, whether it is the faster kernel)"""
    from mivi_v4_b200.ops import kernels as K
    for n, new, before, nh, there in [(1, 2048, 0, 8, True), (16, 200, 0, 32, True), (8, 128, 300, 32, True), (16, 96, 800, 32, True), (3, 32, 800, 32, True), (1, 64, 2000, 32, True),
                                      (16, 32, 800, 8, True), (4, 16, 400, 32, True), (16, 48, 2000, 32, True), (16, 48, 2000, 16, True), (32, 64, 0, 32, False), (32, 128, 0, 32, False),
                                      (16, 64, 190, 32, False), (32, 16, 800, 32, False), (32, 16, 800, 16, False), (32, 16, 800, 8, False), (16, 32, 800, 32, False), (16, 32, 800, 16, False),
                                      (8, 32, 500, 32, False), (6, 32, 500, 32, False), (5, 16, 400, 32, False), (16, 64, 800, 32, False), (32, 64, 800, 32, False)]:
        assert K.latent_tc_takes(n * new, n * (new + before), n, 64, 32, 64, 0.1, nh) == there, (n, new, before, nh)


@gpu
@pytest.mark.parametrize("lens,starts", [([1, 95, 96, 97, 300, 1000], [0, 5, 100, 0, 77, 3]), ([257, 640], [0, 0]), ([1, 31, 128], [700, 500, 383])])
@pytest.mark.parametrize("window", [0, 37, 96, 500])
@pytest.mark.parametrize("rot,sink,gate", [(32, True, "element"), (64, False, None), (32, True, "head")])
def test_against_64_bits_and_the_other_kernel(lens, starts, window, rot, sink, gate, monkeypatch):
    from mivi_v4_b200.ops import kernels as K
    nh = 3
    q, k, v, r, sinks, gates = inputs(lens, starts, nh, 64, rot, 64, window, seed=window + rot)
    sinks = sinks if sink else None
    gates = {None: None, "element": gates, "head": gates[:, :, :1]}[gate]
    with monkeypatch.context() as m:                           # (short sequences behind a window would take the other kernel)
        m.setattr(K, "LATENT_TC_TOKENS", 1)
        assert takes(lens, starts, window, rot)
        got = attend(slice(0, nh), lens, starts, window, q, k, v, r, sinks, gates)
    with monkeypatch.context() as m:                           # every sum in the other kernel's order: the same bits
        m.setattr(K, "LATENT_TC_TOKENS", 1 << 30)
        m.setattr(K, "LATENT_TC_ROWS", 1 << 30)
        assert torch.equal(got, attend(slice(0, nh), lens, starts, window, q, k, v, r, sinks, gates))
    want = exact(lens, starts, window, q, k, v, r, sinks, gates)
    # the result's rounding to bfloat16, the weights' to 16 bits, scores' sums of up to 128 products of up to 5 x 5 in 32 bits
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -13).all())


@gpu
def test_growing_scores_move_the_reference():
    """Every block's scores outgrow the ones before by far: the sums are brought to the new reference each time."""
    lens, starts = [700], [0]
    q, k, v, r, sinks, _ = inputs(lens, starts, 2, 64, 32, 64, 0, seed=9)
    q = q.abs()
    k = (k.abs().float() * (torch.arange(700) / 40.0)[:, None, None]).to(torch.bfloat16)
    got, want = attend(slice(0, 2), lens, starts, 0, q, k, v, r, sinks, None), exact(lens, starts, 0, q, k, v, r, sinks, None)
    # scores of up to some 700 in 32 bits: a weight is off by 700 x 2^-23 of itself
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 5 * 2 ** -11).all())


@gpu
def test_a_sink_far_above_the_keys():
    """Weights of e^-89 of the sink's still count: bfloat16 holds the results."""
    n, nh = 600, 4
    q, k, v, r, _, _ = inputs([n], [0], nh, 64, 32, 64, 0, seed=n)
    v = (v.float() * 2.0 ** 20).to(torch.bfloat16)
    sinks = torch.tensor([89.0, float("-inf"), float("inf"), -89.0])
    got = attend(slice(0, nh), [n], [0], 0, q, k, v, r, sinks, None)
    sinks[2] = 1e4                                             # (64 bits of exp: nothing is left of the weights)
    want = exact([n], [0], 0, q, k, v, r, sinks, None)
    total = exact([n], [0], 0, q, k, torch.ones_like(v), r, sinks, None)
    # as above, the second term for values of 2^20 and the sum of a row's weights; bfloat16's steps below its smallest exponent
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 2.0 ** 7 * total + 2.0 ** -133).all())
    assert bool((got[:, 2] == 0).all())


@gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_values_of_another_sequence_that_are_not_finite(bad):
    lens, starts = [300, 290, 333], [0, 10, 0]
    q, k, v, r, sinks, _ = inputs(lens, starts, 2, 64, 32, 64, 0, seed=3)
    want = attend(slice(0, 2), lens, starts, 0, q, k, v, r, sinks, None)
    k, v, r = k.clone(), v.clone(), r.clone()
    for t in (k, v, r):
        t[300:600] = bad                                       # all of the second sequence's rows
    got = attend(slice(0, 2), lens, starts, 0, q, k, v, r, sinks, None)
    assert torch.equal(got[:300], want[:300]) and torch.equal(got[590:], want[590:]) and not bool(got[300:590].isfinite().any())


@gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("lens,starts,window", [([700], [0], 0), ([300, 520], [70, 601], 0), ([700], [0], 100), ([190, 400], [300, 45], 37), ([1000], [77], 500)])
@pytest.mark.parametrize("gate", [None, "element"])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(bad, lens, starts, window, gate, monkeypatch):
    """Values of the sequence's own, each in a channel of its own: before and behind the edges of blocks, tiles and pairs of tiles, and of windows."""
    from mivi_v4_b200.ops import kernels as K
    monkeypatch.setattr(K, "LATENT_TC_TOKENS", 1)
    nh = 2
    q, k, v, r, sinks, gates = inputs(lens, starts, nh, 64, 32, 64, window, seed=5)
    gates = gates if gate else None
    dirty, clean = v.clone(), v.clone()
    spots, base, row0 = [], 0, 0
    for n, s in zip(lens, starts):
        lo = max(0, s - window + 1) if window else 0
        at = [s + p for p in (-60, -1, 0, 3, 62, 63, 64, 70, 126, 127, 128, 129, 190, 255, 256, 257, n - 70, n - 2, n - 1)]
        spots += [(p, base + p - lo, s, row0, n) for p in sorted(set(at)) if lo <= p < s + n]
        base, row0 = base + s + n - lo, row0 + n
    assert len(spots) <= 64
    for c, (_, row, *_) in enumerate(spots):
        dirty[row, c % nh, c], clean[row, c % nh, c] = bad, 0.0
    assert K.latent_tc_takes(sum(lens), rows_seen(lens, starts, window), len(lens), 64, 32, 64, 0.1)
    got, want = (attend(slice(0, nh), lens, starts, window, q, k, x, r, sinks, gates) for x in (dirty, clean))
    sees = torch.zeros(sum(lens), nh, 64, dtype=torch.bool, device=DEV)
    for c, (p, _, s, first, n) in enumerate(spots):
        pos = torch.arange(s, s + n, device=DEV)
        sees[first:first + n, c % nh, c] = (pos >= p) & ((pos < p + window) if window else True)
    assert torch.equal(got[~sees], want[~sees]) and bool(want.isfinite().all()) and not bool(got[sees].isfinite().any())
    K.check_device_errors()
