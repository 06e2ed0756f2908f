"""Attention over a compressed cache in long steps: every size of the kernel over unequal sequences, offsets, windows, sinks and gates, against
64 bits and, some heads alone against all together, to the bit; a sink far above every key."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS, STARTS = [1, 127, 128, 129, 300], [0, 5, 100, 0, 77]


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def rows_seen(lens, starts, window):
    return sum(s + n - (max(0, s - window + 1) if window else 0) for n, s in zip(lens, starts))


def inputs(lens, starts, nh, dim, rot, dv, window, seed):
    g = torch.Generator().manual_seed(seed)
    rows, N = rows_seen(lens, starts, window), sum(lens)
    q = torch.randn(N, nh, dim + rot, generator=g).to(torch.bfloat16)
    k, v = torch.randn(rows, nh, dim, generator=g).to(torch.bfloat16), torch.randn(rows, nh, dv, generator=g).to(torch.bfloat16)
    r = torch.randn(rows, rot, generator=g).to(torch.bfloat16)
    return q, k, v, r, torch.randn(nh, generator=g), torch.randn(N, nh, dv, generator=g)


def attend(heads, lens, starts, window, q, k, v, r, sinks, gate):
    """The kernel's result for a range of heads, [N, heads, dv]."""
    from mivi_v4_b200.ops import kernels as K
    q, k, v = (x[:, heads].contiguous() for x in (q, k, v))
    N, nh, dk = q.shape
    dim, dv = k.shape[2], v.shape[2]
    kx = torch.cat([k.reshape(-1, nh * dim), v.reshape(-1, nh * dv)], 1).contiguous()
    cu = [sum(lens[:b]) for b in range(len(lens) + 1)]
    out = torch.full((N, nh * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
    if gate is not None:
        gate = gate[:, heads].reshape(N, -1).contiguous().to(DEV)
    K.latent_attention_prefill(q.to(DEV), kx.to(DEV), nh * dim, r.to(DEV), i32(cu), i32(starts), len(lens), out, nh, dim, dk - dim, dv,
                               dk ** -0.5, window=window, sinks=None if sinks is None else sinks[heads].contiguous().to(DEV), gate=gate)
    return out.reshape(N, nh, dv)


def exact(lens, starts, window, q, k, v, r, sinks, gate):
    q, k, v, r = (x.to(DEV).double() for x in (q, k, v, r))
    nh, dk = q.shape[1:]
    out, base, row0 = [], 0, 0
    for n, s in zip(lens, starts):
        lo = max(0, s - window + 1) if window else 0
        seen = slice(base, base + s + n - lo)
        key = torch.cat([k[seen], r[seen][:, None].expand(-1, nh, -1)], 2)
        score = torch.einsum("ihd,jhd->hij", q[row0:row0 + n], key) * dk ** -0.5
        i, j = torch.arange(s, s + n, device=DEV)[:, None], torch.arange(lo, s + n, device=DEV)[None]
        score = score.masked_fill((j > i) | ((j <= i - window) if window else False), float("-inf"))
        if sinks is not None:
            score = torch.cat([score, sinks.to(DEV).double()[:, None, None].expand(-1, n, 1)], 2)
        w = torch.softmax(score, 2)[..., :s + n - lo]
        out.append(torch.einsum("hij,jhd->ihd", w, v[seen]))
        base, row0 = base + s + n - lo, row0 + n
    out = torch.cat(out)
    return out if gate is None else out * torch.sigmoid(gate.to(DEV).double())


@pytest.mark.parametrize("window", [0, 37, 100])
@pytest.mark.parametrize("dim,rot,dv", [(64, 32, 64), (40, 8, 16), (64, 64, 64), (64, 32, 128), (128, 64, 48), (128, 64, 128)])
@pytest.mark.parametrize("sink,gate", [(False, None), (True, "element"), (True, "head")])
def test_all_heads_and_eight_at_a_time(window, dim, rot, dv, sink, gate):
    nh = 32
    q, k, v, r, sinks, gates = inputs(LENS, STARTS, nh, dim, rot, dv, window, seed=window + dim)
    sinks = sinks if sink else None
    gates = {None: None, "element": gates, "head": gates[:, :, :1]}[gate]
    got = attend(slice(0, nh), LENS, STARTS, window, q, k, v, r, sinks, gates)
    for h in range(0, nh, 8):
        assert torch.equal(got[:, h:h + 8], attend(slice(h, h + 8), LENS, STARTS, window, q, k, v, r, sinks, gates)), h
    want = exact(LENS, STARTS, window, q, k, v, r, sinks, gates)
    # the result's rounding to bfloat16, the weights' to 16 bits, scores' sums of up to 96 products of up to 5 x 5 in 32 bits
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -13).all())


@pytest.mark.parametrize("n,nh,dim,rot,dv", [(600, 32, 64, 32, 64), (90, 2, 64, 32, 64), (90, 2, 128, 64, 128)])
def test_a_sink_far_above_the_keys(n, nh, dim, rot, dv):
    """Weights below 2^-126 still count where a row has no larger ones: each is held to a multiple of 2^-133 (its two bfloat16
    numbers), n of them times values of up to 2^20 x 5."""
    lens, starts = [n], [0]
    q, k, v, r, _, _ = inputs(lens, starts, nh, dim, rot, dv, 0, seed=n)
    v = (v.float() * 2.0 ** 20).to(torch.bfloat16)
    sinks = torch.full((nh,), 89.0)
    got = attend(slice(0, nh), lens, starts, 0, q, k, v, r, sinks, None)
    want = exact(lens, starts, 0, q, k, v, r, sinks, None)
    assert float(want.abs().median()) > 2.0 ** -114                 # bfloat16 holds the results
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + n * 2.0 ** -134 * 2.0 ** 22.5).all())
    assert float((got.double() - want).norm() / want.norm()) < 0.05
