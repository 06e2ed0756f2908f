"""The chunked kernels of a decaying matrix state at the edges of their tiles (64 tokens, 64 value columns, 64 and 32 key channels)
and of their dispatch (tile and token groups by the number of tiles; 16-byte copies or not; key sizes above 128), against the
recurrence in 64 bits.

Bound: a result is a sum of at most T products of numbers of order 1 whose factors are exact to a few 2^-24; against the
largest value 64 * 2^-24 = 4e-6 leaves room for the sums' own rounding over a few hundred tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


class Scratch:
    def get(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device=DEV)


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def close(got, want, what):
    err = (got.double().cpu() - want).abs().max().item() / want.abs().max().item()
    assert err <= 4e-6, f"{what}: off by {err:.3g} of the largest value"


def scan(q, k, v, a, S):
    """One head: S [dk, dv] <- a_t S + k_t v_t^T, o_t = S^T q_t."""
    out = []
    for t in range(q.shape[0]):
        S = a[t][:, None] * S + k[t][:, None] * v[t][None]
        out.append(S.T @ q[t])
    return torch.stack(out), S


@pytest.mark.parametrize("heads,group,dk,dv", [(1, 1, 128, 64), (2, 2, 33, 65), (3, 1, 4, 7), (80, 40, 64, 64), (160, 40, 8, 4), (2, 1, 200, 66)])
@pytest.mark.parametrize("lens", [[64], [16, 1, 65], [130, 63]])
@pytest.mark.parametrize("normalizer", [False, True])
def test_scalar_chunks(heads, group, dk, dv, lens, normalizer):
    from mivi_v4_b200.ops import kernels as K
    g = torch.Generator().manual_seed(heads * 1000 + dk + sum(lens))
    N, groups, B = sum(lens), heads // group, len(lens)
    q, k = (torch.randn(N, groups * dk, generator=g, dtype=torch.float32) for _ in "qk")
    v = torch.randn(N, heads * dv, generator=g, dtype=torch.float32)
    log_a = -torch.rand(N, heads, generator=g) * torch.tensor([0.01, 1.0, 90.0])[torch.arange(heads) % 3]
    b, m = torch.rand(N, heads, generator=g) + 0.1, torch.randn(N, heads, generator=g)
    skip = None if normalizer else torch.randn(heads, generator=g)
    cols = dv + int(normalizer)
    state = torch.randn(B + 1, heads, cols, dk, generator=g)
    slots = [B - i for i in range(B)]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    want_o, want_s = torch.zeros(N, heads * dv, dtype=F64), state.double().clone()
    for i in range(B):
        at = slice(cu[i], cu[i + 1])
        for h in range(heads):
            kh, qh = (x[at, h // group * dk:(h // group + 1) * dk].double() for x in (k, q))
            vh = v[at, h * dv:(h + 1) * dv].double()
            va = torch.cat([vh, torch.ones(len(vh), 1, dtype=F64)], 1) if normalizer else vh
            o, S = scan(qh * 0.5, kh * b[at, h:h + 1].double(), va, log_a[at, h:h + 1].double().exp().expand(-1, dk),
                        state[slots[i], h].double().T)
            want_s[slots[i], h] = S.T
            if normalizer:
                o = o[:, :dv] / (torch.maximum(o[:, dv:].abs(), torch.exp(-m[at, h:h + 1].double())) + 1e-6)
            else:
                o = o + skip[h].double() * vh
            want_o[at, h * dv:(h + 1) * dv] = o
    got = state.to(DEV)
    out = torch.full((N, heads * dv), float("nan"), device=DEV)
    K.scalar_scan(q.to(DEV), k.to(DEV), v.to(DEV), log_a.to(DEV), b.to(DEV), got, i32(slots), i32(cu), out, B, heads, dk, dv,
                  heads_per_group=group, skip=None if skip is None else skip.to(DEV), m_tok=m.to(DEV) if normalizer else None,
                  q_scale=0.5, max_len=max(lens), ws=Scratch())
    if normalizer:                  # a quotient of two sums: the denominator may be small beside its terms
        rows = (out.double().cpu() - want_o).abs() / want_o.abs().max()
        assert rows.max() <= 4e-4 and rows.mean() <= 4e-6
    else:
        close(out, want_o, "outputs")
    close(got, want_s, "state")
    assert torch.equal(got[0].cpu(), state[0])           # the slot that is not in the step


@pytest.mark.parametrize("heads,dk,dv", [(1, 128, 64), (2, 33, 65), (3, 160, 70), (40, 64, 130)])
@pytest.mark.parametrize("lens", [[64], [17, 66], [190]])
@pytest.mark.parametrize("kind,act", [("channel", 0), ("channel", 1), ("head", 0), ("head", 1)])
def test_decay_chunks(heads, dk, dv, lens, kind, act):
    from mivi_v4_b200.ops import kernels as K
    g = torch.Generator().manual_seed(heads * 1000 + dk + sum(lens))
    N, B = sum(lens), len(lens)
    q, k, z = (torch.randn(N, heads * dk, generator=g) for _ in "qkz")
    v = torch.randn(N, heads * dv, generator=g)
    z[:, 0] = -40.0                                      # a channel that forgets within a token
    decay = torch.rand(heads, generator=g)
    decay[0] = 0.999
    state = torch.randn(B, heads, dv, dk, generator=g)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    f = (lambda x: x * torch.sigmoid(x)) if act else (lambda x: x)
    want_o, want_s = torch.zeros(N, heads * dv, dtype=F64), state.double().clone()
    for i in range(B):
        at = slice(cu[i], cu[i + 1])
        for h in range(heads):
            a = torch.sigmoid(z[at, h * dk:(h + 1) * dk].double()) ** 0.25 if kind == "channel" else \
                decay[h].double().expand(lens[i], dk)
            o, S = scan(f(q[at, h * dk:(h + 1) * dk].double()) * 0.5, f(k[at, h * dk:(h + 1) * dk].double()),
                        f(v[at, h * dv:(h + 1) * dv].double()), a, state[i, h].double().T)
            want_o[at, h * dv:(h + 1) * dv], want_s[i, h] = o, S.T
    got, out = state.to(DEV), torch.full((N, heads * dv), float("nan"), device=DEV)
    how = dict(decay_logits=z.to(DEV), inv_tau=0.25) if kind == "channel" else dict(head_decay=decay.to(DEV))
    K.decay_scan(q.to(DEV), k.to(DEV), v.to(DEV), got, i32(list(range(B))), i32(cu), out, B, heads, dk, dv, q_scale=0.5, act=act,
                 max_len=max(lens), ws=Scratch(), **how)
    close(out, want_o, "outputs")
    close(got, want_s, "state")


def test_a_later_token_that_is_not_finite():
    """A value that is not finite reaches its own row and later ones, never an earlier one."""
    from mivi_v4_b200.ops import kernels as K
    N, heads, dk, dv = 100, 2, 64, 64
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(N, heads * 64, generator=g).to(DEV) for _ in "qkv")
    v[37, 5] = float("inf")
    out = torch.empty(N, heads * dv, device=DEV)
    K.decay_scan(q, k, v, torch.zeros(1, heads, dv, dk, device=DEV), i32([0]), i32([0, N]), out, 1, heads, dk, dv,
                 head_decay=torch.full((heads,), 0.9, device=DEV), max_len=N, ws=Scratch())
    assert bool(torch.isfinite(out[:37]).all()) and not bool(torch.isfinite(out[37:, 5]).any())
    assert bool(torch.isfinite(out[:, 6:]).all())
