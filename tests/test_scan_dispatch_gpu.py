"""Long steps of the scans with one decay a token and of the delta rule, at the edges of their chunks, tiles and lanes, against
the recurrences in 64 bits: chunks of 32 and 16 tokens full, one short and one over; value columns off the tiles of 64 and 16; key
sizes on both sides of 64, 128; strides off 16 bytes; a slot that is not in the step.

Bound: sums of T products of numbers of order 1 in 32 bits, T a few hundred: 64 * 2^-24 of the largest value, four times that where
a decay's exponent is a difference of sums of up to 100."""
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


def starts_of(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


def close(got, want, tol, what):
    err = (got.double().cpu() - want).abs().max().item() / want.abs().max().item()
    assert err <= tol, f"{what}: off by {err:.3g} of the largest value"


@pytest.mark.parametrize("heads,group,dk,dv,pad", [(1, 1, 128, 64, 0), (2, 2, 33, 65, 0), (3, 1, 4, 7, 1), (6, 3, 64, 64, 3), (2, 1, 200, 66, 0)])
@pytest.mark.parametrize("lens", [[32], [16, 1, 33], [95, 64]])
@pytest.mark.parametrize("normalizer", [False, True])
@pytest.mark.parametrize("few", [False, True])               # the kernels for many tokens, and those for few
def test_scalar_scan(monkeypatch, heads, group, dk, dv, pad, lens, normalizer, few):
    from mivi_v4_b200.ops import kernels as K
    monkeypatch.setattr(K, "scan_takes_few", lambda *a: few)
    g = torch.Generator().manual_seed(heads * 1000 + dk + sum(lens))
    N, groups, B, cu = sum(lens), heads // group, len(lens), starts_of(lens)
    q, k = (torch.randn(N, groups * dk, generator=g) for _ in "qk")
    v = torch.randn(N, heads * dv, generator=g)
    log_a = -torch.rand(N, heads, generator=g) * torch.tensor([0.01, 1.0, 3.0])[torch.arange(heads) % 3]
    b, m = torch.rand(N, heads, generator=g) + 0.1, torch.randn(N, heads, generator=g)
    skip = None if normalizer else torch.randn(heads, generator=g)
    state = torch.randn(B + 1, heads, dv + int(normalizer), dk, generator=g)
    slots = [B - i for i in range(B)]
    want_o, want_s = torch.zeros(N, heads * dv, dtype=F64), state.double().clone()
    room, largest = torch.zeros_like(want_o), 0.0
    for i in range(B):
        for h in range(heads):
            S, hk = state[slots[i], h].double().T.clone(), h // group
            for t in range(cu[i], cu[i + 1]):
                vt = v[t, h * dv:(h + 1) * dv].double()
                va = torch.cat([vt, torch.ones(1, dtype=F64)]) if normalizer else vt
                S = log_a[t, h].double().exp() * S + b[t, h].double() * k[t, hk * dk:(hk + 1) * dk].double()[:, None] * va[None]
                o = S.T @ (q[t, hk * dk:(hk + 1) * dk].double() * 0.5)
                if normalizer:
                    den = torch.maximum(o[-1].abs(), torch.exp(-m[t, h].double())) + 1e-6
                    room[t, h * dv:(h + 1) * dv] = 1 / den + (o[:-1] / den).abs() / den
                    largest = max(largest, o.abs().max().item())
                    o = o[:-1] / den
                else:
                    o = o + skip[h].double() * vt
                want_o[t, h * dv:(h + 1) * dv] = o
            want_s[slots[i], h] = S.T
    wide = torch.zeros(N, q.shape[1] + pad)          # a row stride that is no multiple of 16 bytes
    wide[:, pad:] = q
    got, out = state.to(DEV), torch.full((N, heads * dv), float("nan"), device=DEV)
    K.scalar_scan(wide.to(DEV)[:, pad:], k.to(DEV), v.to(DEV), log_a.to(DEV), b.to(DEV), got, i32(slots), i32(cu), out, B, heads, dk, dv,
                  heads_per_group=group, skip=None if skip is None else skip.to(DEV), m_tok=m.to(DEV) if normalizer else None,
                  q_scale=0.5, max_len=max(lens), ws=Scratch())
    if normalizer:
        # a quotient of two such sums x / d, either off by 1.6e-5 of the largest: off by that much times 1 / d + |x / d| / d
        assert bool(((out.double().cpu() - want_o).abs() <= 1.6e-5 * largest * room).all())
    else:
        close(out, want_o, 1.6e-5, "outputs")
    close(got, want_s, 1.6e-5, "state")
    assert torch.equal(got[0].cpu(), state[0])


@pytest.mark.parametrize("heads,kv,dk,dv", [(2, 1, 128, 16), (2, 2, 64, 17), (3, 1, 65, 40), (2, 1, 130, 33), (1, 1, 192, 16), (2, 1, 193, 9),
                                            (1, 1, 256, 8), (2, 1, 63, 20)])
@pytest.mark.parametrize("lens", [[16], [8, 17], [47, 1, 32]])
@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_scan(heads, kv, dk, dv, lens, head_decay):
    from mivi_v4_b200.ops import kernels as K
    g = torch.Generator().manual_seed(heads * 1000 + dk + sum(lens))
    N, B, cu, n_a = sum(lens), len(lens), starts_of(lens), heads if head_decay else heads * dk
    q, k = (torch.randn(N, kv * dk, generator=g) for _ in "qk")
    v, beta, a = torch.randn(N, heads * dv, generator=g), torch.randn(N, heads, generator=g), torch.randn(N, n_a, generator=g)
    bias, a_log = torch.randn(n_a, generator=g) * 0.1, torch.randn(heads, generator=g) * 0.1
    state = torch.randn(B + 1, heads, dv, dk, generator=g)
    slots = [B - i for i in range(B)]
    want_o, want_s = torch.zeros(N, heads * dv, dtype=F64), state.double().clone()
    decay = torch.exp(-torch.exp(a_log.double()).repeat_interleave(n_a // heads) * torch.nn.functional.softplus(a.double() + bias.double(), threshold=1e9))
    for i in range(B):
        for h in range(heads):
            S, hk = state[slots[i], h].double().T.clone(), h // (heads // kv)
            for t in range(cu[i], cu[i + 1]):
                kt, qt = (x[t, hk * dk:(hk + 1) * dk].double() for x in (k, q))
                kt, qt = kt / torch.sqrt((kt * kt).sum() + 1e-6), qt / torch.sqrt((qt * qt).sum() + 1e-6) * 0.3
                S = (decay[t, h] if head_decay else decay[t, h * dk:(h + 1) * dk][:, None]) * S
                S = S + kt[:, None] * (torch.sigmoid(beta[t, h].double()) * (v[t, h * dv:(h + 1) * dv].double() - S.T @ kt))[None]
                want_o[t, h * dv:(h + 1) * dv] = S.T @ qt
            want_s[slots[i], h] = S.T
    got, out = state.to(DEV), torch.full((N, heads * dv), float("nan"), device=DEV)
    K.delta_scan(q.to(DEV), k.to(DEV), v.to(DEV), beta.to(DEV), a.to(DEV), bias.to(DEV), a_log.to(DEV), got, i32(slots), i32(cu), out, B,
                 heads, kv, dk, dv, q_scale=0.3, max_len=max(lens), ws=Scratch(), head_decay=head_decay)
    close(out, want_o, 4e-6, "outputs")
    close(got, want_s, 4e-6, "state")
    assert torch.equal(got[0].cpu(), state[0])


def test_scalar_scan_few_and_many_agree(monkeypatch):
    """Which kernels a step takes depends on its tokens; the bits do not."""
    from mivi_v4_b200.ops import kernels as K
    g = torch.Generator(device=DEV).manual_seed(5)
    for heads, group, dk, dv, norm, lens in ((4, 4, 128, 64, 0, [127]), (2, 1, 128, 66, 1, [50, 33]), (2, 1, 200, 40, 1, [64, 1, 40])):
        N, B = sum(lens), len(lens)
        r = lambda *s: torch.randn(*s, generator=g, device=DEV)
        q, k, v, m = r(N, heads // group * dk), r(N, heads // group * dk), r(N, heads * dv), r(N, heads)
        log_a, b, state = -r(N, heads).abs(), r(N, heads).abs(), r(B, heads, dv + norm, dk)
        got = []
        for few in (False, True):
            monkeypatch.setattr(K, "scan_takes_few", lambda *a: few)
            s, out = state.clone(), torch.full((N, heads * dv), float("nan"), device=DEV)
            K.scalar_scan(q, k, v, log_a, b, s, i32(list(range(B))), i32(starts_of(lens)), out, B, heads, dk, dv, heads_per_group=group,
                          m_tok=m if norm else None, q_scale=0.1, max_len=max(lens), ws=Scratch())
            got.append((out, s))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("tokens,few", [(16, True), (160, True), (161, False)])
def test_which_kernels(tokens, few):
    from mivi_v4_b200.ops import kernels as K
    x, ones, before = torch.randn(tokens, 32, device=DEV), torch.ones(tokens, 1, device=DEV), K.launch_count()
    K.scalar_scan(x, x, x, -ones, ones, torch.zeros(1, 1, 32, 32, device=DEV), i32([0]), i32([0, tokens]), torch.empty_like(x), 1, 1, 32, 32,
                  max_len=tokens, ws=Scratch())
    assert K.launch_count() - before == (2 if few else 4)
