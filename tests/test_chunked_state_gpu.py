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


@pytest.fixture(autouse=True, params=["few", "many"])
def kernels_for(request, monkeypatch):
    """Every case with the kernels for steps of few tokens and with those for many, whatever the step's size would choose."""
    from mivi_v4_b200.ops import kernels as K
    monkeypatch.setattr(K, "scan_takes_few", lambda *a: request.param == "few")
    return request.param


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


@pytest.mark.parametrize("tokens", [33, 64, 100])
@pytest.mark.parametrize("shift,inv_tau", [(6.0, 1 / 16), (3.0, 1 / 8), (0.0, 1.0), (-2.0, 1.0)])
def test_decay_near_one(kernels_for, tokens, shift, inv_tau):
    """Decays near 1 lose nothing by being multiplied up over a chunk.  Of an output's 2-norm: a product of up to 63 factors is rounded
    63 times (uniform in half a place either way, 0.29 * 2^-23 of a number halfway between two powers of two, so 2^-23 * 0.29 / 1.4 *
    sqrt(63) = 2.0e-7 for the oldest token of a chunk, 1.4e-7 over all), the sum over the key channels averages that down, and the
    sums' own rounding is 1.2e-7 (seen where there are few tokens): below 2.2e-7 together.  The kernels for few tokens multiply
    nothing up."""
    if kernels_for == "few":
        pytest.skip("no products of decays")
    from mivi_v4_b200.ops import kernels as K
    heads, dk, dv = 4, 128, 128
    g = torch.Generator().manual_seed(tokens)
    q, k, z = (torch.randn(tokens, heads * dk, generator=g) for _ in "qkz")
    v, z = torch.randn(tokens, heads * dv, generator=g), z + shift
    state = torch.randn(1, heads, dv, dk, generator=g)
    want = torch.zeros(tokens, heads * dv, dtype=F64)
    for h in range(heads):
        c, d = slice(h * dk, (h + 1) * dk), slice(h * dv, (h + 1) * dv)
        a = torch.exp(torch.nn.functional.logsigmoid(z[:, c].double()) * inv_tau)
        want[:, d] = scan(q[:, c].double() * 0.5, k[:, c].double(), v[:, d].double(), a, state[0, h].double().T)[0]
    out = torch.full((tokens, heads * dv), float("nan"), device=DEV)
    K.decay_scan(q.to(DEV), k.to(DEV), v.to(DEV), state.to(DEV), i32([0]), i32([0, tokens]), out, 1, heads, dk, dv, q_scale=0.5,
                 decay_logits=z.to(DEV), inv_tau=inv_tau, max_len=tokens, ws=Scratch())
    assert (out.double().cpu() - want).norm() / want.norm() <= 2.2e-7


@pytest.mark.parametrize("tokens,few", [(16, True), (320, True), (321, False)])
def test_which_kernels(monkeypatch, tokens, few):
    """Up to ten chunks of 32 tokens one after the other a step takes the two launches that suit a short prompt."""
    from mivi_v4_b200.ops import kernels as K
    monkeypatch.undo()
    x, before = torch.randn(tokens, 32, device=DEV), K.launch_count()
    K.decay_scan(x, x, x, torch.zeros(1, 1, 32, 32, device=DEV), i32([0]), i32([0, tokens]), torch.empty_like(x), 1, 1, 32, 32,
                 decay_logits=x, max_len=tokens, ws=Scratch())
    assert K.launch_count() - before == (2 if few else 3)
