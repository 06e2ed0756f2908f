"""The row kernels that steps of many tokens take, against the ones that steps of few tokens or unaligned rows take, to the bit; and those without such a
twin against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def strided(x, ld):
    wide = torch.full((x.shape[0], ld), float("nan"), device=DEV)
    wide[:, :x.shape[1]] = x
    return wide


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("nh,nkv,dk,dv,dims,per_head,norms", [(6, 2, 64, 64, 64, True, "qk"), (3, 1, 20, 12, 8, True, "q"), (5, 5, 36, 4, 16, False, "qk"),
                                                              (4, 2, 128, 64, 0, False, "k"), (2, 0, 256, 4, 256, True, ""), (1, 1, 4, 4, 0, False, "")])
def test_queries_keys_and_values(dtype, nh, nkv, dk, dv, dims, per_head, norms):
    k, N, page = K(), 259, 16
    need = nh * dk + nkv * (dk + dv)
    proj = rnd(N, need)
    wq = rnd(dk if per_head else nh * dk, seed=1) if "q" in norms else None
    wk = rnd(dk if per_head else nkv * dk, seed=2) if "k" in norms else None
    inv = 10000.0 ** (-torch.arange(dims // 2, device=DEV) / max(dims // 2, 1)) if dims else None
    pos, seq_of = i32([i % 200 for i in range(N)]), i32([i // 200 for i in range(N)])
    table = torch.randperm(26, generator=torch.Generator().manual_seed(3)).int().view(2, 13).to(DEV)
    got = []
    for ld in (-(-need // 4) * 4, need | 1):                   # rows on 16 bytes, and not
        q = torch.zeros(N, nh * dk, dtype=dtype, device=DEV)
        pool = torch.zeros(26, max(nkv, 1) * page * (dk + dv), dtype=dtype, device=DEV)
        k.qkv_prepare_wide(strided(proj, ld), wq, wk, 1e-5, dims, inv, pos, seq_of, table, pool, page, q, nh, nkv, dk, dv, per_head=per_head,
                           amplitude=1.1, q_temp=(0.1, 50.0))
        got.append((q, pool))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert got[0][0].abs().max() > 0 and (nkv == 0 or got[0][1].abs().max() > 0)


@pytest.mark.parametrize("nh,dim,rot,dims", [(3, 64, 32, 32), (2, 20, 12, 8), (1, 4, 4, 0)])
def test_latent_queries(nh, dim, rot, dims):
    k, N = K(), 37
    proj = rnd(N, nh * (dim + rot))
    inv = 10000.0 ** (-torch.arange(dims // 2, device=DEV) / max(dims // 2, 1)) if dims else None
    pos = i32([7 * i for i in range(N)])
    got = [k.latent_query(strided(proj, ld), 0, inv, pos, torch.zeros(N, nh, dim + rot, dtype=BF, device=DEV), nh, dim, rot, dims, amplitude=0.9)
           for ld in (proj.shape[1], proj.shape[1] + 1)]
    assert torch.equal(*got) and got[0].abs().max() > 0


@pytest.mark.parametrize("dtype", [BF, torch.float32])
@pytest.mark.parametrize("N,rank,rot,dims,q_rank", [(768, 256, 32, 32, 512), (771, 37, 6, 4, 0), (801, 300, 8, 8, 1000), (769, 8, 4, 0, 5)])
def test_latent_rows(dtype, N, rank, rot, dims, q_rank):
    k, page = K(), 32
    proj = rnd(N, rank + rot + q_rank)
    w, wq = rnd(rank, seed=1), rnd(max(q_rank, 1), seed=2)[:q_rank]
    inv = 10000.0 ** (-torch.arange(dims // 2, device=DEV) / max(dims // 2, 1)) if dims else None
    pos, seq_of, table = i32(list(range(N))), i32([0] * N), i32([list(range(26))[::-1]])
    got = []
    for n in (N, 100):                                         # all tokens in one call, and in calls of few tokens
        pool = torch.zeros(26, page * (rank + rot), dtype=dtype, device=DEV)
        cq = torch.zeros(N, q_rank, dtype=dtype, device=DEV) if q_rank else None
        for a in range(0, N, n):
            rows = slice(a, min(a + n, N))
            k.latent_prepare(proj[rows], 0, 0, w, 1e-5, inv, pos[rows], seq_of[rows], table, pool, page, None, 2, 4, rot, rank, dims, cq0=rank + rot,
                             w_q=wq if q_rank else None, cq=cq[rows] if q_rank else None, amplitude=1.2)
        got.append((pool, cq if q_rank else pool))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][1].abs().max() > 0


@pytest.mark.parametrize("act", [True, False])
@pytest.mark.parametrize("C,lens", [(2048, [1, 2, 3, 765]), (516, [3049]), (1028, [7, 8, 9, 1550, 1]), (3072, [2] * 257)])
def test_causal_conv(act, C, lens):
    k, N, B = K(), sum(lens), len(lens)
    u, taps, bias = rnd(N, C), rnd(C, 4, seed=1), rnd(C, seed=2)
    cu = i32([sum(lens[:i]) for i in range(B + 1)])
    seq_of = i32([b for b, n in enumerate(lens) for _ in range(n)])
    slots = i32(list(range(B))[::-1])
    got = []
    for ld in (C, C + 1):
        state = rnd(B, 3, C, seed=3)
        out = k.causal_conv(strided(u, ld)[:, :C], taps, bias, state, seq_of, cu, slots, torch.zeros(N, C, device=DEV), B, act=act)
        got.append((out, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][0].abs().max() > 0


@pytest.mark.parametrize("lens", [[65], [512], [513, 100], [1, 1100, 0, 31, 32]])
def test_gates_of_a_matrix_memory(lens):
    k, H, B = K(), 3, len(lens)
    N = sum(lens)
    z, bi, bf = 4 * rnd(N, 2 * H), rnd(H, seed=1), rnd(H, seed=2)
    starts = [sum(lens[:i]) for i in range(B + 1)]
    got = []
    for n in (N, 64):                                          # whole sequences in one call, and 64 tokens a call
        m_state = rnd(B, H, seed=3)
        outs = [torch.zeros(N, H, device=DEV) for _ in range(3)]
        if n == N:
            k.memory_gates(z[:, :H], z[:, H:], bi, bf, 6.0, m_state, i32(list(range(B))), i32(starts), *outs, B, H)
        else:
            for b in range(B):
                for a in range(starts[b], starts[b + 1], n):
                    rows = slice(a, min(a + n, starts[b + 1]))
                    k.memory_gates(z[rows, :H], z[rows, H:], bi, bf, 6.0, m_state, i32([b]), i32([0, rows.stop - a]), *(o[rows] for o in outs), 1, H)
        got.append(outs + [m_state])
    assert all(torch.equal(a, b) for a, b in zip(*got)) and got[0][2].abs().max() > 0


# A float32 sum of squares over n values, its terms all of one sign, is off by at most about (n / threads + 11) 2^-24 of itself, half of that after the
# root; the few roundings after it and the exponential (2 ulp) add 2^-21 of the result: 2e-6 of it covers n = 5,000 over 128 threads.
@pytest.mark.parametrize("act", [0, 1, 2])
@pytest.mark.parametrize("group", [300, 512, 1023, 2048, 2049, 4096, 4097, 5000])
@pytest.mark.parametrize("shared", [True, False])
def test_gated_norm(act, group, shared):
    k, N, C, eps = K(), 5, 2 * group, 1e-5
    x, gate, w = rnd(N, C), rnd(N, C, seed=1), rnd(group if shared else C, seed=2)
    out = k.gated_rmsnorm(x, gate, w, group, eps, act, torch.zeros(N, C, device=DEV))
    x, gate, w = x.double(), gate.double(), w.double().repeat(2 if shared else 1)
    f = torch.nn.functional.silu(gate) if act != 1 else torch.sigmoid(gate)
    if act == 2:
        x = x * f
    want = (x.view(N, 2, group) / (x.view(N, 2, group).pow(2).mean(-1, keepdim=True) + eps).sqrt()).view(N, C) * w
    if act != 2:
        want = want * f
    assert ((out.double() - want).abs() <= 2e-6 * want.abs() + 1e-12).all()


# The norm's rounding as above, its sum with the residual one more rounding of the sum; the layer norm takes a mean away that is within 2e-6 of the
# rows' size, here at most 4, and divides by a deviation of about one: 2e-5 covers the sums' errors with their subtraction.
@pytest.mark.parametrize("H", [4, 100, 512, 513, 1024, 1025, 2047, 2048, 2049])
def test_norm_into_the_residual_and_its_layer_norm(H):
    k, N = K(), 3
    y, w, resid, lw = rnd(N, H), rnd(H, seed=1), rnd(N, H, seed=2), rnd(H, seed=3)
    r64 = resid.double() + y.double() / (y.double().pow(2).mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    want = torch.nn.functional.layer_norm(r64, (H,), lw.double(), eps=1e-5)
    out = k.rmsnorm_add_layernorm(y, w, 1e-6, resid, lw, 1e-5, torch.zeros(N, H, device=DEV))
    assert (resid.double() - r64).abs().max() <= 2e-6 * r64.abs().max() and (out.double() - want).abs().max() <= 2e-5 * want.abs().max()
