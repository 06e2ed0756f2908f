"""Kernels that take over at many rows: float32 attention in tiles of 32 rows (from 32 rows on), the layer norm with a warp a
row (from 592 rows on), the rounding of eight values a thread."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def ints(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("rows", [32, 33, 95])
@pytest.mark.parametrize("nh,nkv,hd,page,window", [(4, 2, 16, 16, 0), (3, 1, 72, 64, 0), (2, 2, 64, 8, 37), (2, 1, 128, 64, 1)])
def test_float32_attention_tiles(rows, nh, nkv, hd, page, window):
    lengths = [1, 33, 200, 64, 129]
    gen = torch.Generator().manual_seed(rows + hd)
    blocks = [-(-n // page) for n in lengths]
    order = torch.randperm(sum(blocks), generator=gen).tolist()
    # what no row reads: not numbers past a sequence's end, which a tile may fetch for its other rows
    pool = torch.full((sum(blocks), 2, nkv, page, hd), float("nan"))
    table = torch.zeros(len(lengths), max(blocks), dtype=torch.int32)
    dense = []
    for b, n in enumerate(lengths):
        k, v = torch.randn(n, nkv, hd, generator=gen), torch.randn(n, nkv, hd, generator=gen)
        dense.append((k, v))
        for blk in range(blocks[b]):
            table[b, blk] = order.pop()
            lo, hi = blk * page, min(n, (blk + 1) * page)
            pool[table[b, blk], 0, :, :hi - lo] = k[lo:hi].transpose(0, 1)
            pool[table[b, blk], 1, :, :hi - lo] = v[lo:hi].transpose(0, 1)
    # runs of one sequence, and rows of several sequences in one tile in any order
    queries = [(2, 199 - i) for i in range(20)] + [(b, n - 1) for b, n in enumerate(lengths)]
    while len(queries) < rows:
        b = int(torch.randint(len(lengths), (1,), generator=gen))
        queries.append((b, int(torch.randint(lengths[b], (1,), generator=gen))))
    q = torch.randn(rows, nh, hd, generator=gen)
    qd = q.reshape(rows, nh * hd).to(DEV)
    out = torch.full_like(qd, float("nan"))
    scale = 1.0 / math.sqrt(hd)
    args = (table.to(DEV), ints([p for _, p in queries]), ints([b for b, _ in queries]))
    K().attention_generic(qd, pool.to(DEV), *args, out, nh, nkv, hd, scale, window)
    # 200 keys and 128 products a score in 32 bits: (200 + 128) * 2^-24 = 2e-5 of values about 1
    got = out.reshape(rows, nh, hd).double().cpu()
    for i, (b, p) in enumerate(queries):
        lo = max(0, p - window + 1) if window else 0
        k, v = (x[lo:p + 1].double().repeat_interleave(nh // nkv, 1) for x in dense[b])
        w = torch.softmax(torch.einsum("hd,thd->ht", q[i].double(), k) * scale, 1)
        assert torch.allclose(got[i], torch.einsum("ht,thd->hd", w, v), rtol=2e-5, atol=2e-5), (i, b, p)


def test_float32_attention_infinite_value():
    """A value that is not finite reaches the rows that see it, also with a weight of 0, and no others."""
    n, hd, page = 40, 16, 64
    pool = torch.randn(1, 2, 1, page, hd, generator=torch.Generator().manual_seed(0))
    pool[0, 0, 0, 20] = -1e4                    # the key's weight is 0 in 32 bits
    pool[0, 1, 0, 20] = float("inf")
    q = torch.ones(n, hd, device=DEV)
    out = torch.zeros_like(q)
    K().attention_generic(q, pool.to(DEV), ints([[0]]), ints(list(range(n))), ints([0] * n), out, 1, 1, hd, 1.0, 0)
    out = out.cpu()
    assert out[:20].isfinite().all() and out[20:].isnan().all()


@pytest.mark.parametrize("H", [128, 256, 384, 512, 768, 1024, 1280, 1536, 1792, 2048, 2560, 3072, 3584, 4096, 4608, 1000])
@pytest.mark.parametrize("rows", [592, 593, 601])
@pytest.mark.parametrize("bias,gather,dtype", [(False, False, torch.bfloat16), (True, True, torch.bfloat16), (True, False, torch.float32)])
def test_layernorm_many_rows(H, rows, bias, gather, dtype):
    """Equal to the kernel for few rows, to the bit."""
    gen = torch.Generator().manual_seed(rows + H)
    x = (torch.randn(rows, H, generator=gen) * 3 + 1).to(DEV)
    w = torch.randn(H, generator=gen).to(DEV)
    b = torch.randn(H, generator=gen).to(DEV) if bias else None
    pick = torch.randperm(rows, generator=gen).to(torch.int32).to(DEV) if gather else None
    out = torch.empty(rows, H, dtype=dtype, device=DEV)
    K().layernorm(x, w, 1e-5, out, pick, b)
    want = torch.empty_like(out)
    for lo in range(0, rows, 300):
        hi = min(rows, lo + 300)
        part = pick[lo:hi].contiguous() if gather else torch.arange(lo, hi, dtype=torch.int32, device=DEV)
        K().layernorm(x, w, 1e-5, want[lo:hi], part, b)
    assert torch.equal(out, want)
    ref = torch.nn.functional.layer_norm(x.double()[pick.long()] if gather else x.double(), (H,), w.double(),
                                         b.double() if bias else None, 1e-5)
    # one rounding to bfloat16; sums of up to 4,608 values in 32 bits
    assert ((out.double() - ref).abs() <= ref.abs() * (2 ** -8 if dtype == torch.bfloat16 else 0) + 1e-5).all()


@pytest.mark.parametrize("n", [1, 7, 8, 2048, 2056, 4099])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_round_rows(n, off):
    x = torch.randn(n + off, generator=torch.Generator().manual_seed(n))
    x[off] = float("-inf")
    x[-1] = float("nan") if n > 1 else x[-1]
    x = x.to(DEV)[off:]
    out = torch.zeros(n + 16, dtype=torch.bfloat16, device=DEV)
    K().round_rows(x, out[8:8 + n])
    assert torch.equal(out[8:8 + n].nan_to_num(7.0), x.to(torch.bfloat16).nan_to_num(7.0))
    assert (out[:8] == 0).all() and (out[8 + n:] == 0).all()
