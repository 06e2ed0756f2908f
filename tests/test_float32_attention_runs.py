"""Float32 attention of a step whose sequences bring unequal numbers of rows: long runs of rows of one sequence are worked out in tiles,
short ones a warp a row, wherever they lie; against 64 bits, and which kernel took a row by its bits and the launches."""
import math

import pytest
import torch

from mivi_v4_b200.ops import kernels as K

DEV = "cuda:0"


def test_kinds_of_runs():
    assert K.attention_runs(None) == 0 and K.attention_runs([]) == 0
    assert K.attention_runs([16, 700]) == 1 and K.attention_runs([16]) == 1
    assert K.attention_runs([1, 15]) == 2 and K.attention_runs([3] * 64) == 2
    assert K.attention_runs([15, 16]) == 0 and K.attention_runs([512] + [1] * 31) == 0


def ints(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def tile_rows(lens):
    """Which packed rows the tiles take: runs of 16 in a tile of 32, and runs that go on across its edges."""
    seq_of = [b for b, n in enumerate(lens) for _ in range(n)]
    out = []
    for i, b in enumerate(seq_of):
        lo, hi = i // 32 * 32, min(len(seq_of), i // 32 * 32 + 32)
        run = [j for j in range(lo, hi) if seq_of[j] == b]
        long = len(run) >= 16 or (run[0] == lo and lo > 0 and seq_of[lo - 1] == b)
        out.append(long or (run[-1] == hi - 1 and hi < len(seq_of) and seq_of[hi] == b))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,page,window", [(4, 2, 16, 16, 0), (2, 2, 64, 8, 37), (3, 1, 72, 64, 0), (2, 1, 128, 64, 1)])
@pytest.mark.parametrize("lens,before", [([100] + [1] * 40, [0] + [77] * 40), ([1] * 40 + [100], [77] * 40 + [5]), ([3] * 30, [50] * 30),
                                         ([15, 16, 17, 31, 32, 33, 1, 2, 64], [9] * 9), ([20, 16, 300, 64], [0, 3, 0, 130]), ([32], [1])])
def test_unequal_runs(nh, nkv, hd, page, window, lens, before):
    gen = torch.Generator().manual_seed(sum(lens) + hd)
    total = [n + c for n, c in zip(lens, before)]
    blocks = [-(-n // page) for n in total]
    order = torch.randperm(sum(blocks), generator=gen).tolist()
    pool = torch.full((sum(blocks), 2, nkv, page, hd), float("nan"))
    table, dense = torch.zeros(len(lens), max(blocks), dtype=torch.int32), []
    for b, n in enumerate(total):
        k, v = torch.randn(n, nkv, hd, generator=gen), torch.randn(n, nkv, hd, generator=gen)
        dense.append((k.double(), v.double()))
        for blk in range(blocks[b]):
            table[b, blk] = order.pop()
            lo, hi = blk * page, min(n, (blk + 1) * page)
            pool[table[b, blk], 0, :, :hi - lo] = k[lo:hi].transpose(0, 1)
            pool[table[b, blk], 1, :, :hi - lo] = v[lo:hi].transpose(0, 1)
    rows = [(b, before[b] + i) for b, n in enumerate(lens) for i in range(n)]
    N, scale, pool, table = len(rows), 1.0 / math.sqrt(hd), pool.to(DEV), table.to(DEV)
    q = torch.randn(N, nh * hd, generator=gen)
    qd, positions, seq_of = q.to(DEV), ints([p for _, p in rows]), ints([b for b, _ in rows])

    def attend(at, **how):
        out = torch.full_like(qd[at], float("nan"))
        K.attention_generic(qd[at], pool, table, positions[at], seq_of[at], out, nh, nkv, hd, scale, window, **how)
        return out
    launches, everything = K.launch_count(), slice(0, N)
    out = attend(everything, lens=lens)
    assert K.launch_count() - launches == (2 if K.attention_runs(lens) == 0 else 1)
    mixed = attend(everything)                           # without the lengths: rows for both kernels
    # 430 keys and 128 products a score in 32 bits, of values about 1
    got = out.reshape(N, nh, hd).double().cpu()
    for i, (b, p) in enumerate(rows):
        lo = max(0, p - window + 1) if window else 0
        k, v = (x[lo:p + 1].repeat_interleave(nh // nkv, 1) for x in dense[b])
        w = torch.softmax(torch.einsum("hd,thd->ht", q[i].reshape(nh, hd).double(), k) * scale, 1)
        assert torch.allclose(got[i], torch.einsum("ht,thd->hd", w, v), rtol=3e-5, atol=3e-5), (i, b, p)
    # a warp a row, as a step of fewer than 32 rows has it
    alone = torch.cat([attend(slice(i, min(i + 31, N))) for i in range(0, N, 31)])
    tiled = torch.tensor(tile_rows(lens), device=DEV)
    assert torch.equal(mixed[~tiled], alone[~tiled])
    assert not tiled.any() or window == 1 or not torch.equal(mixed[tiled], alone[tiled])
    if K.attention_runs(lens) == 0:
        assert torch.equal(out, mixed)
    elif K.attention_runs(lens) == 2:
        assert torch.equal(out, alone)
    elif tiled.all():
        assert torch.equal(out, mixed)
