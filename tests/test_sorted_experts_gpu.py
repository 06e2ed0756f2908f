"""Steps of many tokens through experts: the sort over several rounds and with identity experts, the grouped product on tiles of 256 rows against one product an
expert, the sums of the chosen rows, and a mixture with identity experts against itself without the sort; all to the bit."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def sort(pick, E, x, in_w=None, tile_rows=128):
    k = K()
    N, top = pick.shape
    tiles = k.grouped_tiles(N * top, E, tile_rows)
    rank, place = (torch.full((N * top,), -7, dtype=torch.int32, device=DEV) for _ in range(2))
    counts, offsets = (torch.empty(E, dtype=torch.int32, device=DEV) for _ in range(2))
    tile_group = torch.empty(tiles, dtype=torch.int32, device=DEV)
    xs = torch.zeros(tiles * tile_rows, x.shape[1], dtype=x.dtype, device=DEV)
    k.expert_sort(pick, E, x, rank, counts, place, xs, offsets, tile_group, in_w=in_w, tile_rows=tile_rows)
    return counts, offsets, tile_group, place, xs


def picks(N, top, entries, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.stack([torch.randperm(entries, generator=g)[:top] for _ in range(N)]).int()


@pytest.mark.parametrize("dtype,H", [(BF, 72), (BF, 20), (torch.float32, 36), (torch.float32, 5)])        # rows of whole 16-byte words, and not
@pytest.mark.parametrize("N,top,E,identity", [(1, 1, 1, 0), (1100, 4, 7, 3), (4097, 1, 5, 0), (1365, 3, 40, 0)])
@pytest.mark.parametrize("weighted,tile_rows", [(False, 128), (True, 128), (False, 256)])
def test_sort(dtype, H, N, top, E, identity, weighted, tile_rows):
    pick = picks(N, top, E + identity, N)
    x = torch.randn(N, H, generator=torch.Generator().manual_seed(1)).to(dtype)
    w = torch.rand(N, top, generator=torch.Generator().manual_seed(2))
    counts, offsets, tile_group, place, xs = sort(pick.to(DEV), E, x.to(DEV), w.to(DEV) if weighted else None, tile_rows)
    flat = pick.flatten().long()
    order = torch.argsort(flat, stable=True)
    cnt = torch.bincount(flat, minlength=E + identity)[:E]
    start = torch.cat([torch.zeros(1, dtype=torch.long), ((cnt + tile_rows - 1) // tile_rows).cumsum(0)[:-1]]) * tile_rows
    want = torch.full((N * top,), -1)
    for e in range(E):
        mine = order[flat[order] == e]
        want[mine] = start[e] + torch.arange(len(mine))
    assert counts.cpu().tolist() == cnt.tolist() and offsets.cpu().tolist() == start.tolist() and torch.equal(place.cpu().long(), want)
    real = want >= 0
    rows = x[torch.arange(N * top) // top].float() * (w.flatten()[:, None] if weighted else 1.0)
    assert torch.equal(xs.cpu()[want[real]], rows[real].to(dtype))


@pytest.mark.parametrize("n,Hk,swiglu,clamped", [(1664, 96, True, False), (1664, 96, True, True), (96, 64, True, False), (1160, 200, False, False), (40, 72, False, False)])
@pytest.mark.parametrize("N", [3, 700, 1700])
def test_grouped_products_on_tiles_of_256_rows(n, Hk, swiglu, clamped, N):
    """One below the other (gate and up rows) and side by side (down columns)."""
    k = K()
    E, top = 5, 2
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(N, Hk, generator=g, device=DEV).to(BF)
    pick = picks(N, top, E - 1, 3)                             # the last expert: never
    counts, offsets, tile_group, place, xs = sort(pick.to(DEV), E, x, tile_rows=256)
    w = torch.randn(E * n, Hk, generator=g, device=DEV).to(BF) if swiglu else torch.randn(n, E * Hk, generator=g, device=DEV).to(BF)
    limits = k.glu_limits([(n // 2, 1.5)], 1.7, DEV) if clamped else None
    out = torch.full((xs.shape[0], n // 2 if swiglu else n), float("nan"), dtype=BF if swiglu else torch.float32, device=DEV)
    k.gemm_tc_grouped(xs, w, out, tile_group, n, Hk, row_step=n if swiglu else 0, k_step=0 if swiglu else Hk, swiglu=swiglu, limits=limits,
                      tile_rows=256)
    k.check_device_errors()
    for e in range(E):
        c, o = int(counts[e]), int(offsets[e])
        if c == 0:
            continue
        we = w[e * n:(e + 1) * n] if swiglu else w[:, e * Hk:(e + 1) * Hk].contiguous()
        want = torch.empty(c, out.shape[1], dtype=out.dtype, device=DEV)
        k.gemm_tc(xs[o:o + c].contiguous(), we, want, swiglu=swiglu, **({"limits": limits} if clamped else {}))
        assert torch.equal(out[o:o + c], want), e


@pytest.mark.parametrize("H", [64, 66])                                     # four columns a thread, and one
@pytest.mark.parametrize("top,shared,weighted", [(1, False, True), (4, True, True), (5, True, False)])
def test_combine(H, top, shared, weighted):
    k = K()
    N = 37
    g = torch.Generator(device=DEV).manual_seed(top)
    ys, sh, base = torch.randn(N * top + 11, H, generator=g, device=DEV), torch.randn(N, H, generator=g, device=DEV), torch.randn(N, H, generator=g, device=DEV)
    place = torch.randperm(N * top + 11, generator=g, device=DEV)[:N * top].int()
    w, gate = torch.rand(N, top, generator=g, device=DEV), torch.rand(N, 1, generator=g, device=DEV)
    for accumulate in (False, True):
        out = base.clone()
        k.expert_combine(ys, place, w if weighted else None, sh if shared else None, gate if shared and weighted else None, out, accumulate)
        rows = ys[place.long()].view(N, top, H).double()
        want = (rows * (w.double()[..., None] if weighted else 1.0)).sum(1)
        want = want + (sh.double() * (gate.double() if weighted else 1.0) if shared else 0.0) + (base.double() if accumulate else 0.0)
        # top + 2 additions of float32 numbers of up to some 5
        assert float((out - want).abs().max()) <= (top + 2) * 2.0 ** -23 * 5 * (top + 2)


@pytest.mark.parametrize("clamped", [False, True])
def test_identity_experts_with_and_without_the_sort(clamped, monkeypatch):
    from mivi_v4_b200.engine.step import Workspace
    from mivi_v4_b200.parts.feed_forward import RoutedExperts
    H, E, I, ff, N = 64, 6, 2, 48, 300
    part = RoutedExperts(H, E, ff, 3, n_identity=I, score="softmax", out_scale=2.0, **(dict(act="clamped", limit=0.7) if clamped else {}))
    g = torch.Generator(device=DEV).manual_seed(5)
    part.load({name: torch.randn(spec.shape, generator=g, device=DEV).to(BF) / spec.shape[-1] ** 0.5 for name, spec in part.param_specs().items()})
    x = torch.randn(N, H, generator=g, device=DEV).to(BF)
    step = types.SimpleNamespace(ws=Workspace(DEV), dtype=BF, is_decode=False, n_tokens=N)
    got = []
    for rows in (1, 1 << 30):
        monkeypatch.setattr(RoutedExperts, "SORTED_ROWS_AN_EXPERT", rows)
        assert part._sorted_up_ok(x, step, N) == (rows == 1)
        out = torch.zeros(N, H, device=DEV)
        part.forward(x, out, step, accumulate=False)
        got.append(out)
    assert torch.equal(got[0], got[1]) and float(got[0].abs().mean()) > 0.1
