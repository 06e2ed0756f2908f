"""The 32-bit matrix product's two kernels (few rows: W is streamed; many rows: tiles, K cut over a cluster) and their
neighbours in the dispatch (K no multiple of 4, rows off 16 bytes) against 64 bits.

Bound: a sum of K products that is added up in order in 32 bits is off by at most K * 2^-24 times the sum of the
magnitudes; the kernels add in 2 or more parts, and rounding errors do not all point one way, so sqrt(K) * 2^-23 of it is
ample."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def rnd(*shape, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g).to(DEV)


def close(got, x, w, extra, step=0.0):
    want = x.double() @ w.double().T + extra
    room = math.sqrt(x.shape[1]) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T + abs(extra)) + step * want.abs()
    assert bool(((got.double() - want).abs() <= room + 1e-30).all())


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16, 31, 32, 33, 64, 65, 300])
@pytest.mark.parametrize("N,Kd", [(1, 4), (7, 36), (127, 100), (128, 32), (129, 1024), (300, 33), (1030, 2052), (9, 9000)])
def test_gemm_f32(M, N, Kd):
    x, w, bias, base = rnd(M, Kd), rnd(N, Kd, seed=1), rnd(N, seed=2), rnd(M, N, seed=3)
    out = torch.full((M, N), float("nan"), device=DEV)
    K().gemm_simt(x, w, out)
    close(out, x, w, 0.0)
    acc = base.clone()
    K().gemm_simt(x, w, acc, bias=bias, accumulate=True)
    close(acc, x, w, base.double() + bias.double())
    again = base.clone()
    K().gemm_simt(x, w, again, bias=bias, accumulate=True)
    assert torch.equal(acc, again)
    narrow = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    K().gemm_simt(x, w, narrow, bias=bias)
    close(narrow, x, w, bias.double(), step=2.0 ** -8)


@pytest.mark.parametrize("rows,cut,M,N,Kd", [(32, 1, 9, 65, 36), (32, 2, 1200, 129, 260), (32, 4, 600, 129, 132), (32, 8, 9, 65, 132),
                                             (64, 1, 257, 4100, 36), (64, 1, 1165, 9216, 1024), (64, 2, 257, 2049, 1024),
                                             (64, 4, 1200, 129, 2052), (64, 8, 1010, 129, 9000)])
def test_every_tile_and_cut(rows, cut, M, N, Kd):
    """Both tiles with K whole and cut in 2, 4 and 8, none of them filled; the rule that chooses them still chooses each."""
    assert K()._fn("core", "mv_gemm_f32_plan")(M, N, Kd) == rows + cut
    x, w, bias, base = rnd(M, Kd), rnd(N, Kd, seed=1), rnd(N, seed=2), rnd(M, N, seed=3)
    acc, again = base.clone(), base.clone()
    K().gemm_simt(x, w, acc, bias=bias, accumulate=True)
    close(acc, x, w, base.double() + bias.double())
    K().gemm_simt(x, w, again, bias=bias, accumulate=True)
    assert torch.equal(acc, again)


@pytest.mark.parametrize("M", [3, 40])
def test_rows_off_16_bytes(M):
    """Operands that begin 4 bytes past a 16-byte boundary take the kernel without wide loads."""
    store = rnd(M * 64 + 1)
    x, w = store[1:].view(M, 64), rnd(70, 64, seed=4)
    assert x.data_ptr() % 16 == 4
    out = torch.empty(M, 70, device=DEV)
    K().gemm_simt(x, w, out)
    close(out, x, w, 0.0)


def test_not_finite():
    """An infinity or a NaN stays in its own row and column, at tile edges too."""
    for M in (4, 70):
        x, w = rnd(M, 1028), rnd(130, 1028, seed=5)
        x[M - 1, 1027] = float("inf")
        w[129, 0] = float("nan")
        out = torch.empty(M, 130, device=DEV)
        K().gemm_simt(x, w, out)
        assert bool(torch.isnan(out[:, 129]).all()) and bool(torch.isinf(out[M - 1, :129]).all())
        assert bool(torch.isfinite(out[:M - 1, :129]).all())
