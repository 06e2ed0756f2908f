"""Large float32 products on the tensor cores: edges of tiles in rows, columns and K, every way a result leaves, against 64 bits; numbers that do
not split; which products go there."""
import pytest
import torch

gpu = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from mivi_v4_b200.ops import kernels
    return kernels


def test_which_products_go_there():
    takes = K().gemm_f32_tc_takes
    assert takes(1165, 1024, 4608, 148) and takes(16, 9216, 1024, 148) and not takes(8, 9216, 1024, 148)
    assert not takes(128, 1024, 4608, 148) and not takes(1165, 1024, 1020, 148) and not takes(1165, 1024, 1026, 148)


@pytest.fixture
def everything(monkeypatch):
    monkeypatch.setattr(K(), "gemm_f32_tc_takes", lambda M, N, Kd, sms: Kd % 4 == 0)


@gpu
@pytest.mark.parametrize("M", [1, 127, 128, 130, 300])
@pytest.mark.parametrize("N", [1, 95, 96, 97, 130, 1153])                      # (one tile of 96 columns, or of 128)
@pytest.mark.parametrize("Kd", [4, 32, 36, 128, 132, 1000])
def test_edges(M, N, Kd, everything):
    g = torch.Generator(device=DEV).manual_seed(M * N + Kd)
    x, w = torch.randn(M, Kd, generator=g, device=DEV), torch.randn(N, Kd, generator=g, device=DEV)
    bias, base = torch.randn(N, generator=g, device=DEV), torch.randn(M, N, generator=g, device=DEV)
    want = x.double() @ w.double().T
    # a sum of 64 of K is 4 additions (8 allowed for, and so half as many float32 additions), each cut off at 2^-22 of what they add up; then float32 additions; the smaller products, 2^-8 of it, are 5 K / 16
    # additions; the ones left out 2^-25
    size = x.double().abs() @ w.double().abs().T
    tol = size * (8 * 2.0 ** -22 + (Kd // 128 + 2) * 2.0 ** -24 + 5 * Kd / 16 * 2.0 ** -30 + 2.0 ** -25) + 2.0 ** -22 * (bias.double().abs() + base.double().abs())
    out = torch.full((M, N), float("nan"), device=DEV)
    K().gemm_simt(x, w, out)
    assert bool(((out - want).abs() <= tol).all())
    again = torch.empty_like(out)
    assert torch.equal(K().gemm_simt(x, w, again), out)                        # the same bits in every run
    K().gemm_simt(x, w, out, bias=bias)
    assert bool(((out - want - bias).abs() <= tol).all())
    K().gemm_simt(x, w, out.copy_(base), accumulate=True)
    assert bool(((out - want - base).abs() <= tol).all())
    half = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    K().gemm_simt(x, w, half)
    assert bool(((half.double() - want).abs() <= tol + 2.0 ** -8 * want.abs()).all())
    K().check_device_errors()


@gpu
@pytest.mark.parametrize("Kd", [1024, 2048, 4608])
def test_no_less_exact_than_multiply_adds(Kd, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(Kd)
    x, w = torch.randn(256, Kd, generator=g, device=DEV), torch.randn(512, Kd, generator=g, device=DEV)
    want, off = x.double() @ w.double().T, []
    for there in (True, False):
        monkeypatch.setattr(K(), "gemm_f32_tc_takes", lambda *a: there)
        out = torch.empty(256, 512, device=DEV)
        K().gemm_simt(x, w, out)
        off.append(float((out - want).norm() / want.norm()))
    assert off[0] <= off[1], off


@gpu
@pytest.mark.parametrize("Kd", [1024, 2048, 4608])
@pytest.mark.parametrize("values", ["X of one sign", "one sign", "a common offset"])
def test_how_exact_beside_multiply_adds(Kd, values, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(Kd)
    x, w = torch.randn(256, Kd, generator=g, device=DEV), torch.randn(512, Kd, generator=g, device=DEV)
    if values == "X of one sign":
        x = x.abs()
    elif values == "one sign":
        x, w = x.abs(), w.abs()
    else:
        x, w = x + 30.0, w + 1.0
    want, off = x.double() @ w.double().T, []
    for there in (True, False):
        monkeypatch.setattr(K(), "gemm_f32_tc_takes", lambda *a: there)
        out = torch.empty(256, 512, device=DEV)
        K().gemm_simt(x, w, out)
        off.append(float((out - want).norm() / want.norm()))
    if values == "X of one sign":                                              # (the terms have both)
        assert off[0] <= off[1], off
    else:
        # Sums of one sign.  The four additions of a run of 64 each cut off half a unit in the last place of the run so far, of 1/4 to 4/4 of it: 2.5 halves.  The K / 64 runs are
        # rounded to a sum that grows from nothing: 0.29 units (a rounding's deviation) times the root of a third of them.  A unit is 0.72 2^-23 of a number on average; and 15 % for the rest.
        unit = 0.72 * 2.0 ** -23
        assert off[0] <= 1.15 * unit * ((2.5 / 2) ** 2 + 0.29 ** 2 * Kd / 64 / 3) ** 0.5, off


@gpu
@pytest.mark.parametrize("e", [100, 112, 118, 122, 126, 134, 137, 145])
@pytest.mark.parametrize("small", ["x", "w"])
@pytest.mark.parametrize("large", [0, 20, 31, 33, 120])
def test_operands_far_apart(e, small, large, everything):
    """Numbers whose lower parts, or all of them, fall out of bfloat16's range, against ordinary and against large ones."""
    Kd = 1024
    g = torch.Generator(device=DEV).manual_seed(e)
    a, b = torch.randn(140, Kd, generator=g, device=DEV), torch.randn(130, Kd, generator=g, device=DEV)
    a, b = (a.double() * 2.0 ** -e).float(), b * 2.0 ** large
    b[7] = torch.randn(Kd, generator=g, device=DEV)
    a[5, ::2], a[6] = 0.0, 0.0
    x, w = (a, b) if small == "x" else (b, a)
    got, want = torch.empty(x.shape[0], w.shape[0], device=DEV), x.double() @ w.double().T
    K().gemm_simt(x, w, got)
    # K roundings of half a unit in the last place of what there is so far, of any sign; float32's steps below its smallest exponent
    row = (x.double() ** 2).sum(1)[:, None].sqrt() * (w.double() ** 2).sum(1)[None].sqrt()
    bound = 4 * 2.0 ** -24 * row + Kd * 2.0 ** -150
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound).max())
    K().check_device_errors()


@gpu
def test_numbers_that_do_not_split(everything, monkeypatch):
    """Infinities, NaNs, numbers that round to infinity in bfloat16, sums that overflow, and numbers that fall out of bfloat16's range: what multiply-adds give."""
    Kd = 96
    g = torch.Generator(device=DEV).manual_seed(1)
    x, w = torch.randn(140, Kd, generator=g, device=DEV), torch.randn(130, Kd, generator=g, device=DEV)
    x[1, 3], x[2, 5], x[3, 7], x[4, 9], x[5] = float("inf"), float("-inf"), float("nan"), 3.4e38, 3e38
    x[6] *= 1e-38
    x[7] *= 1e-30
    x[8] = 0.0
    w[2, 3], w[3, 3], w[5, 11] = 0.0, float("inf"), float("nan")
    w[4] *= 1e-20
    got, want = torch.empty(140, 130, device=DEV), torch.empty(140, 130, device=DEV)
    K().gemm_simt(x, w, got)
    monkeypatch.setattr(K(), "gemm_f32_tc_takes", lambda *a: False)
    K().gemm_simt(x, w, want)
    # a sum that overflows on the way or not hangs on its order: such elements are left out
    size = x.double().abs() @ w.double().abs().T
    sure = ~((size > 3e38) & size.isfinite())
    assert torch.equal(got[sure].isnan(), want[sure].isnan()) and torch.equal(got[sure].isinf(), want[sure].isinf())
    fine = sure & want.isfinite()
    assert bool(((got - want).abs()[fine].double() <= 2.0 ** -18 * size[fine] + 2.0 ** -149).all()) and bool((got[:, 3][sure[:, 3]].isfinite() == want[:, 3][sure[:, 3]].isfinite()).all())
