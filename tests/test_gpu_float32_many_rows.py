"""32-bit products of many rows on the tensor cores (each value cut into three bfloat16 parts), at the edges
of their tiles, of K's sections and of its parts over clusters, against 64 bits and the FMA kernels."""

import pytest
import torch

from test_gpu_kernels import ops  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


def both(ops, *arguments):
    """The product on the tensor cores and by FMAs; each has to have been taken."""
    kept, taken, call = ops.f32_split, [], ops._call
    ops._call = lambda name, *rest: (taken.append(name), call(name, *rest))[1]
    try:
        results = []
        for ops.f32_split in (True, False):
            results.append(ops.linear(*arguments))
    finally:
        ops.f32_split, ops._call = kept, call
    assert taken == ["mlxone_gemm_f32_split", "mlxone_gemm_f32"]
    ops.check_errors()
    return results


def bound(a, w, bias=None):
    """Of a section of 32 values the largest order is cut twice behind the 24th bit (2^-23 each) and its 32
    products once each where they are lined up (2^-25); eight sections and K / 256 sums are rounded."""
    sums = a.abs().double() @ w.abs().double().T
    if bias is not None:
        sums += bias.abs().double()
    return (4 + 16 + 8 + a.shape[1] / 256 + 1) * 2.0 ** -24 * sums


# (rows around a tile's, columns around every tile width's, K around a section's, a stage's and a group's;
# with few tiles K is cut over clusters of 2, 4 and 8 blocks)
@pytest.mark.parametrize("m,n,k", [
    (131, 1, 8), (131, 63, 24), (255, 64, 32), (256, 65, 40), (257, 161, 64), (300, 1000, 72), (131, 96, 256),
    (200, 100, 264), (131, 512, 512), (385, 2048, 1032), (131, 1024, 4608), (257, 600, 2056), (640, 4000, 288),
    (1200, 2048, 520), (1200, 2049, 256), (1153, 2400, 136), (2100, 9500, 64), (900, 3072, 96)])
def test_against_64_bits(ops, m, n, k):
    generator = torch.Generator(DEVICE).manual_seed(m * 7 + n * 3 + k)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    wide, w, bias = normal(m, k + 12), normal(n, k), normal(n)
    for a in (wide[:, 4:k + 4], wide[:, 4:k + 4].contiguous()):
        for b in (bias, None):
            got, plain = both(ops, a, w, b)
            want = a.double() @ w.double().T + (0 if b is None else b.double())
            assert ((got.double() - want).abs() <= bound(a, w, b)).all()
            if b is None and k >= 256 and n >= 64:
                assert (got.double() - want).norm() <= (plain.double() - want).norm()


def test_what_stays_with_the_fma_kernels(ops):
    """Few rows, K or rows that 16-byte loads cannot take: the FMA kernels, whose order of additions is
    one for all numbers of rows."""
    generator = torch.Generator(DEVICE).manual_seed(1)
    wide, w = torch.randn(2, 200, 530, generator=generator, device=DEVICE)[:, :, :529]
    kept = ops.f32_split
    for a, v in ((wide[:130, :520].contiguous(), w[:, :520].contiguous()), (wide[:, 1:521], w[:, :520].contiguous()),
                 (wide[:, :516].contiguous(), w[:, :516].contiguous())):
        first = ops.linear(a, v)
        try:
            ops.f32_split = False
            assert torch.equal(first, ops.linear(a, v))
        finally:
            ops.f32_split = kept


@pytest.mark.parametrize("m,n,k", [(200, 100, 520), (300, 2048, 512), (1200, 2048, 64)])
def test_values_that_are_not_ordinary(ops, m, n, k):
    """Infinities, NaN, values that bfloat16 rounds up to infinity, sums that overflow and rows of tiny
    values: the FMA kernels' results where they are not finite, 64 bits' elsewhere; other rows are as before."""
    generator = torch.Generator(DEVICE).manual_seed(k)
    a = torch.randn(m, k, generator=generator, device=DEVICE)
    w = torch.randn(n, k, generator=generator, device=DEVICE)
    clean, _ = both(ops, a, w)
    special = {3: float("inf"), 70: -float("inf"), 129: float("nan"), 150: torch.finfo(torch.float32).max}
    for row, value in special.items():
        a[row, 7] = value
    a[5] *= 1e-36
    a[6] *= 1e-40
    a[140] = 1.5e38 * a[140].sign()
    w[9, 7] = 0.0                               # (zero times infinity)
    got, plain = both(ops, a, w)
    touched = [3, 5, 6, 70, 129, 140, 150]
    others = [r for r in range(m) if r not in touched]
    keep = torch.arange(n, device=DEVICE) != 9
    assert torch.equal(got[others][:, keep], clean[others][:, keep])
    odd = ~plain.isfinite()
    assert odd[3].all() and odd[129].all() and torch.equal(odd, ~got.isfinite())
    assert torch.equal(got[odd].nan_to_num(0.0, 1.0, -1.0), plain[odd].nan_to_num(0.0, 1.0, -1.0))
    assert torch.equal(got[odd].isnan(), plain[odd].isnan())
    fine = ~odd
    a[[3, 70, 129]] = 0.0                       # (so that the bound is a number everywhere)
    want = a.double() @ w.double().T
    fine[[3, 70, 129]] = False
    # (results below 2^-126 have an absolute rounding; the FMA kernels' chains are up to 32 values long)
    error = (got.double() - want).abs()[fine]
    assert (error <= bound(a, w)[fine] * 2 + 2.0 ** -140).all()
