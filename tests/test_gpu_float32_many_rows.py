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
    """The leading products of 16 values are cut once each where they are lined up (2^-25 of the largest at most,
    so 16 2^-25 of the sum), and their sum once behind the 24th bit (2^-23): 10 2^-24. Sections and parts are
    rounded: 2 additions within a section, 8 sections a part and one taken with the others (or K / 256 for K beyond
    2,048), 8 parts, the bias. The others are 2^-8 of the leading ones: their cuts, and l l, are below 2^-24."""
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


def absolute(*shape, generator):
    return torch.randn(shape, generator=generator, device=DEVICE).abs()


# K of one part, of parts of 256 values, of eight parts of several groups; few columns (K over clusters of 2, 4 and 8
# blocks for some numbers of rows) and many (every tile width)
@pytest.mark.parametrize("n,k", [(100, 264), (1024, 1032), (1024, 4608), (2048, 8192), (9216, 1024), (4100, 72), (600, 2056)])
def test_a_row_has_the_same_bits_among_any_others(ops, n, k):
    generator = torch.Generator(DEVICE).manual_seed(n + k)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    a, w, bias = normal(2500, k), normal(n, k), normal(n)
    whole = ops.linear(a, w, bias)
    for first, count in ((0, 131), (77, 256), (5, 300), (1, 513), (640, 640), (300, 1200), (2, 2048)):
        assert torch.equal(ops.linear(a[first:first + count], w, bias), whole[first:first + count]), (first, count)
    # up to 130 rows: the FMA kernels' order, which is theirs for any number of rows
    few = ops.linear(a[:130], w, bias)
    plain = both(ops, a[:300], w, bias)[1]
    assert torch.equal(few, plain[:130])
    allowed = bound(a[:130], w, bias) + (32 + k / 256 + 10) * 2.0 ** -24 * (
        a[:130].abs().double() @ w.abs().double().T + bias.abs().double())
    assert ((few.double() - whole[:130].double()).abs() <= allowed).all()
    ops.check_errors()


@pytest.mark.parametrize("m,n,k", [(384, 384, 256), (384, 384, 512), (384, 384, 2048), (384, 384, 8192), (1200, 9216, 1024)])
def test_products_of_one_sign(ops, m, n, k):
    """Where nothing cancels the tensor cores' cuts, all towards zero, add up: the error stays within a tenth of the
    FMA kernels' (measured 0.65 to 1.03 of it), and its mean below half of a rounding (measured 1.6e-8)."""
    generator = torch.Generator(DEVICE).manual_seed(k)
    a, w = absolute(m, k, generator=generator), absolute(n, k, generator=generator)
    got, plain = both(ops, a, w)
    want = a.double() @ w.double().T
    error, others = ((x.double() - want).norm() / want.norm() for x in (got, plain))
    assert error <= 1.1 * others, (error, others)
    assert ((got.double() - want) / want).mean().abs() <= 2.0 ** -25


@pytest.mark.parametrize("m,n,k", [(200, 100, 520), (300, 2048, 512)])
def test_values_beyond_the_scale(ops, m, n, k):
    """Inputs of 2^112 and more leave the range of bfloat16 once they are scaled: their outputs are the FMA
    kernels', as are results of 2^95 and more; results just within are not, and hold the bound."""
    generator = torch.Generator(DEVICE).manual_seed(k)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    a, w = normal(m, k), normal(n, k)
    a[3] *= 2.0 ** 118
    a[131, 5] = 2.0 ** 122
    a[7] *= 2.0 ** 80
    a[9] *= 2.0 ** -120
    w[11] *= 2.0 ** 30
    got, plain = both(ops, a, w)
    beyond = torch.zeros(m, n, dtype=torch.bool, device=DEVICE)
    beyond[[3, 131]] = True
    beyond[:, 11] = False                       # (infinities of either sign there)
    beyond[7, 11] = True
    assert torch.equal(got[beyond], plain[beyond])
    want, allowed = a.double() @ w.double().T, bound(a, w)
    for row in (0, 7, 9):
        assert ((got[row].double() - want[row]).abs() <= allowed[row] + 2.0 ** -149).all(), row


def test_an_infinity_costs_little(ops):
    """The outputs of a row with an infinity are computed again by FMAs, a warp each (by a thread each the call took
    fifteen times as long, now one and a half)."""
    generator = torch.Generator(DEVICE).manual_seed(5)
    a, w = (torch.randn(rows, 2048, generator=generator, device=DEVICE) for rows in (1200, 16384))
    odd = a.clone()
    odd[17, 3] = float("inf")

    def milliseconds(x):
        times = []
        for _ in range(4):
            events = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            events[0].record()
            ops.linear(x, w)
            events[1].record()
            torch.cuda.synchronize()
            times.append(events[0].elapsed_time(events[1]))
        return min(times)

    assert milliseconds(odd) < 6 * milliseconds(a)
    ops.check_errors()
