"""The gated tcgen05 product where blocks work in pairs on tiles of 256 rows: full and ragged last tiles, a
pair whose second block has no rows, rows of the output that 16-byte stores cannot take, one and several
stages of K, with biases and without."""

import pytest
import torch

from test_gpu_kernels import ops  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("m,width,k", [(1024, 4608, 8), (1000, 4600, 72), (1281, 4605, 64), (1500, 8192, 520),
                                       (2049, 4608, 136), (1025, 7001, 1032)])
def test_pairs(ops, m, width, k):
    rounds = lambda rows, columns, blocks: -(-(-(-m // rows) * -(-width // columns)) // (ops._sm_count // blocks))
    assert ops._sm_count != 148 or (rounds(128, 96, 1) > rounds(128, 128, 1) >= rounds(256, 128, 2))
    generator = torch.Generator(DEVICE).manual_seed(m + width + k)
    a = torch.randn(m, k, generator=generator, device=DEVICE).bfloat16()
    w = (torch.randn(2 * width, k, generator=generator, device=DEVICE) / k ** 0.5).bfloat16()
    bias = torch.randn(2 * width, generator=generator, device=DEVICE)
    for b in (None, bias):
        got = torch.empty(m, width, dtype=torch.bfloat16, device=DEVICE)
        ops._tcgen05_call(a, w, b, got, width, ops._SWIGLU)
        ops.check_errors()
        gate, up = (a.double() @ w.double().T + (0 if b is None else b.double())).chunk(2, -1)
        want = gate * torch.sigmoid(gate) * up
        # the result's rounding to bfloat16, the fast exponential and 32-bit sums of values around one
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()


@pytest.mark.parametrize("m,n,k", [(1024, 4096, 8), (1000, 4090, 72), (1281, 8192, 64), (2049, 4100, 136),
                                   (1500, 8191, 1032)])
def test_squared_relu(ops, m, n, k):
    generator = torch.Generator(DEVICE).manual_seed(m + n + k)
    a = torch.randn(m, k, generator=generator, device=DEVICE).bfloat16()
    w = (torch.randn(n, k, generator=generator, device=DEVICE) / k ** 0.5).bfloat16()
    got = torch.empty(m, n, dtype=torch.bfloat16, device=DEVICE)
    ops._tcgen05_call(a, w, None, got, n, ops._RELU2)
    ops.check_errors()
    want = torch.relu(a.double() @ w.double().T) ** 2
    # the result's rounding to bfloat16, and 32-bit sums of values around one, squared
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
    assert torch.equal(ops.linear_act(a, w, "relu2"), got) or not ops._tcgen05(a, w, ops._RELU2)


@pytest.mark.parametrize("k", [64, 320, 384, 448])         # fewer stages of K than the ring has, as many, more
def test_pairs_one_after_the_other(ops, k):
    """A block leaves once its last stages' products have reported, so that the blocks which take its place
    find their barriers untouched: products without a pause between them have the bits of the first."""
    generator = torch.Generator(DEVICE).manual_seed(k)
    a = torch.randn(1281, k, generator=generator, device=DEVICE).bfloat16()
    w = (torch.randn(2 * 4608, k, generator=generator, device=DEVICE) / k ** 0.5).bfloat16()
    gated = [torch.empty(1281, 4608, dtype=torch.bfloat16, device=DEVICE) for _ in range(40)]
    squared = [torch.empty(1281, 2 * 4608, dtype=torch.bfloat16, device=DEVICE) for _ in range(40)]
    for one, other in zip(gated, squared):
        ops._tcgen05_call(a, w, None, one, 4608, ops._SWIGLU)
        ops._tcgen05_call(a, w, None, other, 2 * 4608, ops._RELU2)
    ops.check_errors()
    assert all(torch.equal(gated[0], one) for one in gated)
    assert all(torch.equal(squared[0], one) for one in squared)


@pytest.mark.parametrize("k,n,rows,taken", [(2048, 8192, (300, 512, 800, 850, 1040, 1240), False),
                                            (2048, 8192, (1024, 1536, 2048, 2560, 4096), True),
                                            (1024, 4096, (512, 1024, 1600, 1800), False), (1024, 4096, (2048, 3000), True)])
def test_squared_relu_where_pairs_are_faster(ops, k, n, rows, taken):
    """Tiles count by the rows that they hold: where the pairs' rounds are mostly padding the library's product and
    the activation's kernel take the call."""
    if ops._sm_count != 148:
        pytest.skip("the lines lie where 148 SMs put them")
    w = torch.empty(n, k, dtype=torch.bfloat16, device=DEVICE)
    for m in rows:
        assert ops._tcgen05(torch.empty(m, k, dtype=torch.bfloat16, device=DEVICE), w, ops._RELU2) == taken, m
