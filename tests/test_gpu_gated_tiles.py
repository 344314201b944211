"""The gated tcgen05 product at sizes for which its narrower tiles (96 + 96 rows of the weights) take
no more rounds over the SMs: full and ragged last tiles, rows of the output that 16-byte stores cannot
take, one and several values of K a stage."""

import pytest
import torch

from test_gpu_kernels import ops  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("m,width,k", [(300, 6912, 64), (424, 6912, 1536), (257, 6904, 72), (300, 6850, 192),
                                       (384, 6816, 8), (511, 6815, 136)])
def test_narrower_tiles(ops, m, width, k):
    rounds = lambda columns: -(-(-(-m // 128) * -(-width // columns)) // ops._sm_count)
    assert ops._sm_count != 148 or rounds(96) <= rounds(128)
    generator = torch.Generator(DEVICE).manual_seed(m + width + k)
    a = torch.randn(m, k, generator=generator, device=DEVICE).bfloat16()
    w = (torch.randn(2 * width, k, generator=generator, device=DEVICE) / k ** 0.5).bfloat16()
    kept, ops.tcgen05_always = ops.tcgen05_always, True
    try:
        assert ops._tcgen05(a, w, ops._SWIGLU)
        got = ops.linear_swiglu(a, w)
    finally:
        ops.tcgen05_always = kept
    ops.check_errors()
    gate, up = (a.double() @ w.double().T).chunk(2, -1)
    want = gate * torch.sigmoid(gate) * up
    # the result's rounding to bfloat16, the fast exponential and 32-bit sums of values around one
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()
