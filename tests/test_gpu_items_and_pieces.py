"""Prefill attention with one to two items an SM (tiles of 64 keys, two blocks an SM), the gate kernel's
16-byte pieces and its single values, and how many parts decode attention cuts few keys into."""

import pytest
import torch

from test_gpu_kernels import attention_case, ops, plain, tolerance  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("heads,kv_heads,portions,histories,window", [
    (16, 8, [1180], [0], None), (16, 8, [640, 1, 500], [130, 40, 0], None), (24, 8, [760, 77], [0, 300], None),
    (16, 8, [1300], [65], 200), (16, 16, [1100, 3], [0, 64], None)])
def test_prefill_with_one_to_two_items_an_sm(ops, plain, heads, kv_heads, portions, histories, window):
    tile = 128 // (heads // kv_heads)
    items = (-(-sum(portions) // tile) + len(portions)) * kv_heads
    assert ops._sm_count != 148 or 148 <= items < 296
    attention_case(ops, plain, torch.bfloat16, heads, kv_heads, 64, 16, portions=portions, histories=histories,
                   window=window, tensor_cores=True, tcgen05=True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,width", [(1, 4), (3, 8), (1000, 12), (7, 7), (129, 1024), (5, 1030)])
def test_gate_in_pieces_and_alone(ops, dtype, rows, width):
    generator = torch.Generator(DEVICE).manual_seed(rows + width)
    both = (3 * torch.randn(rows, 2 * width, generator=generator, device=DEVICE)).to(dtype)
    both[0, 0] = float("-inf")
    both[-1, -1] = float("nan")
    gate, up = both.double().chunk(2, -1)
    want = (gate / (1 + torch.exp(-gate)) * up).to(dtype)
    torch.testing.assert_close(ops.swiglu(both).float(), want.float(), equal_nan=True, **tolerance(dtype))


def test_parts_of_few_keys(ops):
    """Where three or four parts would fill the wave: one less up to 1,024 keys, as many behind more."""
    resident = ops.lib.mlxone_attention_decode_resident(64) * ops._sm_count
    for wanted, parts in ((2, 2), (3, 2), (4, 3), (5, 5)):
        blocks = resident // wanted
        assert ops.decode_splits(blocks, 1, 1, 64, 1024, None) == parts
        assert ops.decode_splits(blocks, 1, 1, 64, 2048, None) == wanted
