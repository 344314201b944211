"""Prefill attention with one to two items an SM (tiles of 128 keys, or of 64 with two blocks an SM), the gate
kernel's 16-byte pieces and its single values, and how many parts decode attention cuts few keys into."""

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


@pytest.mark.parametrize("tokens,requests,heads,max_context,window,keys", [
    (704, 1, 32, 704, 0, 128), (704, 1, 32, 1216, 0, 128), (704, 1, 32, 2752, 0, 64), (688, 1, 32, 2752, 0, 128),
    (2048, 1, 16, 2048, 0, 128), (2048, 1, 16, 4096, 0, 128), (2048, 1, 16, 6144, 0, 64), (2016, 1, 16, 8192, 0, 128),
    (735, 1, 24, 9000, 0, 128),                     # 144 items: fewer than SMs
    (560, 1, 32, 9000, 0, 128), (2304, 1, 16, 2304, 0, 128), (2368, 1, 16, 2368, 0, 64),    # ... two for every SM
    (1019, 1, 32, 7019, 1024, 64), (1019, 1, 32, 1019, 1024, 128), (1043, 1, 32, 1043, 512, 64),
    (1019, 1, 32, 7019, -512, 64),
    (512, 4, 32, 200, 0, 128), (608, 4, 32, 152, 0, 64), (320, 16, 32, 20, 0, 128), (256, 64, 32, 4, 0, 64)])
def test_keys_a_tile(ops, tokens, requests, heads, max_context, window, keys):
    """At the measured points on both sides of every line."""
    if ops._sm_count != 148:
        pytest.skip("the lines lie where 148 SMs put them")
    assert ops.lib.mlxone_attention_tcgen05_keys(tokens, requests, heads, 8, max_context, window, 1) == keys
    assert ops.lib.mlxone_attention_tcgen05_keys(tokens, requests, heads, 8, max_context, window, 2) == 64


@pytest.mark.parametrize("portions,histories,window", [
    ([1216], [2500], None), ([1216], [100], None), ([1190], [2500], None), ([1184], [1500], 512), ([1190], [40], 300),
    ([592, 592], [40, 700], None)])
def test_prefill_on_both_sides_of_the_line(ops, plain, portions, histories, window):
    """152 items of 16 heads over 8: one request, whole and ragged last tiles behind few and many keys and with
    windows; two requests."""
    attention_case(ops, plain, torch.bfloat16, 16, 8, 64, 16, portions=portions, histories=histories,
                   window=window, tensor_cores=True, tcgen05=True)


def test_parts_where_clusters_of_three_find_no_place(ops):
    if ops._sm_count != 148:
        pytest.skip("the lines lie where 148 SMs put them")
    for heads, kv_heads, dim, requests, parts in (
            (24, 8, 64, 23, 3), (24, 8, 64, 24, 2), (32, 8, 128, 11, 3), (32, 8, 128, 12, 2), (16, 4, 64, 46, 3),
            (16, 4, 64, 48, 2), (8, 2, 32, 160, 3), (8, 2, 32, 168, 2), (24, 8, 64, 16, 3), (32, 8, 128, 9, 4)):
        assert ops.decode_splits(requests, heads, kv_heads, dim, 1024, None) == parts, (heads, kv_heads, dim, requests)
    assert ops.decode_splits(24, 24, 8, 64, 2048, None) == 3
