"""The preparation of queries and keys in eights of values: several tokens a block with a last block
that is not full, heads shorter than the pages' rows, each norm mode, against the plain formulas."""

import pytest
import torch

from test_gpu_kernels import make_batch, ops  # noqa: F401  (fixture)
from mlx_one_b200.parts.base import PagedKeyValues, PagedView

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("tokens", [1, 5, 1023, 1025, 1030])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim,row,rotary_dim,norm_after,amplitude", [
    (32, 8, 64, 64, 64, 32, True, 1.2), (4, 2, 48, 64, 64, 16, True, 1.0), (3, 1, 128, 8, 128, 128, False, 1.1),
    (2, 2, 24, 32, 32, 0, True, 1.0), (5, 1, 256, 256, 256, 64, False, 0.9), (2, 1, 8, 8, 8, 0, True, 1.0)])
def test_preparation(ops, tokens, heads, kv_heads, dim, vdim, row, rotary_dim, norm_after, amplitude):
    page, eps, histories = 16, 1e-6, [0, 37]
    portions = [tokens] if tokens < 5 else [2, tokens - 2]
    ctx, table, pages = make_batch(portions, histories[:len(portions)], page, DEVICE)
    generator = torch.Generator().manual_seed(dim + tokens)
    wide = torch.randn(tokens, (heads + kv_heads) * dim + kv_heads * vdim + 16,
                       generator=generator).bfloat16().to(DEVICE)
    qkv = wide[:, 8:-8]
    weights = [None, None] if norm_after else [torch.rand(dim, generator=generator).to(DEVICE) + 0.5
                                               for _ in range(2)]
    frequencies = torch.rand(rotary_dim // 2, generator=generator).to(DEVICE)
    kv = torch.full((2, pages, kv_heads, page, row), 7.0, dtype=torch.bfloat16, device=DEVICE)
    q = ops.qk_norm_rope_store(qkv, heads=heads, kv_heads=kv_heads, head_dim=dim, q_weight=weights[0],
                               k_weight=weights[1], eps=eps,
                               rotary=(frequencies, rotary_dim) if rotary_dim else None, ctx=ctx,
                               view=PagedView(kv, table, page, PagedKeyValues(kv_heads, row, None)),
                               write=True, value_dim=vdim, amplitude=amplitude, norm_after=norm_after)
    ops.check_errors()

    def prepared(x, weight):
        x = x.double()
        rms = lambda y: y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)
        if weight is not None:
            x = rms(x) * weight.double()
        half = rotary_dim // 2
        if half:
            angles = (ctx.positions.float()[:, None] * frequencies[None]).double()[:, None]
            cos, sin = angles.cos() * amplitude, angles.sin() * amplitude
            a, b = x[..., :half], x[..., half:rotary_dim]
            x = torch.cat((a * cos - b * sin, b * cos + a * sin, x[..., rotary_dim:]), -1)
        return rms(x) if norm_after else x

    edge = (heads + kv_heads) * dim
    want_q = prepared(qkv[:, :heads * dim].reshape(tokens, heads, dim), weights[0])
    want_k = prepared(qkv[:, heads * dim:edge].reshape(tokens, kv_heads, dim), weights[1])
    at = table[ctx.token_request.long(), (ctx.positions // page).long()].long()
    got_k, got_v = (kv[part, at, :, (ctx.positions % page).long()] for part in (0, 1))
    # half a unit of bfloat16's last place, and 32-bit angles of up to 1,100
    for got, want in ((q[..., :dim], want_q), (got_k[..., :dim], want_k)):
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 3e-4).all()
    assert torch.equal(got_v[..., :vdim], qkv[:, edge:].reshape(tokens, kv_heads, vdim))
    assert not q[..., dim:].any() and not got_k[..., dim:].any() and not got_v[..., vdim:].any()
    assert (kv == 7.0).all(dim=-1).sum() == 2 * kv_heads * (pages * page - tokens)   # nothing else written
