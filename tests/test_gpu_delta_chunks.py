"""The gated delta rule over portions that are worked on 32 tokens at a time: portions at the edges of
a chunk, several requests in a step, decays of zero, against the plain recurrence token by token."""

import pytest
import torch

from test_gpu_galarax import DEVICE, DTYPES, bound, context, delta_pieces, ops  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def short_portions_in_chunks_too(ops):
    kept, ops.delta_chunk_from = ops.delta_chunk_from, 8
    yield
    ops.delta_chunk_from = kept


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads, kv_heads, value_dim", [(2, 1, 16), (3, 3, 48), (20, 2, 32)])
@pytest.mark.parametrize("steps", [[(32, 40)], [(33, 31)], [(64, 1), (95, 65)], [(1, 70), (127, 3), (1, 30)],
                                   [(40, 30), (7, 8), (8, 8)]])
@pytest.mark.parametrize("forget", [-5.0, 5.0])
def test_portions_around_a_chunk(ops, dtype, heads, kv_heads, value_dim, steps, forget):
    """``forget``: log of the decay's rate; at 5 most decays are zero in 32-bit."""
    from mlx_one_b200.parts import FixedState, StateView
    from mlx_one_b200.parts.mixers import GatedDeltaRule

    H, G, D, V, taps = heads, kv_heads, 128, value_dim, 4
    sizes = dict(heads=H, kv_heads=G, key_dim=D, value_dim=V, taps=taps)
    channels, inner = 2 * G * D + H * V, H * V
    width = channels + inner + 2 * H
    generator = torch.Generator().manual_seed(V)
    lengths = [sum(step[r] for step in steps) for r in (0, 1)]
    projected = [(1.5 * torch.randn(n, width, generator=generator)).to(dtype) for n in lengths]
    conv = 0.5 * torch.randn(channels, taps, generator=generator)
    a_log = forget + torch.randn(H, generator=generator)
    dt_bias, eps = torch.randn(H, generator=generator), 1e-5
    norm_weight = 1 + 0.2 * torch.randn(V, generator=generator)
    size = GatedDeltaRule.state_size(sizes)
    state = torch.full((5, size), float("nan"), device=DEVICE)
    state[[3, 1]] = 0
    slots = torch.tensor([3, 1], dtype=torch.int32, device=DEVICE)
    view = StateView(state, slots, FixedState((size,), "float32"))
    constants = dict(conv=conv.to(DEVICE), a_log=a_log.to(DEVICE), dt_bias=dt_bias.to(DEVICE),
                     norm_weight=norm_weight.to(DEVICE), eps=eps, unit_eps=1e-6, view=view, write=True,
                     **sizes)
    got, fed = [[], []], [0, 0]
    for step in steps:
        rows = torch.cat([projected[r][fed[r]:fed[r] + step[r]] for r in (0, 1)]).to(DEVICE)
        before = ops.launches
        out = ops.gated_delta_rule(rows, ctx=context(list(step), list(fed)), **constants)
        assert ops.launches - before == 4          # preparation, chunks, walk, finish
        got[0].append(out[:step[0]].cpu())
        got[1].append(out[step[0]:].cpu())
        fed = [fed[r] + step[r] for r in (0, 1)]
    ops.check_errors()
    for r in (0, 1):
        want = delta_pieces(projected[r].double(), conv.double(), a_log.double(), dt_bias.double(),
                            norm_weight.double(), eps, sizes)
        difference = (torch.cat(got[r]).double() - want).abs().max()
        # (the bounds of the recurrence's own test: 32-bit sums, 8 bits of mantissa at values of up to 8)
        assert difference < bound(dtype, 5e-5, 0.1), f"request {r}: {difference}"
    assert torch.isnan(state[[0, 2, 4]]).all() and torch.isfinite(state[[1, 3]]).all()


@pytest.mark.parametrize("part", ["query", "key", "value", "gate", "beta", "decay"])
@pytest.mark.parametrize("spoilt", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [1, 37, 69])
def test_what_is_not_finite_stays_behind_its_token(ops, part, spoilt, at):
    """An infinity or NaN in one token of a portion of 70 (in the middle of a chunk of 32, near its start
    and in the last, short one): the tokens before it keep their bits, other requests too."""
    from mlx_one_b200.parts import FixedState, StateView
    from mlx_one_b200.parts.mixers import GatedDeltaRule

    H, G, D, V, taps = 4, 2, 128, 32, 4
    sizes = dict(heads=H, kv_heads=G, key_dim=D, value_dim=V, taps=taps)
    channels, inner = 2 * G * D + H * V, H * V
    column = {"query": 5, "key": G * D + 5, "value": 2 * G * D + 5, "gate": channels + 5,
              "beta": channels + inner, "decay": channels + inner + H}[part]
    generator = torch.Generator(DEVICE).manual_seed(3)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    rows = normal(70 + 40, channels + inner + 2 * H)
    constants = dict(conv=0.5 * normal(channels, taps), a_log=normal(H) - 2, dt_bias=normal(H),
                     norm_weight=1 + 0.2 * normal(V), eps=1e-5, unit_eps=1e-6, write=True, **sizes)
    outputs = []
    for value in (None, spoilt):
        if value is not None:
            rows[at, column] = value
        size = GatedDeltaRule.state_size(sizes)
        view = StateView(torch.zeros(2, size, device=DEVICE),
                         torch.tensor([1, 0], dtype=torch.int32, device=DEVICE), FixedState((size,), "float32"))
        outputs.append(ops.gated_delta_rule(rows, ctx=context([70, 40], [0, 0]), view=view, **constants))
    ops.check_errors()
    assert torch.isfinite(outputs[0]).all()
    assert torch.equal(outputs[1][:at], outputs[0][:at]) and torch.equal(outputs[1][70:], outputs[0][70:])
    if part in ("value", "key"):
        assert not torch.isfinite(outputs[1][at]).all()


@pytest.mark.parametrize("portion", [1, 5, 7, 8, 40, 63, 64])
@pytest.mark.parametrize("chunk_from", [8, 64])
@pytest.mark.parametrize("beside, lead", [([1] * 30, 30), ([1] * 30, 4), ([2, 3], 0), ([100], 0), ([7, 300, 1], 0)])
def test_a_portion_does_not_depend_on_its_neighbours(ops, portion, chunk_from, beside, lead):
    """A request's portion by itself and behind others of all kinds (the first ``lead`` of them known to
    bring one token): the same output and the same state, bit for bit."""
    ops.delta_chunk_from = chunk_from
    from mlx_one_b200.parts import FixedState, StateView
    from mlx_one_b200.parts.mixers import GatedDeltaRule

    sizes = dict(heads=4, kv_heads=2, key_dim=128, value_dim=48, taps=4)
    channels, inner = 2 * 2 * 128 + 4 * 48, 4 * 48
    generator = torch.Generator(DEVICE).manual_seed(portion)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    constants = dict(conv=0.5 * normal(channels, 4), a_log=normal(4) - 2, dt_bias=normal(4),
                     norm_weight=1 + 0.2 * normal(48), eps=1e-5, unit_eps=1e-6, write=True, **sizes)
    rows = normal(sum(beside) + portion, channels + inner + 8)
    size = GatedDeltaRule.state_size(sizes)
    kept = normal(len(beside) + 1, size)
    results = []
    for portions in ([portion], list(beside) + [portion]):
        n = len(portions)
        state = kept[-n:].clone()
        ctx = context(portions, [9] * n)
        ctx.leading_single = lead if n > 1 and portion > 1 else 0
        # (one token by itself runs in the kernel of single tokens: here it is a portion all the same)
        ctx.max_portion = max(ctx.max_portion, 2)
        view = StateView(state, torch.arange(n, dtype=torch.int32, device=DEVICE), FixedState((size,), "float32"))
        out = ops.gated_delta_rule(rows[-sum(portions):].contiguous(), ctx=ctx, view=view, **constants)
        results.append((out[-portion:].clone(), state[-1].clone()))
    ops.check_errors()
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("offset", [0, 2])
def test_values_of_128(ops, dtype, offset):
    """Eight tiles of columns in the walk, the largest block of the single-token kernel, and the output's norm
    four values a lane, or one where the rows do not allow it (``offset``): portions, single tokens, portions."""
    from mlx_one_b200.parts import FixedState, StateView
    from mlx_one_b200.parts.mixers import GatedDeltaRule

    H, G, D, V, taps = 4, 2, 128, 128, 4
    sizes = dict(heads=H, kv_heads=G, key_dim=D, value_dim=V, taps=taps)
    channels, inner = 2 * G * D + H * V, H * V
    width = channels + inner + 2 * H
    generator = torch.Generator().manual_seed(11)
    steps = [(70, 33), (1, 1), (1, 1), (1, 1), (2, 1), (65, 64), (1, 1)]
    lengths = [sum(step[r] for step in steps) for r in (0, 1)]
    projected = [(1.5 * torch.randn(n, width, generator=generator)).to(dtype) for n in lengths]
    conv = 0.5 * torch.randn(channels, taps, generator=generator)
    a_log, dt_bias = torch.randn(H, generator=generator) - 2, torch.randn(H, generator=generator)
    norm_weight = 1 + 0.2 * torch.randn(V, generator=generator)
    size = GatedDeltaRule.state_size(sizes)
    view = StateView(torch.zeros(2, size, device=DEVICE), torch.tensor([1, 0], dtype=torch.int32, device=DEVICE),
                     FixedState((size,), "float32"))
    constants = dict(conv=conv.to(DEVICE), a_log=a_log.to(DEVICE), dt_bias=dt_bias.to(DEVICE),
                     norm_weight=norm_weight.to(DEVICE), eps=1e-5, unit_eps=1e-6, view=view, write=True, **sizes)
    got, fed = [[], []], [0, 0]
    for step in steps:
        wide = torch.zeros(sum(step), width + 8, dtype=dtype, device=DEVICE)
        rows = wide[:, offset:offset + width]
        rows.copy_(torch.cat([projected[r][fed[r]:fed[r] + step[r]] for r in (0, 1)]))
        ctx = context(list(step), list(fed))
        ctx.leading_single = 2 if max(step) == 1 else 0
        out = ops.gated_delta_rule(rows, ctx=ctx, **constants)
        got[0].append(out[:step[0]].cpu())
        got[1].append(out[step[0]:].cpu())
        fed = [fed[r] + step[r] for r in (0, 1)]
    ops.check_errors()
    for r in (0, 1):
        want = delta_pieces(projected[r].double(), conv.double(), a_log.double(), dt_bias.double(),
                            norm_weight.double(), 1e-5, sizes)
        # (the bounds of the test above)
        assert (torch.cat(got[r]).double() - want).abs().max() < bound(dtype, 5e-5, 0.1), f"request {r}"
