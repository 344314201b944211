"""The 32-bit engine's products and attention at the edges of their tiles, sections of K and units of
keys, against 64 bits; and that a row's or a query's result is the same bits in every kernel."""

import pytest
import torch

from test_gpu_kernels import make_batch, on_cpu, ops, plain  # noqa: F401  (fixtures)
from tiny_models import CONFIGS, make_model_dir, prompts
from mlx_one_b200.parts.base import PagedKeyValues, PagedView

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("n,k", [(1, 8), (5, 7), (37, 520), (64, 512), (100, 1032), (50, 4608),
                                 (33, 30), (2500, 136), (9500, 72)])
def test_products_of_any_number_of_rows(ops, n, k):
    """1 to 16 rows (the streaming kernel where K is a multiple of 8), then tiles of 32, 64 and 128
    rows; rows that are a slice of wider ones, aligned or not."""
    generator = torch.Generator(DEVICE).manual_seed(n * 10000 + k)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    w, bias = normal(n, k), normal(n)
    wide = normal(130, k + 9)
    want = wide[:, 1:k + 1].double() @ w.double().T + bias.double()
    # every value passes one chain of at most 32 FMAs and k / 256 + 10 additions
    bound = (32 + k / 256 + 10) * 2.0 ** -24 * (wide[:, 1:k + 1].abs().double() @ w.abs().double().T +
                                                bias.abs().double())
    first = None
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 130):
        for a in (wide[:m, 1:k + 1], wide[:m, 1:k + 1].contiguous()):
            got = ops.linear(a, w, bias)
            assert ((got.double() - want[:m]).abs() <= bound[:m]).all(), (m, a.stride())
            first = got[0] if first is None else first
            assert torch.equal(got[0], first), (m, a.stride())


@pytest.mark.parametrize("n,k", [(2500, 4608), (2501, 2056), (5000, 1032), (9500, 520)])
def test_products_walk_groups_and_sections(ops, n, k):
    """Weights streamed by warps that take several groups of rows and several sections of K each, with the
    rows of the input brought in one or several parts: every row has the bits that the tiles give it."""
    generator = torch.Generator(DEVICE).manual_seed(n + k)
    normal = lambda *shape: torch.randn(shape, generator=generator, device=DEVICE)
    a, w, bias = normal(130, k), normal(n, k), normal(n)
    tiles = ops.linear(a, w, bias)
    want = a.double() @ w.double().T + bias.double()
    bound = (32 + k / 256 + 10) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double())
    assert ((tiles.double() - want).abs() <= bound).all()
    for m in (1, 2, 3, 4, 7, 8, 9, 17, 32, 33, 64):
        assert torch.equal(ops.linear(a[:m], w, bias), tiles[:m]), m
    # weights that are aligned to 16 bytes only: tiles at every number of rows
    shifted = torch.empty(n * k + 4, device=DEVICE)[4:].view(n, k).copy_(w)
    for m in (1, 8, 17):
        assert torch.equal(ops.linear(a[:m], shifted, bias), tiles[:m]), m


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size", [
    (16, 8, 64, 16), (24, 8, 64, 16), (4, 4, 32, 4), (12, 1, 128, 32), (32, 1, 64, 64)])
@pytest.mark.parametrize("portions,histories", [
    ([1, 1, 1, 1, 1], [0, 62, 63, 64, 700]), ([1, 1, 70, 2, 9], [5, 300, 0, 64, 127]),
    ([400], [0]), ([1] * 40, list(range(40, 80))), ([700, 1, 900], [0, 3, 130])])
def test_attention_whole_and_in_units(ops, plain, heads, kv_heads, head_dim, page_size, portions,
                                      histories):
    """Against the plain function; then the same with the units of every token cut apart and with
    none cut: the same bits. An infinite value that only later tokens see leaves earlier ones alone."""
    ctx, table, pages = make_batch(portions, histories, page_size, DEVICE, seed=heads)
    ctx.leading_single = next((i for i, n in enumerate(portions) if n > 1), len(portions))
    generator = torch.Generator().manual_seed(head_dim)
    kv = torch.randn(2, pages, kv_heads, page_size, head_dim, generator=generator)
    q = torch.randn(ctx.tokens, heads, head_dim, generator=generator)
    need = PagedKeyValues(kv_heads, head_dim, None)
    view = PagedView(kv.to(DEVICE), table, page_size, need)
    arguments = dict(heads=heads, kv_heads=kv_heads, head_dim=head_dim, scale=head_dim ** -0.5,
                     window=None)
    want = plain.paged_attention(q, ctx=on_cpu(ctx), view=PagedView(kv, table.cpu(), page_size, need),
                                 **arguments)
    got = ops.paged_attention(q.to(DEVICE), ctx=ctx, view=view, **arguments)
    torch.testing.assert_close(got.cpu(), want, atol=2e-5, rtol=2e-5)
    count, some = ops._sm_count, []
    try:
        for ops._sm_count in (0, 1 << 30):
            some.append(ops.paged_attention(q.to(DEVICE), ctx=ctx, view=view, **arguments))
    finally:
        ops._sm_count = count
    assert torch.equal(some[0], some[1]) and torch.equal(some[0], got)
    ctx.leading_single = 0
    assert torch.equal(ops.paged_attention(q.to(DEVICE), ctx=ctx, view=view, **arguments), got)
    last = max(range(len(portions)), key=lambda r: portions[r])
    if portions[last] > 1:
        at = histories[last] + portions[last] - 1
        view.kv[1, int(table[last, at // page_size]), :, at % page_size] = float("inf")
        spoilt = ops.paged_attention(q.to(DEVICE), ctx=ctx, view=view, **arguments)
        end = int(ctx.request_start[last + 1]) - 1
        assert torch.isinf(spoilt[end]).all()
        assert torch.equal(torch.cat((spoilt[:end], spoilt[end + 1:])), torch.cat((got[:end], got[end + 1:])))
    ops.check_errors()


@pytest.mark.parametrize("name", ["B", "C"])      # heads of 32 and of 48 (the general kernel's)
def test_decode_loops_with_and_without_graphs(tmp_path, name):
    """Loops of decode steps whose positions pass several borders of units of 64 keys: the same tokens,
    and behind them the same logits to the bit, whether the steps are replayed or launched one by one."""
    from mlx_one_b200.cache import CacheManager
    from mlx_one_b200.engine.loading import load_model
    from mlx_one_b200.engine.runner import Runner, StepEntry

    config, _, page = CONFIGS[name]
    loaded = load_model(make_model_dir(name, tmp_path, dtype=torch.float32), "float32", DEVICE)
    results = []
    for graphs in (True, False):
        cache = CacheManager(loaded.model.cache_needs, page_size=page, capacity_tokens=1024, max_requests=2,
                             dtype=torch.float32, device=DEVICE)
        runner = Runner(loaded.model, cache)
        runner.use_graphs = graphs
        last = []
        for i, tokens in enumerate(prompts(config["vocab_size"], (100, 59), seed=21)):
            cache.open(i)
            last.append(int(runner.step([StepEntry(i, tokens, (len(tokens) - 1,))]).argmax()))
        chosen = runner.decode_steps([StepEntry(i, [t]) for i, t in enumerate(last)], 170)
        logits = runner.step([StepEntry(i, [t], (0,)) for i, t in enumerate(chosen[-1].tolist())])
        loaded.model.ops.check_errors()
        assert (runner.graph_replays > 160) == graphs
        results.append((chosen.cpu(), logits.cpu().clone()))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("portions", [[1, 1], [1, 9]])
def test_positions_behind_the_table(ops, portions):
    """A host bound that the device's positions have outgrown changes nothing; a position behind the
    block table raises the error flag, with the units of a token cut apart and with none cut."""
    page, heads, kv_heads, dim = 16, 4, 2, 32
    ctx, table, pages = make_batch(portions, [700, 63], page, DEVICE)
    ctx.leading_single = 1 if portions[1] > 1 else 2
    generator = torch.Generator(DEVICE).manual_seed(1)
    kv = torch.randn(2, pages, kv_heads, page, dim, generator=generator, device=DEVICE)
    q = torch.randn(ctx.tokens, heads, dim, generator=generator, device=DEVICE)
    count, need = ops._sm_count, PagedKeyValues(kv_heads, dim, None)

    def attend(table):
        return ops.paged_attention(q, heads=heads, kv_heads=kv_heads, head_dim=dim, scale=0.2, window=None,
                                   ctx=ctx, view=PagedView(kv, table, page, need))

    try:
        for ops._sm_count in (0, 1 << 30):
            want, ctx.max_context = attend(table), 65
            assert torch.equal(attend(table), want)
            ops.check_errors()
            attend(table[:, :40].contiguous())          # 640 keys, position 700
            with pytest.raises(RuntimeError):
                ops.check_errors()
    finally:
        ops._sm_count = count


@pytest.mark.parametrize("portions,histories,spoilt", [([1], [128], range(128, 129)), ([1, 1], [200, 70], range(128, 192)),
                                                       ([40], [100], range(128, 129)), ([70], [128], range(64, 128))])
def test_scores_that_are_nan(ops, portions, histories, spoilt):
    """Keys that are NaN, all of a unit of 64 or all that a query sees of it: every query that sees one is NaN,
    the others keep their bits."""
    page, heads, kv_heads, dim = 16, 4, 2, 32
    ctx, table, pages = make_batch(portions, histories, page, DEVICE)
    generator = torch.Generator(DEVICE).manual_seed(7)
    kv = torch.randn(2, pages, kv_heads, page, dim, generator=generator, device=DEVICE)
    q = torch.randn(ctx.tokens, heads, dim, generator=generator, device=DEVICE)
    view = PagedView(kv, table, page, PagedKeyValues(kv_heads, dim, None))
    attend = lambda: ops.paged_attention(q, heads=heads, kv_heads=kv_heads, head_dim=dim, scale=0.2, window=None,
                                         ctx=ctx, view=view)
    count = ops._sm_count
    try:
        for ops._sm_count in (0, 1 << 30):
            view.kv = kv.clone()
            want = attend()
            for at in spoilt:
                view.kv[0, int(table[0, at // page]), :, at % page] = float("nan")
            got = attend()
            sees = (ctx.token_request == 0) & (ctx.positions >= spoilt[0])
            assert torch.isnan(got[sees]).all() and torch.equal(got[~sees], want[~sees])
    finally:
        ops._sm_count = count
    ops.check_errors()


def test_scratch_of_units_side_by_side(ops):
    """Tokens whose units would not fit the scratch together go one part after the other: the same bits,
    and no more memory than stated, down to one tile of tokens at a time."""
    heads, kv_heads, dim, page = 16, 4, 64, 16
    ctx, table, pages = make_batch([1, 1, 1, 150], [3000, 5, 64, 2900], page, DEVICE)
    ctx.leading_single = 3
    generator = torch.Generator(DEVICE).manual_seed(2)
    kv = torch.randn(2, pages, kv_heads, page, dim, generator=generator, device=DEVICE)
    q = torch.randn(ctx.tokens, heads, dim, generator=generator, device=DEVICE)
    view = PagedView(kv, table, page, PagedKeyValues(kv_heads, dim, None))
    kept, results = ops.split_scratch, []
    tile = 32 // (heads // kv_heads) * heads * -(-table.shape[1] * page // 64) * (dim + 4)
    try:
        for ops.split_scratch in (kept, 3 * tile + 5, 1):
            torch.cuda.reset_peak_memory_stats()
            base, before = torch.cuda.memory_allocated(), ops.launches
            results.append(ops.paged_attention(q, heads=heads, kv_heads=kv_heads, head_dim=dim, scale=0.1,
                                               window=None, ctx=ctx, view=view))
            peak = torch.cuda.max_memory_allocated() - base - 4 * q.numel()
            # (the allocator hands out blocks whole that are up to 1 MB larger)
            assert peak <= 4 * max(tile, ops.split_scratch) + (1 << 20)
            # singles and portion, each with its merge; tiles of 8 tokens, three or one at a time
            assert ops.launches - before == {kept: 4, 1: 2 * 3 + 2 * 19}.get(ops.split_scratch, 2 + 2 * 7)
    finally:
        ops.split_scratch = kept
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])
    ops.check_errors()
