"""Decode steps with programmatic dependent launches (a kernel may start, and fetch its
weights, while its predecessor finishes) give the same logits as without."""

import pytest
import torch

from tiny_models import CONFIGS, make_model_dir, prompts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["A", "C"])
def test_same_logits_with_dependent_launches(tmp_path, name):
    from mlx_one_b200.cache import CacheManager
    from mlx_one_b200.engine.loading import load_model
    from mlx_one_b200.engine.runner import Runner, StepEntry

    config, _, page = CONFIGS[name]
    loaded = load_model(make_model_dir(name, tmp_path), torch.bfloat16, "cuda:0")
    ops = loaded.model.ops
    requests = prompts(config["vocab_size"], (40, 15, 77), seed=9)
    results = []
    try:
        for enabled in (False, True):
            ops.set_dependent_launches(enabled)
            cache = CacheManager(loaded.model.cache_needs, page_size=page, capacity_tokens=512,
                                 max_requests=4, dtype=torch.bfloat16, device="cuda:0")
            runner = Runner(loaded.model, cache)
            for i in range(len(requests)):
                cache.open(i)
            runner.step([StepEntry(i, tokens[:-12]) for i, tokens in enumerate(requests)])
            collected = []
            for step in range(12):       # eager first, then captured as a graph and replayed
                entries = [StepEntry(i, [tokens[len(tokens) - 12 + step]], (0,))
                           for i, tokens in enumerate(requests)]
                collected.append(runner.step(entries).float().cpu().clone())
            ops.check_errors()
            assert runner.graph_replays >= 10
            results.append(torch.stack(collected))
    finally:
        ops.set_dependent_launches(True)
    assert torch.equal(results[0], results[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", ["B", "D", "G1", "G2", "G3", "G5"])
def test_same_logits_in_32_bit_and_with_the_delta_rule(tmp_path, name, dtype):
    """The 32-bit engine's kernels and the delta rule's: portions, single tokens beside a portion, single
    tokens step by step and in a loop without the host."""
    import galarax_models
    from mlx_one_b200.cache import CacheManager
    from mlx_one_b200.engine.loading import load_model
    from mlx_one_b200.engine.runner import Runner, StepEntry

    if name in CONFIGS:
        vocab, folder = CONFIGS[name][0]["vocab_size"], make_model_dir(name, tmp_path, dtype=dtype)
    else:
        vocab, folder = galarax_models.CONFIGS[name][0]["vocab"], galarax_models.make_model_dir(name, tmp_path)
    loaded = load_model(folder, dtype, "cuda:0")
    ops = loaded.model.ops
    requests = prompts(vocab, (90, 15, 77), seed=9)
    late = prompts(vocab, (70,), seed=10)[0]
    results = []
    try:
        for enabled in (False, True):
            ops.set_dependent_launches(enabled)
            cache = CacheManager(loaded.model.cache_needs, page_size=8, capacity_tokens=1024, max_requests=4,
                                 dtype=dtype, device="cuda:0")
            runner = Runner(loaded.model, cache)
            for i in range(4):
                cache.open(i)
            collected = []

            def step(entries):
                collected.append(runner.step(entries).float().cpu().clone())

            step([StepEntry(i, tokens[:-8], (0,)) for i, tokens in enumerate(requests)])
            for at in range(-8, 0):
                step([StepEntry(i, [tokens[at]], (0,)) for i, tokens in enumerate(requests)] +
                     ([StepEntry(3, late, (69,))] if at == -4 else []))
            chosen = runner.decode_steps([StepEntry(i, [5], (0,)) for i in range(4)], 40)
            collected.append(chosen.float().cpu())
            step([StepEntry(i, [6], (0,)) for i in range(4)])
            ops.check_errors()
            results.append(collected)
    finally:
        ops.set_dependent_launches(True)
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(32, 8, 64), (16, 8, 64), (8, 2, 128)])
def test_decode_attention_reads_its_row_behind_the_wait(heads, kv_heads, head_dim):
    """A projection and the decode attention that starts from its row, two inputs in turn through one buffer:
    a query, key or value asked for ahead of the wait would be the other input's."""
    from mlx_one_b200.kernels.cuda_ops import CudaOps
    from mlx_one_b200.parts.base import PagedKeyValues, PagedView
    from test_gpu_kernels import make_batch

    ops, hidden = CudaOps("cuda:0", verbose=False), 4096
    generator = torch.Generator("cuda:0").manual_seed(head_dim)
    normal = lambda *shape: torch.randn(shape, generator=generator, device="cuda:0").bfloat16()
    w, inputs = normal((heads + 2 * kv_heads) * head_dim, hidden) / 64, [normal(4, hidden) for _ in range(2)]
    ctx, table, pages = make_batch([1] * 4, [0, 31, 70, 700], 16, "cuda:0")
    kv = normal(2, pages, kv_heads, 16, head_dim)
    need = PagedKeyValues(kv_heads, head_dim, None)
    results = []
    try:
        for enabled in (False, True):
            ops.set_dependent_launches(enabled)
            for i in range(400):
                qkv = ops.linear(inputs[i % 2], w)
                got = ops.qkv_attention(qkv, q_weight=None, k_weight=None, rotary=None, ctx=ctx, eps=None,
                                        view=PagedView(kv, table, 16, need), heads=heads, kv_heads=kv_heads,
                                        head_dim=head_dim, scale=0.125, window=None, write=True)
                del qkv
                results.append(got)
    finally:
        ops.set_dependent_launches(True)
    ops.check_errors()
    assert not torch.equal(results[0], results[1])
    assert all(torch.equal(got, results[i % 2]) for i, got in enumerate(results))
