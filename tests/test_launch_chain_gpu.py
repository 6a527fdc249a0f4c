"""Layers launched as a chain (each kernel's prologue and first weights under the tail of the kernel before) against the same
layers launched one after the other: the same bits, step after step."""

from contextlib import nullcontext

import numpy as np
import pytest
import torch

from parallax_b200.engine.batch import BatchBuilder
from parallax_b200.engine.worker import StageWorker
from parallax_b200.models.config import config_from_hf, named_config

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
PAGE = 16


def _config(name):
    if name == "hybrid":
        return config_from_hf(dict(
            architectures=["Qwen3NextForCausalLM"], model_type="qwen3_next", hidden_size=1024, num_hidden_layers=12,
            num_attention_heads=8, num_key_value_heads=2, head_dim=128, intermediate_size=2048, vocab_size=512, rope_theta=1e4,
            partial_rotary_factor=0.25, full_attention_interval=4, max_position_embeddings=4096, linear_num_key_heads=4,
            linear_num_value_heads=8, linear_key_head_dim=128, linear_value_head_dim=128, linear_conv_kernel_dim=4))
    return named_config(name)


@pytest.mark.parametrize("name,start,layers,kv", [("qwen3-30b-a3b", 8, 2, "bf16"), ("deepseek-v3", 1, 2, "bf16"),
                                                  ("deepseek-v3.2", 1, 2, "bf16"), ("hybrid", 4, 4, "bf16"),
                                                  ("qwen3-8b", 8, 2, "fp8_e4m3")])
def test_chained_layers_give_the_same_bits(name, start, layers, kv):
    from parallax_b200.ops import cuda as cu

    cfg = _config(name)
    prompts, decode = [(70, 70), (33, 50)], [300, 2300, 17, 1]         # (new tokens, context); contexts of decoding rows
    seqs = prompts + [(1, c) for c in decode]
    blocks = sum(-(-t // PAGE) for _n, t in seqs)
    table = np.zeros((len(seqs), -(-2300 // PAGE)), dtype=np.int32)
    order, at = np.random.RandomState(3).permutation(blocks).astype(np.int32), 0
    for i, (_n, t) in enumerate(seqs):
        n = -(-t // PAGE)
        table[i, :n] = order[at:at + n]
        at += n
    pos = np.concatenate([np.arange(t - n, t, dtype=np.int32) for n, t in seqs])
    row = np.repeat(np.arange(len(seqs)), [n for n, _t in seqs])
    slots = table[row, pos // PAGE].astype(np.int64) * PAGE + pos % PAGE
    last = np.cumsum([n for n, _t in seqs]).astype(np.int32) - 1
    worker = StageWorker(cfg, start, start + layers, DEV, torch.bfloat16, PAGE, num_blocks=blocks, seed=1, max_positions=2400,
                         num_linear_slots=len(seqs), kv_cache_dtype=kv)
    fb = BatchBuilder(DEV, len(pos), len(seqs), 2 * table.shape[1]).build(
        None, pos, slots, [n for n, _t in prompts], [t for _n, t in prompts], table[:2, :5], np.asarray(decode, dtype=np.int32),
        table[2:], last, np.arange(len(seqs), dtype=np.int32))
    g = torch.Generator(device=DEV).manual_seed(5)
    hidden = torch.randn(len(pos), cfg.hidden_size, device=DEV, dtype=torch.bfloat16, generator=g)
    caches = [[t for t in (c.k, c.v, c.index_k, c.conv_state, c.rec_state) if t is not None] for c in worker.pool.layers]
    for layer in caches:
        for t in layer:
            t.copy_((torch.randn(t.shape, device=DEV, generator=g) * 0.5).to(t.dtype))
    kept = [[t.clone() for t in layer] for layer in caches]

    def step():
        for layer, old in zip(caches, kept):
            for t, o in zip(layer, old):
                t.copy_(o)
        return worker.run(fb, hidden)

    worker.model.chained = lambda h: nullcontext()
    want = step()
    after = [[t.clone() for t in layer] for layer in caches]
    del worker.model.chained
    for _ in range(4):
        y = step()
        if cfg.index_topk:      # lists of chosen keys come in any order, and sums over them in the order of the list: bf16 roundings
            assert float((y.float() - want.float()).norm() / want.float().norm()) < 1e-2
            continue
        assert torch.equal(y, want)
        for layer, old in zip(caches, after):
            for t, o in zip(layer, old):
                assert torch.equal(t.view(torch.uint8), o.view(torch.uint8))
    cu.check_status(DEV)


@pytest.mark.parametrize("M", [1, 3, 33, 64, 97, 128, 200])
def test_weights_written_just_before_a_chain(M):
    """The first kernel of a chain follows what the caller had on the stream, also where it loads weights ahead of its wait."""
    from parallax_b200.ops import cuda as cu

    g = torch.Generator(device=DEV).manual_seed(M)
    x = torch.randn(M, 2048, device=DEV, dtype=torch.bfloat16, generator=g)
    ws = [torch.randn(4096, 2048, device=DEV, dtype=torch.bfloat16, generator=g) for _ in range(3)]
    want = [cu.linear(x, w) for w in ws]
    live = torch.zeros_like(ws[0])
    for w, y in zip(ws, want):
        live.copy_(w)
        with cu.launch_chain():
            assert torch.equal(cu.linear(x, live), y)
    cu.check_status(DEV)
