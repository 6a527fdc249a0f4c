"""One or two rows through a dense stage: which heads go together with their rotation, and that both ways leave the same cache."""

import numpy as np
import pytest
import torch

from parallax_b200.engine.batch import BatchBuilder
from parallax_b200.engine.worker import StageWorker
from parallax_b200.models.config import config_from_hf

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def test_a_wave_of_clusters():
    from parallax_b200.ops import _lib

    pays, sms = _lib.lib().pxl_gemv_bf16_qkv_pays, torch.cuda.get_device_properties(0).multi_processor_count
    for Hq, Hkv in ((1, 1), (8, 2), (16, 2), (16, 8), (24, 4), (28, 4), (32, 4), (32, 8), (64, 8)):
        ctas = 8 * (Hq + 2 * Hkv)
        assert bool(pays(2, Hq, Hkv)) == (ctas <= 7 * sms // 4)
        assert bool(pays(1, Hq, Hkv)) == (sms <= ctas <= 7 * sms // 4)


@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize("Hq,Hkv", [(4, 2), (16, 8), (32, 4)])
def test_rows(rows, Hq, Hkv):
    cfg = config_from_hf(dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=1024, num_hidden_layers=4,
                              num_attention_heads=Hq, num_key_value_heads=Hkv, head_dim=128, intermediate_size=2048, vocab_size=512,
                              rope_theta=1e4, max_position_embeddings=512))
    w = StageWorker(cfg, 1, 3, DEV, torch.bfloat16, 16, num_blocks=16, seed=3, max_positions=300)
    ctx = np.asarray([37, 100][:rows], dtype=np.int32)
    table = np.arange(16, dtype=np.int32).reshape(2, 8)[:rows]
    slots = np.asarray([table[i, (c - 1) // 16] * 16 + (c - 1) % 16 for i, c in enumerate(ctx)], dtype=np.int64)

    def batch(n):       # the rows, and copies of the last one that write no cache, so that other kernels take the batch
        c = np.concatenate([ctx, np.repeat(ctx[-1:], n - rows)])
        t = np.concatenate([table, np.repeat(table[-1:], n - rows, axis=0)])
        s = np.concatenate([slots, np.full(n - rows, -1)])
        return BatchBuilder(DEV, 8, 8, 16).build(None, c - 1, s, [], [], None, c, t, np.arange(n, dtype=np.int32))

    g = torch.Generator(device=DEV).manual_seed(1)
    h = torch.randn(rows, 1024, device=DEV, dtype=torch.bfloat16, generator=g)
    kept = [[torch.randn(t.shape, device=DEV, generator=g).to(t.dtype) for t in (c.k, c.v)] for c in w.pool.layers]
    out = []
    for n in (rows, 6):
        for c, old in zip(w.pool.layers, kept):
            c.k.copy_(old[0]), c.v.copy_(old[1])
        y = w.run(batch(n), torch.cat([h, h[-1:].repeat(n - rows, 1)]))[:rows].clone()
        out.append([y] + [t.clone() for c in w.pool.layers for t in (c.k, c.v)])
    for a, b in zip(*out):      # bf16 roundings of another order of sums in each of two layers
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2 ** -6
