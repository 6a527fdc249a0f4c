"""Latent attention of prompts with expanded keys and values, against the fp32 restatement."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,lens", [
    (128, [65]), (2, [128, 1, 129]), (3, [256, 257, 383]), (8, [700, 90]),      # ends on and off tiles, one and two blocks of queries
])
def test_expanded_prompts(H, lens):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(H)
    T, nope, R, V, L = sum(lens), 128, 64, 128, 512
    q, rows = torch.randn(T, H * (nope + R)).bfloat16(), torch.randn(T, L + R).bfloat16()
    w = (torch.randn(H * (nope + V), L) * 0.05).bfloat16()
    cs, pos = ref.build_cos_sin(800, R, 1e4), torch.cat([torch.arange(n) for n in lens]).int()
    cu_q = torch.tensor([0] + lens).cumsum(0).int()
    a, b = q.clone(), q.cuda()
    want = ref.mla_prefill(a, rows, w, cs, pos, cu_q, H, nope, V, L, 192 ** -0.5, max(lens))
    got = cu.mla_prefill(b, rows.cuda(), w.cuda(), cs.cuda(), pos.cuda(), cu_q.cuda(), H, nope, V, L, 192 ** -0.5, max(lens)).cpu()
    cu.check_status(torch.device("cuda", 0))
    assert float((b.cpu().float() - a.float()).norm() / a.float().norm()) < 2 ** -8      # rotated in place
    # probabilities, expanded values and outputs are rounded to bf16 (2^-9 each)
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2 ** -7


@pytest.mark.parametrize("lens", [[65, 63], [1, 300], [129, 1, 127], [255, 2], [383, 200]])     # last tiles of either block of queries
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_prompts_do_not_see_the_next_one(lens, bad):
    """Keys and values of the next prompt of the batch that are no numbers change no bit of the prompts before it."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(sum(lens))
    H, T, nope, R, V, L = 3, sum(lens), 128, 64, 128, 512
    q, rows = torch.randn(T, H * (nope + R)).bfloat16().cuda(), torch.randn(T, L + R).bfloat16().cuda()
    w = (torch.randn(H * (nope + V), L) * 0.05).bfloat16().cuda()
    cs, pos = ref.build_cos_sin(800, R, 1e4).cuda(), torch.cat([torch.arange(n) for n in lens]).int().cuda()
    cu_q = torch.tensor([0] + lens).cumsum(0).int().cuda()
    out = []
    for value in (0.0, bad):
        other = rows.clone()
        other[lens[0]:] = value
        out.append(cu.mla_prefill(q.clone(), other, w, cs, pos, cu_q, H, nope, V, L, 192 ** -0.5, max(lens))[:lens[0]])
    cu.check_status(torch.device("cuda", 0))
    assert bool(torch.isfinite(out[0].float()).all())
    assert torch.equal(*out)


def test_engine_expands_fresh_prompts(monkeypatch):
    """367 rows of fresh prompts through the engine, expanded and absorbed, against the absorbed form in fp32 on the CPU. Dense
    layers: a routed choice near a tie would fall differently between two roundings."""
    from parallax_b200 import ops
    from parallax_b200.engine.engine import Engine
    from parallax_b200.engine.request import Request, SamplingParams
    from parallax_b200.models.config import named_config
    from parallax_b200.models.deepseek import DeepseekStage
    from parallax_b200.ops import cuda as cu

    cfg = named_config("small-mla")
    cfg.first_k_dense_replace = cfg.num_hidden_layers
    g = torch.Generator().manual_seed(6)
    prompts = [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in (150, 97, 120)]
    calls, plain = [], ops.mla_prefill
    monkeypatch.setattr(ops, "mla_prefill", lambda *a, **kw: (calls.append(a[0].shape[0]), plain(*a, **kw))[1])

    def logits(device, like=None):
        eng = Engine(cfg, device=device, dtype=torch.float32 if like else torch.bfloat16, num_blocks=64, page_size=16, max_batch_size=4,
                     max_num_tokens_per_batch=512, max_total_length=256, seed=0)
        stage = eng.stages[0].model
        if like:        # the GPU stage's weights, and no expanded form
            for a, b in [(like, stage)] + list(zip(like.layers, stage.layers)):
                for name in ("embed", "norm_w", "lm_head") if a is like else type(a).__slots__:
                    t = getattr(a, name)
                    if isinstance(t, torch.Tensor):
                        setattr(b, name, None if name == "w_kvb" else t.detach().cpu().float())
        eng.keep_logits = True
        for p in prompts:
            eng.add_request(Request(input_ids=p, sampling_params=SamplingParams(max_new_tokens=2, temperature=0.0, ignore_eos=True),
                                    max_total_length=256))
        eng.step()
        return eng.last_logits.float().cpu(), stage

    expanded, stage = logits("cuda:0")
    assert calls == [sum(len(p) for p in prompts)] * cfg.num_hidden_layers
    with monkeypatch.context() as m:
        m.setattr(DeepseekStage, "_expands", lambda *a: False)
        absorbed, _ = logits("cuda:0")
    assert len(calls) == cfg.num_hidden_layers
    want, _ = logits("cpu", stage)
    cu.check_status(torch.device("cuda", 0))
    for got in (expanded, absorbed):        # bf16 activations through three layers: some ten roundings of 2^-9 on the way
        assert float((got - want).norm() / want.norm()) < 2 ** -5
    assert float((expanded - absorbed).norm() / want.norm()) < 2 ** -5
