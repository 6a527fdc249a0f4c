"""Chunked and stepped gated delta rule and the convolution in runs of tokens, against the fp32 restatement at the sizes where
tiles end."""

import pytest
import torch

from parallax_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / (b.norm() + 1e-30))


def _batch(lens, starts):
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).int()
    slots = torch.randperm(len(lens) + 2)[:len(lens)].int()
    pos = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, lens)]).int()
    return cu, slots, pos


# lens, starts, prompt slices among them (they come first), Hk, Hv, Dv, A (log), padding of the rows
CASES = [
    ([1], [0], 1, 1, 1, 32, 0.0, 0),
    ([63, 1], [0, 9], 1, 2, 2, 64, 1.0, 0),
    ([64, 65, 1, 1], [0, 7, 3, 0], 2, 1, 2, 128, 2.0, 0),
    ([16, 17, 200], [5, 0, 64], 3, 2, 4, 96, -3.0, 0),       # long memories
    ([129], [0], 1, 1, 2, 128, 6.0, 0),                      # states that vanish within a token
    ([80, 2], [1, 1], 1, 1, 2, 128, 0.0, 3),                 # rows that do not start on 16 bytes: token by token
    ([70, 1], [0, 4], 1, 1, 1, 40, 0.0, 0),                  # columns that no slice divides: token by token
    ([1, 1, 1], [4, 0, 8], 0, 2, 4, 128, 0.0, 0),
]


@pytest.mark.parametrize("lens,starts,prompts,Hk,Hv,Dv,log_a,pad", CASES)
def test_gated_delta_rule(lens, starts, prompts, Hk, Hv, Dv, log_a, pad):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(len(lens) * 100 + Dv)
    T, Dk = sum(lens), 128
    seq_cu, slots, pos = _batch(lens, starts)
    C = 2 * Hk * Dk + Hv * Dv
    rows = (torch.randn(T, C + pad) * 0.7).bfloat16()
    z, ab = torch.randn(T, Hv * Dv).bfloat16(), torch.randn(T, 2 * Hv).bfloat16()
    A, dt = torch.full((Hv,), float(log_a)), torch.linspace(-1, 1, Hv)
    w = (torch.rand(Dv) + 0.5).bfloat16()
    state = torch.randn(len(lens) + 2, Hv, Dv, Dk) * 0.1

    def run(mod, to, **kw):
        st = to(state.clone())
        a = to(ab)
        out = mod.gated_delta_rule(to(rows)[:, :C], a[:, :Hv], a[:, Hv:], to(A), to(dt), to(z), to(w), st, to(seq_cu), to(slots),
                                   to(pos), Hk, Hv, Dk, Dv, 1e-6, **kw)
        return out, st

    want, want_state = run(ref, lambda x: x)
    got, got_state = run(cu, lambda x: x.cuda(), prefill_seqs=prompts, prefill_tokens=sum(lens[:prompts]))
    torch.cuda.synchronize()
    # outputs: one rounding to bf16 on either side (2^-9 each); state: fp32 with operands of 17 bits in the chunked form
    assert _rel(got, want) < 2 ** -7, _rel(got, want)
    assert _rel(got_state, want_state) < 1e-4, _rel(got_state, want_state)
    untouched = [s for s in range(state.shape[0]) if s not in slots.tolist()]
    assert torch.equal(got_state.cpu()[untouched], state[untouched])


def test_gated_delta_rule_in_several_runs():
    """Chunks that do not fit the workspace at once: the state goes through memory between the runs."""
    from parallax_b200.ops import cuda as cu

    lib = cu._lib.lib()
    torch.manual_seed(3)
    lens, Hk, Hv, Dk, Dv = [150, 100], 1, 2, 128, 64
    T, C = sum(lens), 2 * 128 + 2 * 64
    seq_cu, slots, pos = (t.cuda() for t in _batch(lens, [0, 5]))
    rows, z, ab = (torch.randn(T, n).bfloat16().cuda() for n in (C, Hv * Dv, 2 * Hv))
    A, dt, w = torch.zeros(Hv).cuda(), torch.zeros(Hv).cuda(), torch.ones(Dv).bfloat16().cuda()
    state = (torch.randn(4, Hv, Dv, Dk) * 0.1).cuda()
    got = []
    full = lib.pxl_gated_delta_workspace(Hv, Dv, 2, T)
    for nbytes in (full, full // 5 * 2):        # five chunks at most: all at once, or two at a time
        st, out = state.clone(), torch.empty(T, Hv * Dv, dtype=torch.bfloat16, device="cuda")
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        code = lib.pxl_gated_delta_rule(rows.data_ptr(), C, ab.data_ptr(), ab[:, Hv:].data_ptr(), 2 * Hv, A.data_ptr(), dt.data_ptr(),
                                        z.data_ptr(), Hv * Dv, w.data_ptr(), st.data_ptr(), seq_cu.data_ptr(),
                                        slots.data_ptr(), pos.data_ptr(), out.data_ptr(), Hv * Dv, 2, Hk, Hv, Dk, Dv, 1e-6,
                                        2, T, ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
        assert code == 0
        torch.cuda.synchronize()
        got.append((out, st))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("K", [2, 3, 4, 5])
@pytest.mark.parametrize("C,bias", [(8, False), (1032, True), (20, True)])
def test_convolution_in_runs(K, C, bias):
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(K * C)
    lens, starts, prompts = [1, 2, 70, 3, 1], [4, 0, 9, 1, 2], 4
    T = sum(lens)
    seq_cu, slots, pos = _batch(lens, starts)
    x = torch.randn(T, C + 8).bfloat16()
    w, b = (torch.randn(C, K) * 0.3).bfloat16(), torch.randn(C).bfloat16() if bias else None
    state = torch.randn(len(lens) + 2, C, K - 1).bfloat16()
    s0, s1 = state.clone(), state.cuda()
    want = ref.causal_conv1d_silu(x[:, :C], w, b, s0, seq_cu, slots, pos)
    got = cu.causal_conv1d_silu(x.cuda()[:, :C], w.cuda(), None if b is None else b.cuda(), s1, seq_cu.cuda(), slots.cuda(), pos.cuda(),
                                prefill_seqs=prompts, prefill_tokens=sum(lens[:prompts]))
    assert torch.equal(s1.cpu(), s0)                    # inputs are copied as they are
    assert _rel(got, want) < 2 ** -7                    # one rounding to bf16 on either side


@pytest.mark.parametrize("log_a", [-6.0, -2.0, 0.0])
def test_kept_state_over_slices(log_a):
    """The state behind several slices of a prompt stays as close to 64 bits in chunks as token by token: both hold fp32 numbers
    and add fp32 products, in another order (a factor of two), and the chunks' factors take a few more roundings of 2^-24."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(int(-log_a))
    Hk, Hv, D, T = 1, 2, 128, 150
    A, dt, w = torch.full((Hv,), log_a).cuda(), torch.linspace(-2, 1, Hv).cuda(), torch.ones(D).bfloat16().cuda()
    cu_t, slot = torch.tensor([0, T]).int().cuda(), torch.zeros(1).int().cuda()
    want = torch.zeros(Hv, D, D, dtype=torch.float64, device="cuda")
    states = [torch.zeros(1, Hv, D, D, device="cuda") for _ in range(2)]
    for s in range(4):
        rows, z, ab = (torch.randn(T, n).bfloat16().cuda() for n in (2 * Hk * D + Hv * D, Hv * D, 2 * Hv))
        for st, prompts in zip(states, (1, 0)):
            cu.gated_delta_rule(rows, ab[:, :Hv], ab[:, Hv:], A, dt, z, w, st, cu_t, slot, (torch.arange(T) + s * T).int().cuda(), Hk, Hv,
                                D, D, 1e-6, prefill_seqs=prompts, prefill_tokens=T * prompts)
        k, v = rows[:, D:2 * D].double(), rows[:, 2 * D:].double().view(T, Hv, D)
        k = k / (k.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        g = torch.exp(-torch.exp(A.double()) * torch.nn.functional.softplus(ab[:, :Hv].double() + dt.double()))
        b = torch.sigmoid(ab[:, Hv:].double())
        for t in range(T):
            want *= g[t, :, None, None]
            want += ((v[t] - want @ k[t]) * b[t, :, None])[:, :, None] * k[t]
    chunks, steps = (float((st[0].double() - want).norm() / want.norm()) for st in states)
    assert chunks < 2 * steps + 2 ** -22, (chunks, steps)


def test_steps_of_a_long_memory():
    """Decays of about 0.002 per token: a state remembers some 500 tokens, each of which rounds it twice (2^-25 each, independent)."""
    from parallax_b200.ops import cuda as cu

    torch.manual_seed(5)
    Hv, D, T, slices = 2, 128, 257, 8
    A, dt, w = torch.full((Hv,), -6.0).cuda(), torch.linspace(-2, 1, Hv).cuda(), torch.ones(D).bfloat16().cuda()
    cu_t, slot = torch.tensor([0, T]).int().cuda(), torch.zeros(1).int().cuda()
    want, st = torch.zeros(Hv, D, D, dtype=torch.float64, device="cuda"), torch.zeros(1, Hv, D, D, device="cuda")
    common = torch.randn(1, 2 * D + Hv * D)
    for s in range(slices):
        rows = (common * 0.9 + torch.randn(T, 2 * D + Hv * D) * 0.4).bfloat16().cuda()
        z, ab = (torch.randn(T, n).bfloat16().cuda() for n in (Hv * D, 2 * Hv))
        cu.gated_delta_rule(rows, ab[:, :Hv], ab[:, Hv:], A, dt, z, w, st, cu_t, slot, (torch.arange(T) + s * T).int().cuda(), 1, Hv, D, D,
                            1e-6)
        k, v = rows[:, D:2 * D].double(), rows[:, 2 * D:].double().view(T, Hv, D)
        k = k / (k.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        g = torch.exp(-torch.exp(A.double()) * torch.nn.functional.softplus(ab[:, :Hv].double() + dt.double()))
        b = torch.sigmoid(ab[:, Hv:].double())
        for t in range(T):
            want *= g[t, :, None, None]
            want += ((v[t] - want @ k[t]) * b[t, :, None])[:, :, None] * k[t]
    err = float((st[0].double() - want).norm() / want.norm())
    assert err < 2 ** -25 * (2 * 500) ** 0.5, err
