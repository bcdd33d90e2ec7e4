"""Calls of few rows through one library call each: ``ops.project`` against a float64 product, the mixer's cached token and
its prompt against the same module run stage by stage, the decode cache that goes on in the prefill's memory, spans of
decode tokens against single tokens."""

import types

import pytest
import torch

from kvm_paper_b200 import ops
from kvm_paper_b200.mixer import SequenceMixer, StatesCache
from oracle import kvm_oracle as ko
from tests import gpu_helpers as gh

pytestmark = pytest.mark.gpu


# tiles of 8 input rows (1, 2, 4 or 8 of them, a second layer of CTAs above 64), 16 weight rows, 32 of the width per warp
@pytest.mark.parametrize("rows,width,sizes", [
    (1, 32, (8,)), (8, 2048, (256, 64, 5)), (9, 96, (16, 24)), (17, 512, (40, 8, 8, 8, 1)), (33, 288, (17,)), (64, 256, (128,)),
    (65, 256, (48, 16)), (128, 2048, (16,) * 8),
])
@pytest.mark.parametrize("layout", ["contiguous", "column_range", "misaligned"])
def test_project(rows, width, sizes, layout):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    wide = torch.randn(rows, width + 16, generator=gen, device="cuda").bfloat16()
    x = {"contiguous": wide[:, :width].contiguous(), "column_range": wide[:, 8:width + 8], "misaligned": wide[:, 3:width + 3]}[layout]
    ws = [(torch.randn(n, width, generator=gen, device="cuda") * width ** -0.5).bfloat16() for n in sizes]
    got = ops.project(x, ws)[:, :sum(sizes)].double()
    w = torch.cat(ws).double()
    want = x.double() @ w.T
    # fp32 sums of `width` exact products (each addition 2^-24 of the running sum of magnitudes), one rounding to bf16
    bound = 2.0 ** -8 * want.abs() + width * 2.0 ** -23 * (x.double().abs() @ w.abs().T)
    assert bool(((got - want).abs() <= bound).all())


def _mixer(H, Hkv, D, block, hidden, residual="rwkv", shift="rwkv", gated=1):
    config = types.SimpleNamespace(
        num_attention_heads=H, num_key_value_heads=Hkv, d_qk_head=None, d_v_head=None, d_head=D, hidden_size=hidden,
        num_hidden_layers=4, mup_base_dim=768, rope_partial_dim=D // 2, use_value_residual=int(residual != "none"),
        kvm_value_residual_mode=residual, kvm_token_shift_mode=shift, use_tokenshift_att=int(shift != "none"),
        kvm_apply_merge_gate_to_initial_state=0, kvm_apply_merge_gate_to_appends=0, kvm_use_merge_gate_keys=gated,
        kvm_use_merge_gate_values=gated, kvm_use_head_temps=1, kvm_use_vlens=1, sink_len=1, chunk_len=block, n_max_d_chunks=4,
        n_bswa_chunks=2, state_budget_mode="power_law", state_growth_factor=4.0, state_growth_exponent=0.5, state_round_down=1,
        state_min_len=block, state_saturation_n=None)
    torch.manual_seed(7)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        m = SequenceMixer(config, 1)
    finally:
        torch.set_default_dtype(old)
    with torch.no_grad():
        for p in m.parameters():
            p.add_(0.05 * torch.randn(p.shape))
    return m.cuda().eval()


def _rot(D, at, n):
    freq = torch.cat([(1e-4 ** torch.linspace(0, 1, D // 4)).repeat_interleave(2), torch.zeros(D // 2)]).cuda()
    theta = (at + torch.arange(n, device="cuda")).view(1, n, 1, 1) * freq.view(1, 1, 1, -1)
    cos, sin = theta.cos().bfloat16(), theta.sin().bfloat16()
    sin[..., 1::2] *= -1
    return cos, sin


def _drive(m, x, vf, T, n, staged):
    """Prompt of T tokens and n single tokens; ``staged``: through the separate stages (the status is read between them)."""
    m.check_device_status = staged
    past, D, ys = StatesCache(), m.d_qk_head, []
    with torch.no_grad():
        for a, b in [(0, T)] + [(t, t + 1) for t in range(T, T + n)]:
            ys.append(m.forward_inference(x[:, a:b], None if vf is None else vf[:, a:b], _rot(D, a, b - a), None, past_key_values=past))
    cache = past.get_states(m.layer_idx)[m._CACHE_DECODE]
    S, total = int(cache.state_len_h[0]), T + n
    live = torch.arange(ops.bswa_begin_for_total_len(total, m.chunk_len, 2), total, device="cuda") % cache.ring_capacity
    mem = [getattr(cache.memory, f)[:, :S] for f in ("k_sum", "v_sum", "vlen", "k_attn", "v_attn")]
    return torch.cat(ys, 1), mem + [t[:, live] for t in (cache.ring_k, cache.ring_v, cache.ring_gate)]


# query heads, kv heads, head dim, block, batch, prompt, tokens: first block, block boundaries, prompts above and below the
# rows of one project call, more sequences than one tile of rows
@pytest.mark.parametrize("H,Hkv,D,block,B,T,n", [
    (4, 4, 32, 16, 1, 1, 40), (4, 2, 64, 32, 3, 29, 70), (4, 1, 128, 64, 2, 200, 3), (2, 2, 128, 128, 1, 385, 1), (2, 2, 64, 32, 40, 96, 3),
])
@pytest.mark.parametrize("residual,shift,gated", [("rwkv", "rwkv", 1), ("none", "none", 0), ("linear", "rwkv", 1)])
def test_one_call_mixer_equals_its_stages(H, Hkv, D, block, B, T, n, residual, shift, gated):
    m = _mixer(H, Hkv, D, block, 256, residual, shift, gated)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(B, T + n, 256, generator=gen, device="cuda").bfloat16()
    vf = None if residual == "none" else torch.randn(B, T + n, Hkv * D, generator=gen, device="cuda").bfloat16()
    y0, s0 = _drive(m, x, vf, T, n, staged=True)
    y1, s1 = _drive(m, x, vf, T, n, staged=False)
    # the same kernels on the same numbers
    assert torch.equal(y0, y1)
    for a, b in zip(s0, s1):
        assert torch.equal(a, b)


def test_token_takes_any_layout_and_sees_parameters_written_in_place():
    """What the separate layers take, one call takes: inputs off a 16-byte boundary, a broadcast first value; and a parameter
    written through ``.data`` (which leaves no version behind) counts from the next token on."""
    m = _mixer(4, 2, 64, 32, 256)
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(2, 40, 256, generator=gen, device="cuda").bfloat16()
    vf = torch.randn(2, 40, 128, generator=gen, device="cuda").bfloat16()

    def off(t):
        flat = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:]
        return flat.view(t.shape).copy_(t)

    y0, _ = _drive(m, x, vf, 20, 20, staged=True)
    y1, _ = _drive(m, off(x), off(vf), 20, 20, staged=False)
    assert torch.equal(y0, y1)
    one = vf[:1, :1]
    y0, _ = _drive(m, x, one.expand(2, 40, 128), 20, 20, staged=True)
    past = StatesCache()
    m.check_device_status = False
    with torch.no_grad():
        ys = [m.forward_inference(x[:, a:b], one, _rot(64, a, b - a), None, past_key_values=past)
              for a, b in [(0, 20)] + [(t, t + 1) for t in range(20, 40)]]
    assert torch.equal(y0, torch.cat(ys, 1))
    for p in (m.ln_q.weight, m.ln_k.bias, m.x_k, m.v_gate0):
        p.data.add_(torch.randn(p.shape, generator=gen, device="cuda").bfloat16())
    y2, _ = _drive(m, x, vf, 20, 20, staged=False)
    m.use_fused_prologue = False  # the prologue in PyTorch reads the parameters themselves
    y3, _ = _drive(m, x, vf, 20, 20, staged=False)
    # two prologues whose LayerNorm moments are summed in different orders: neighbouring bf16 numbers here and there, where
    # stale parameters (changed by their own size) would leave nothing in common
    assert float((y2.double() - y3.double()).norm() / y3.double().norm()) <= 1e-2
    assert float((y2.double() - y1.double()).norm() / y1.double().norm()) >= 0.1


@pytest.mark.parametrize("T", [5, 32, 64, 65, 200])
def test_cache_in_the_prefills_memory(T):
    """A cache that adopts the prefill's arrays, whose unused rows and slots hold NaN, decodes like a copied one."""
    spec = gh.bf16_spec(ko.KvmSpec(4, 2, 64, 64, 32, 32, 2, 4, 1, "power_law", state_growth_factor=4.0, state_min_len=32))
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(T)
    n = 70
    rnd = lambda h, d: torch.randn(2, h, T + n, d, generator=gen, device="cuda")  # noqa: E731
    q, v, g = rnd(4, 64).bfloat16(), rnd(2, 64).bfloat16(), rnd(2, 1).sigmoid().bfloat16()
    k = torch.nn.functional.layer_norm(rnd(2, 64), (64,)).bfloat16()
    plan = ops.build_prefill_plan(T, 32, 2, gh.desired_fn(spec))
    outs = []
    for adopt in (False, True):
        runner = ops.PrefillRunner(params, 2, plan, memory_capacity=plan.final_state_len + 32, zero_memory=False)
        for t in (runner.memory.k_sum, runner.memory.v_sum, runner.memory.vlen, runner.memory.k_attn, runner.memory.v_attn):
            t.fill_(float("nan"))
        out = runner.run(*(t[:, :, :T] for t in (q, k, v, g)))
        res = ops.PrefillResult(out, runner.memory, plan, None)
        cache = ops.decode_cache_from_prefill(params, res, k[:, :, :T], v[:, :, :T], g[:, :, :T], gh.desired_fn(spec), adopt_memory=adopt)
        assert (cache.memory is res.memory) == adopt
        if adopt:
            free = (torch.arange(64) < plan.bswa_begin) | (torch.arange(64) >= T) if T <= 64 else torch.zeros(64, dtype=torch.bool)
            cache.ring_k[:, free.cuda()] = float("nan")
            cache.ring_v[:, free.cuda()] = float("nan")
        outs.append(torch.cat([cache.step(*(t[:, :, i:i + 1] for t in (q, k, v, g))).clone() for i in range(T, T + n)], 1))
    assert bool(outs[0].isfinite().all()) and torch.equal(outs[0], outs[1])


# query heads, kv heads, head dim, block: one to sixteen query heads per kv head (32 to 2 tokens a span), every head dim
@pytest.mark.parametrize("Hq,Hkv,D,C", [(2, 2, 32, 16), (3, 3, 128, 64), (6, 2, 64, 32), (16, 2, 128, 64), (16, 1, 128, 32)])
def test_spans_equal_single_tokens(Hq, Hkv, D, C):
    """Ragged batch: sequences inside their first block, at a boundary, long past the window; spans cut by boundaries."""
    _spans_against_tokens(Hq, Hkv, D, C, None)


@pytest.mark.parametrize("Hq,Hkv,D,C", [(2, 2, 32, 16), (3, 3, 128, 64), (6, 2, 64, 32), (16, 1, 128, 32)])
@pytest.mark.parametrize("odd", [float("inf"), float("-inf"), float("nan")])
def test_spans_leave_values_that_are_not_numbers_to_the_tokens_that_see_them(Hq, Hkv, D, C, odd):
    _spans_against_tokens(Hq, Hkv, D, C, odd)


def _spans_against_tokens(Hq, Hkv, D, C, odd):
    """``odd``: a value that some elements of the last block's tokens have (they stay in the window until the end)."""
    lens, n = [1, C - 1, C, 2 * C, 2 * C + 1, 3 * C, 9 * C - 7, 20 * C + 3], 3 * C + 5
    spec = gh.bf16_spec(ko.KvmSpec(Hq, Hkv, D, D, D // 2, C, 2, 8, 1, "power_law", state_growth_factor=4.0, state_min_len=C))
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(D + Hq)
    caches = [ops.KvmDecodeCache(params, len(lens), 4 * C, gh.desired_fn(spec)) for _ in range(2)]
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    gate = lambda *s: (1 + torch.nn.functional.elu(rnd(*s))).bfloat16()  # noqa: E731
    norm = lambda *s: torch.nn.functional.layer_norm(rnd(*s), (D,)).bfloat16()  # noqa: E731
    for b, T in enumerate(lens):
        plan = ops.build_prefill_plan(T, C, 2, gh.desired_fn(spec))
        k, v, g = norm(1, Hkv, T, D), rnd(1, Hkv, T, D).bfloat16(), gate(1, Hkv, T, 1)
        res = ops.PrefillRunner(params, 1, plan)
        res.run(rnd(1, Hq, T, D).bfloat16(), k, v, g)
        S, at = plan.final_state_len, plan.bswa_begin
        for c in caches:
            c.load_sequence(b, **{f: getattr(res.memory, f)[:, :S] for f in ("k_sum", "v_sum", "vlen", "k_attn", "v_attn")},
                            window_k=k[0, :, at:], window_v=v[0, :, at:], window_gate=g[0, :, at:], total_len=T)
    for c in caches:
        c.commit_lengths()
    B = len(lens)
    q, k, v, g = rnd(n, B, Hq, 1, D).bfloat16(), norm(n, B, Hkv, 1, D), rnd(n, B, Hkv, 1, D).bfloat16(), gate(n, B, Hkv, 1, 1)
    if odd is not None:  # (one element of every head: the memory of a sequence must not take part, so only the last tokens)
        for i in range(n - 6, n):
            for s in range(B):
                v[i, s, :, 0, (7 * i + 5 * s) % D] = odd
    want = torch.stack([caches[0].step(q[i], k[i], v[i], g[i]).view(B, -1).clone() for i in range(n)])
    got = caches[1].run(q, k, v, g)
    for c in caches:
        c.check_status()
    a, b = caches
    if odd is not None:
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
        assert not bool(want.isfinite().all()) and bool(want[:n - 6].isfinite().all())
        fine = want.isfinite()
        got, want = got[fine], want[fine]
        diff = (got.float() - want.float()).abs()
        assert float(diff.max()) <= 2.0 ** -7 * max(1.0, float(want.float().abs().max())) + 2.0 ** -8 * 6
        return
    assert torch.equal(a.total_len, b.total_len) and torch.equal(a.state_len, b.state_len) and (a.state_len_h == b.state_len_h).all()
    for f in ("k_sum", "v_sum", "vlen", "k_attn", "v_attn"):
        x, y = getattr(a.memory, f), getattr(b.memory, f)
        for s, rows in enumerate(a.state_len_h.tolist()):
            r = slice(s * Hkv, (s + 1) * Hkv)
            assert torch.equal(x[r, :rows], y[r, :rows]), f
    assert torch.equal(a.ring_k, b.ring_k) and torch.equal(a.ring_v, b.ring_v) and torch.equal(a.ring_gate, b.ring_gate)
    # Probabilities are rounded to bf16 against a running maximum, and rows are cut between CTAs at other chunks: each weight
    # may differ by 2^-8 of itself, so a sum of weighted values |v| < 6 by 2^-8 x the weighted mean of |v| (about 0.8), and
    # one rounding of the result
    diff = (got.float() - want.float()).abs()
    assert float(diff.max()) <= 2.0 ** -7 * max(1.0, float(want.float().abs().max())) + 2.0 ** -8 * 6
    assert float(diff.mean()) <= 2.0 ** -8 * float(want.float().abs().mean())


@pytest.mark.parametrize("B,T", [(2, 5), (3, 1)])
def test_hidden_states_of_another_width_are_refused(B, T):
    """Prompts and tokens, as the layers themselves refuse them; the cache still serves the right width afterwards."""
    m = _mixer(2, 2, 32, 16, 256)
    vf = torch.zeros(B, T, 64, device="cuda").bfloat16()
    past = StatesCache()
    with torch.no_grad():
        m.forward_inference(torch.randn(B, T, 256, device="cuda").bfloat16(), vf, _rot(32, 0, T), None, past_key_values=past)
        for width in (128, 224, 288, 512):
            for n, cache, at in ((T, StatesCache(), 0), (1, past, T)):
                with pytest.raises(RuntimeError):
                    m.forward_inference(torch.randn(B, n, width, device="cuda").bfloat16(), vf[:, :n], _rot(32, at, n), None,
                                        past_key_values=cache)
        y = m.forward_inference(torch.randn(B, 1, 256, device="cuda").bfloat16(), vf[:, :1], _rot(32, T, 1), None, past_key_values=past)
    assert y.shape == (B, 1, 256) and past.get_seq_length(m.layer_idx) == T + 1


@pytest.mark.parametrize("T", [20, 150])
@pytest.mark.parametrize("own", ["instance", "subclass", "fp32 parameter"])
def test_a_value_gate_of_ones_own_is_called(T, own):
    """Prompts of few and of many rows and cached tokens, staged and as one call, against the prologue in PyTorch."""
    m = _mixer(4, 2, 64, 32, 256)
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(1, T + 8, 256, generator=gen, device="cuda").bfloat16()
    vf = torch.randn(1, T + 8, 128, generator=gen, device="cuda").bfloat16()
    stock, _ = _drive(m, x, vf, T, 8, staged=False)
    calls = []

    def gate(x):
        calls.append(tuple(x.shape))
        return 0.25 + 0.0 * m.v_gate2(m.v_gate1(x))

    if own == "instance":
        m._value_gate = gate
    elif own == "subclass":
        m.__class__ = type("Own", (SequenceMixer,), {"_value_gate": lambda self, x: gate(x)})
    else:
        m.v_gate0 = torch.nn.Parameter(m.v_gate0.detach().float() * 3.0)
    ys = [_drive(m, x, vf, T, 8, staged=staged)[0] for staged in (False, True)]
    assert torch.equal(*ys)
    assert own == "fp32 parameter" or calls == 2 * ([(1, T, 256)] + 8 * [(1, 1, 256)])
    m.use_fused_prologue = False
    want, _ = _drive(m, x, vf, T, 8, staged=False)
    # (neighbouring bf16 numbers here and there, as above; the stock gate is far off)
    assert float((ys[0].double() - want.double()).norm() / want.double().norm()) <= 1e-2
    assert float((stock.double() - want.double()).norm() / want.double().norm()) >= 0.05
