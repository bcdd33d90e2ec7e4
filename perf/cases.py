"""The calls that the speed of this package is judged by: what a program that serves or evaluates a model with the
Key-Value-Means mixer has the package do, through the entry points such a program uses.

  prefill       ``ops.PrefillRunner.run``: a batch of post-QKV tensors through the memory chain and the block attention,
                with the runner kept between calls (as a server keeps one per shape)
  prompt        ``SequenceMixer.forward_inference`` with an empty layer cache: projections, token shift, value residual,
                q/k LayerNorm, rotary embedding, prefill, output projection and the hand-over to the decode cache
  decode_step   ``ops.KvmDecodeCache.step``: one token for every sequence of a (ragged) batch
  decode_run    ``ops.KvmDecodeCache.run``: several tokens whose inputs are on the device (scoring a given continuation)
  token         ``SequenceMixer.forward_inference`` with a filled layer cache: one token through the whole mixer

A case is described by plain values:

  call, batch, tokens (prompt length; for decoding the context length, or its upper end for a ragged batch), tokens_lo
  (lower end of a ragged batch, 0 = all alike), steps (tokens of one decode_run), q_heads, kv_heads, head_dim, block
  (tokens per block), window (blocks), schedule ("fixed": a memory of `cap` means, "sqrt": 16 * sqrt(context) means up to
  `cap`, "plus_one": one more mean per block up to `cap`), cap, clusters (keys drawn from that many Gaussian clusters,
  0 = none), hidden (width of the layer, for the calls that go through the class).

All of it is bf16, as the package is.
"""

import math
import types

import numpy as np
import torch

from kvm_paper_b200 import ops
from kvm_paper_b200.mixer import SequenceMixer, StatesCache

ROPE_DIM = 64   # rotary dimensions per head (half of them at head_dim 64: with all of them rotary no key content is left to route by)
SINK = 1


def _case(name, call, batch, tokens, q_heads, kv_heads, head_dim, block, schedule, cap, *, tokens_lo=0, steps=1, window=2,
          clusters=0, hidden=0):
    c = dict(call=call, batch=batch, tokens=tokens, tokens_lo=tokens_lo, steps=steps, q_heads=q_heads, kv_heads=kv_heads,
             head_dim=head_dim, block=block, window=window, schedule=schedule, cap=cap, clusters=clusters, hidden=hidden)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one layer of a 2048-wide model prefilling four 32k documents, one new mean per 256-token block
        _case("prefill_4x32768", "prefill", 4, 32768, 16, 16, 128, 256, "plus_one", 1024),
        # the same layer with the square-root memory schedule (hundreds of appends per block at first, then merges only),
        # three documents of an odd length
        _case("prefill_3x30011_sqrt", "prefill", 3, 30011, 16, 16, 128, 256, "sqrt", 1024),
        # a very long document: 4096-wide layer, blocks of 512, up to 4096 means, keys with a cluster structure
        _case("prefill_1x262144_block512", "prefill", 1, 262144, 32, 32, 128, 512, "sqrt", 4096, clusters=64),
        # a batch of medium prompts with a fixed memory of one block: many short chains side by side
        _case("prefill_8x4096_fixed", "prefill", 8, 4096, 32, 32, 128, 256, "fixed", 256),
        # a small model: 8 heads x 64, blocks of 128, a fixed memory of 256 means
        _case("prefill_1x4096_d64", "prefill", 1, 4096, 8, 8, 64, 128, "fixed", 256),
        # a request's prompt through the whole mixer, grouped queries, odd length
        _case("prompt_1x4099_gqa", "prompt", 1, 4099, 16, 4, 128, 256, "sqrt", 1024, hidden=2048),
        # the shortest ordinary prompt (a chat turn, less than one block): launches and host work
        _case("prompt_1x77", "prompt", 1, 77, 16, 16, 128, 256, "sqrt", 1024, hidden=2048),
        # a serving batch of 64 conversations at contexts of 4k to 64k, 32 tokens each
        _case("decode_64x32_ragged", "decode_run", 64, 65536, 16, 16, 128, 256, "sqrt", 1024, tokens_lo=4096, steps=32),
        # one conversation: the latency of a token
        _case("decode_step_1", "decode_step", 1, 20480, 16, 16, 128, 256, "sqrt", 1024),
        # a batch of grouped-query conversations with a fixed memory, contexts that have left the window only just or long ago
        _case("decode_step_24_gqa", "decode_step", 24, 6000, 32, 8, 128, 256, "fixed", 256, tokens_lo=700),
        # many conversations of a small model
        _case("decode_step_200_d64", "decode_step", 200, 9000, 8, 8, 64, 128, "fixed", 256, tokens_lo=300),
        # a token of eight conversations of one length through the whole mixer
        _case("token_8", "token", 8, 1500, 16, 16, 128, 256, "fixed", 256, hidden=2048),
    ]


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    def size(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    call = rng.choice(["prefill", "prefill", "prompt", "decode_run", "decode_step", "token"])
    head_dim = rng.choice([64, 128, 128])
    block = rng.choice([128, 256]) if head_dim == 64 else rng.choice([128, 256, 256, 512])
    q_heads = rng.choice([8, 16, 32])
    kv_heads = q_heads // rng.choice([1, 1, 2, 4])
    if call in ("prompt", "token"):  # layers of up to 2048
        q_heads = min(q_heads, 2048 // head_dim)
        kv_heads = min(kv_heads, q_heads)
    schedule = rng.choice(["fixed", "sqrt", "plus_one"])
    cap = block if schedule == "fixed" and rng.random() < 0.5 else rng.choice([2, 4]) * block
    if schedule == "sqrt" and block == 512 and rng.random() < 0.5:
        cap = 4096
    clusters = rng.choice([0, 0, 64])
    kw = dict(clusters=clusters)
    if call == "prefill":
        batch = size(1, 8)
        tokens = size(block // 2, 40000)
        while batch * tokens * q_heads > 4 * 32768 * 16:  # at most the headline's tokens x heads
            tokens = max(1, tokens * 2 // 3)
    elif call == "prompt":
        batch, tokens = size(1, 4), size(20, 12000)
        while batch * tokens > 16384:
            tokens = tokens * 2 // 3
        kw["hidden"] = q_heads * head_dim
    elif call == "token":
        batch, tokens = size(1, 48), size(20, 3000)
        schedule, cap = "fixed", rng.choice([1, 2]) * block
        kw["hidden"] = q_heads * head_dim
    else:
        # contexts whose memory has reached its size: a program decodes on, the cost of a token stays what it is
        batch = size(1, 128 if kv_heads * head_dim <= 1024 else 64)
        lo = 3 * block + size(1, 2000)
        tokens = lo + size(1, 50000)
        if schedule != "fixed":
            schedule, cap = "sqrt", min(cap, 1024)
            lo, tokens = lo + 6 * cap, tokens + 6 * cap
        kw["tokens_lo"] = lo
        kw["steps"] = size(4, 32) if call == "decode_run" else 1
        kw["clusters"] = 0
    return _case("", call, batch, tokens, q_heads, kv_heads, head_dim, block, schedule, cap, **kw)


# ------------------------------------------------------------------------------------------------ the schedules
def _desired_fn(case):
    block, cap, kind = case["block"], case["cap"], case["schedule"]

    def desired(ctx_len, available_context, current):
        cur, avail = max(int(current), 0), max(int(available_context), 0)
        if kind == "fixed":
            want = cap
        elif kind == "sqrt":
            want = max(int(math.floor(16.0 * float(max(int(ctx_len), 0)) ** 0.5)), block)
        else:
            want = cur + 1
        return max(min(want, avail, cap), cur)

    return desired


def _plan_sizes(case):
    """(memory rows before, appended) of every block a prompt's chain consumes, and the rows in the end."""
    T, C, W = case["tokens"], case["block"], case["window"]
    want = _desired_fn(case)
    S = min(T, C)
    out = [(0, S)]
    for u in range(1, max(1, -(-T // C) - W)):
        n = min(max(want((u + W) * C, (u + 1) * C, S) - S, 0), C)
        out.append((S, n))
        S += n
    return out, S


def _contexts(case):
    """Context length of every sequence of a decode batch (a property of the case, like its other sizes)."""
    if not case["tokens_lo"]:
        return [case["tokens"]] * case["batch"]
    return np.random.RandomState(17).randint(case["tokens_lo"], case["tokens"] + 1, size=case["batch"]).tolist()


def _memory_rows(case, context):
    """Rows of the memory of a sequence that decodes at this context: the schedule's limit, or one per covered token."""
    covered = max(min(context, case["block"]), ops.bswa_begin_for_total_len(context, case["block"], case["window"]))
    return min(covered, case["cap"])


# ------------------------------------------------------------------------------------------------ inputs
def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32)


def _keys(case, gen, B, T, H, D):
    """Per-head normalised keys, as the key LayerNorm leaves them; with `clusters` around a few directions."""
    ln = torch.nn.functional.layer_norm
    if not case["clusters"]:
        return ln(_normal(gen, B, T, H, D), (D,)).bfloat16()
    centres = _normal(gen, case["clusters"], D)
    which = torch.randint(0, case["clusters"], (B, T, H), generator=gen, device="cuda")
    return ln(centres[which].add_(_normal(gen, B, T, H, D), alpha=0.5), (D,)).bfloat16()


def _gates(gen, *shape):
    return (1.0 + torch.nn.functional.elu(0.5 * _normal(gen, *shape))).bfloat16()


def _rope_dim(case):
    return min(ROPE_DIM, case["head_dim"] // 2)


def _layer(case, gen):
    D = case["head_dim"]
    cfg = ops.LayerConfig(n_q_heads=case["q_heads"], n_kv_heads=case["kv_heads"], head_dim=D, chunk_len=case["block"],
                          n_bswa_chunks=case["window"], rope_dim=_rope_dim(case), sink_len=SINK)
    temps = [1.0 + 0.2 * torch.rand(case["q_heads"], generator=gen, device="cuda") for _ in range(2)]
    return ops.LayerParams(cfg, 1.0 + 0.1 * _normal(gen, D), 0.05 * _normal(gen, D), temps[0], temps[1], "cuda")


def _post_qkv(case, gen, B, T):
    """q, k, v, gate as the projections leave them: [B,T,H,D] storage, handed over as [B,H,T,D] views."""
    Hq, Hkv, D = case["q_heads"], case["kv_heads"], case["head_dim"]
    q = torch.nn.functional.layer_norm(_normal(gen, B, T, Hq, D), (D,)).bfloat16()
    k = _keys(case, gen, B, T, Hkv, D)
    v = _normal(gen, B, T, Hkv, D).bfloat16()
    g = _gates(gen, B, T, Hkv, 1)
    return tuple(t.transpose(1, 2) for t in (q, k, v, g))


def _mixer(case, seed):
    """The layer as a model holds it: token shift and value residual on, as in the reference's model configurations."""
    H, D = case["q_heads"], case["head_dim"]
    config = types.SimpleNamespace(
        num_attention_heads=H, num_key_value_heads=case["kv_heads"], d_qk_head=None, d_v_head=None, d_head=D,
        hidden_size=case["hidden"], num_hidden_layers=24, mup_base_dim=768, rope_partial_dim=_rope_dim(case),
        use_value_residual=1, kvm_value_residual_mode="rwkv", kvm_token_shift_mode="rwkv", use_tokenshift_att=1,
        kvm_apply_merge_gate_to_initial_state=0, kvm_apply_merge_gate_to_appends=0, kvm_use_merge_gate_keys=1,
        kvm_use_merge_gate_values=1, kvm_use_head_temps=1, kvm_use_vlens=1, sink_len=SINK, chunk_len=case["block"],
        n_max_d_chunks=max(1, case["cap"] // case["block"]), n_bswa_chunks=case["window"],
        state_budget_mode="fixed" if case["schedule"] == "fixed" else "power_law",
        state_growth_factor=16.0, state_growth_exponent=0.5, state_round_down=1,
        state_min_len=case["cap"] if case["schedule"] == "fixed" else case["block"], state_saturation_n=None)
    torch.manual_seed(seed)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        m = SequenceMixer(config, 3)
    finally:
        torch.set_default_dtype(old)
    with torch.no_grad():  # a trained layer: no parameter at its neutral start value
        m.c_proj.weight.normal_(std=case["hidden"] ** -0.5)
        m.v_gate1.weight.normal_(std=case["hidden"] ** -0.5)
        m.ln_s_k.weight.add_(0.1 * torch.randn(D))
        m.ln_s_k.bias.add_(0.05 * torch.randn(D))
        m.front_head_temp.add_(0.2 * torch.rand(H))
        m.state_head_temp.add_(0.2 * torch.rand(H))
    if case["schedule"] == "plus_one":
        m._desired_state_len = _desired_fn(case)
    return m.cuda().eval()


def _rotary(case, n):
    D, rope = case["head_dim"], _rope_dim(case)
    freq = (1 / 10000.0) ** torch.linspace(0.0, 1.0, steps=rope // 2, dtype=torch.float32, device="cuda")
    freq = torch.cat([freq.repeat_interleave(2), freq.new_zeros(D - rope)])
    theta = torch.arange(n, device="cuda", dtype=torch.float32).view(1, n, 1, 1) * freq.view(1, 1, 1, -1)
    cos, sin = theta.cos().bfloat16(), theta.sin().bfloat16()
    sin[..., 1::2] *= -1
    return cos, sin


def _hidden(case, gen, T):
    x = torch.nn.functional.layer_norm(_normal(gen, case["batch"], T, case["hidden"]), (case["hidden"],)).bfloat16()
    v_first = _normal(gen, case["batch"], T, case["kv_heads"] * case["head_dim"]).bfloat16()
    return x, v_first


def _decode_cache(case, gen, params):
    """A decode batch in mid-flight: memories of sums over many merged tokens, full windows, ragged lengths."""
    Hkv, D, C, W = case["kv_heads"], case["head_dim"], case["block"], case["window"]
    contexts = _contexts(case)
    cache = ops.KvmDecodeCache(params, case["batch"], case["cap"] + C, _desired_fn(case))
    ln = torch.nn.functional.layer_norm
    for b, T in enumerate(contexts):
        S = _memory_rows(case, T)
        begin = ops.bswa_begin_for_total_len(T, C, W)
        count = 1.0 + 4.0 * torch.rand(Hkv, S, 1, generator=gen, device="cuda") ** 2 * max(1.0, T / S)
        d = _normal(gen, 2, Hkv, S, D)
        d[0, :, :, :_rope_dim(case)] = 0.0
        noise = _normal(gen, 2, Hkv, S, D)
        k_sum = ln(d[0], (D,)) * count + noise[0] * count.sqrt()
        v_sum = d[1] * count.sqrt() + noise[1]
        cache.load_sequence(
            b, k_sum=k_sum.bfloat16(), v_sum=v_sum.bfloat16(), vlen=d[1].norm(dim=-1),
            window_k=ln(_normal(gen, Hkv, T - begin, D), (D,)).bfloat16(), window_v=_normal(gen, Hkv, T - begin, D).bfloat16(),
            window_gate=_gates(gen, Hkv, T - begin), total_len=T)
    cache.commit_lengths(refresh_attention_view=True)
    return cache


def _token_inputs(case, gen, *lead):
    B, Hq, Hkv, D = case["batch"], case["q_heads"], case["kv_heads"], case["head_dim"]
    ln = torch.nn.functional.layer_norm
    return (ln(_normal(gen, *lead, B, Hq, 1, D), (D,)).bfloat16(), ln(_normal(gen, *lead, B, Hkv, 1, D), (D,)).bfloat16(),
            _normal(gen, *lead, B, Hkv, 1, D).bfloat16(), _gates(gen, *lead, B, Hkv, 1, 1))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    call, s = case["call"], {"call": case["call"]}
    with torch.no_grad():
        if call == "prefill":
            params = _layer(case, gen)
            plan = ops.build_prefill_plan(case["tokens"], case["block"], case["window"], _desired_fn(case))
            s["runner"] = ops.PrefillRunner(params, case["batch"], plan)
            s["in"] = _post_qkv(case, gen, case["batch"], case["tokens"])
        elif call in ("decode_step", "decode_run"):
            s["cache"] = _decode_cache(case, gen, _layer(case, gen))
            s["in"] = _token_inputs(case, gen, case["steps"]) if call == "decode_run" else _token_inputs(case, gen)
        else:
            s["mixer"] = _mixer(case, seed)
            s["in"] = _hidden(case, gen, case["tokens"])
            s["rotary"] = _rotary(case, case["tokens"])
            if call == "token":
                s["past"] = StatesCache()
                s["mixer"].forward_inference(*s["in"], s["rotary"], None, past_key_values=s["past"])
                s["in"] = _hidden(case, gen, 1)
                s["rotary"] = tuple(t[:, -1:] for t in _rotary(case, case["tokens"] + 1))
    return s


def _carried(memory, rows):
    """The carried memory behind a call: sums, magnitudes and the view the attention reads."""
    return [t[:, :rows] for t in (memory.k_sum, memory.v_sum, memory.vlen, memory.k_attn, memory.v_attn)]


@torch.no_grad()
def run(state):
    call = state["call"]
    if call == "prefill":
        runner = state["runner"]
        out = runner.run(*state["in"])
        return [out] + _carried(runner.memory, runner.plan.final_state_len)
    if call == "decode_step":
        cache = state["cache"]
        return [cache.step(*state["in"]), cache.memory.k_attn, cache.memory.v_attn, cache.ring_k, cache.ring_v]
    if call == "decode_run":
        cache = state["cache"]
        return [cache.run(*state["in"]), cache.memory.k_attn, cache.memory.v_attn, cache.ring_k, cache.ring_v]
    mixer, (x, v_first) = state["mixer"], state["in"]
    past = StatesCache() if call == "prompt" else state["past"]
    y = mixer.forward_inference(x, v_first, state["rotary"], None, past_key_values=past)
    cache = past.get_states(mixer.layer_idx)["kvm_b200_decode_cache"]
    return [y] + _carried(cache.memory, int(cache.state_len_h[0]))


# ------------------------------------------------------------------------------------------------ what a call cannot do without
def _prefill_work(case):
    """Bytes and operations of the operator: every post-QKV tensor read once, the output and the carried memory written
    once; scores and weighted sums of every visible (query, key) pair, the routing scores of every consumed token."""
    B, T, C, W, D = case["batch"], case["tokens"], case["block"], case["window"], case["head_dim"]
    Hq, Hkv = case["q_heads"], case["kv_heads"]
    sizes, S = _plan_sizes(case)
    front = min(T, W * C)
    pairs = front * (front + 1) // 2
    for j in range(W, -(-T // C)):
        n, start = min(T, (j + 1) * C) - j * C, (j + 1 - W) * C
        pairs += n * (j * C - start) + n * (n + 1) // 2 + n * sum(sizes[j - W])
    routing = sum((C - n) * (s + n) + (C * s if 0 < n < C else 0) for s, n in sizes[1:])
    flops = 4.0 * D * pairs * B * Hq + 2.0 * D * routing * B * Hkv
    nbytes = 2.0 * B * T * (2 * Hq * D + 2 * Hkv * D + Hkv) + B * Hkv * S * (4 * D * 2 + 4)
    return nbytes, flops


def _projection_work(case, T):
    """The mixer's linear layers around the operator for `T` tokens: weights once, activations in and out once."""
    B, h, dq, dk = case["batch"], case["hidden"], case["q_heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    weights = h * (2 * dq + 2 * dk + case["kv_heads"])
    return 2.0 * weights + 2.0 * B * T * (2 * h + dk), 2.0 * B * T * weights


def work(case):
    call = case["call"]
    Hq, Hkv, D = case["q_heads"], case["kv_heads"], case["head_dim"]
    if call in ("prefill", "prompt"):
        nbytes, flops = _prefill_work(case)
        if call == "prompt":  # q, k, v and the operator's output stay inside the call
            nbytes -= 2.0 * case["batch"] * case["tokens"] * (2 * Hq * D + 2 * Hkv * D + Hkv)
            more = _projection_work(case, case["tokens"])
            nbytes, flops = nbytes + more[0], flops + more[1]
        return {"bytes": nbytes, "flops": flops}
    C, W = case["block"], case["window"]
    rows = 0.0  # memory and window rows the tokens attend to (the window holds W - 1/2 blocks on average)
    for T in _contexts(case):
        win = (W - 0.5) * C
        rows += (_memory_rows(case, T) + win if T > W * C else T) * case["steps"]
    nbytes = rows * Hkv * 2 * D * 2 + case["steps"] * case["batch"] * (2 * Hq * D + 4 * Hkv * D) * 2.0
    flops = 4.0 * D * rows * Hq
    if call == "token":
        more = _projection_work(case, 1)
        nbytes, flops = nbytes + more[0], flops + more[1]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bf16 operands and results (8 bits of mantissa): scores, probabilities and sums are each rounded to bf16 on the way
    return {"rel": 1e-2}
