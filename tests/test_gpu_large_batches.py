"""Decode batches beyond what travels with a launch: more sequences updating at one token than a list holds (their append
counts go through a device array), more sequences than the lengths are passed for (the kernel reads the device's).  Against
the same sequences in batches small enough for both."""

import pytest
import torch

from kvm_paper_b200 import _lib, ops
from oracle import kvm_oracle as ko
from tests import gpu_helpers as gh

pytestmark = pytest.mark.gpu

D, C, H = 32, 16, 1
SPEC = ko.KvmSpec(H, H, D, D, D // 2, C, 2, 8, 1, "power_law", state_growth_factor=4.0, state_min_len=C)
FIELDS = ("k_sum", "v_sum", "vlen", "k_attn", "v_attn")


def _inputs(gen, *lead, h=H):
    rnd = lambda *s: torch.randn(*lead, *s, generator=gen, device="cuda")  # noqa: E731
    norm = lambda t: torch.nn.functional.layer_norm(t, (D,)).bfloat16()  # noqa: E731
    return norm(rnd(h, 1, D)), norm(rnd(h, 1, D)), rnd(h, 1, D).bfloat16(), (1 + torch.nn.functional.elu(rnd(h, 1, 1))).bfloat16()


def _caches(params, spec, prompt, size):
    """Decode caches behind the prompt [B,H,T,..], `size` sequences each."""
    out = []
    for lo in range(0, prompt[0].size(0), size):
        q, k, v, g = (t[lo:lo + size] for t in prompt)
        plan = ops.build_prefill_plan(q.size(2), C, 2, gh.desired_fn(spec))
        runner = ops.PrefillRunner(params, q.size(0), plan)
        res = ops.PrefillResult(runner.run(q, k, v, g), runner.memory, plan, None)
        out.append(ops.decode_cache_from_prefill(params, res, k, v, g, gh.desired_fn(spec)))
    return out


def _same_state(big, small, h=H):
    """The batch `big` and the caches `small` of its sequences in order: lengths, live memory rows, rings."""
    for c in (big, *small):
        c.check_status()
        assert c.total_len.tolist() == c.total_len_h.tolist() and c.state_len.tolist() == c.state_len_h.tolist()
    assert big.total_len_h.tolist() == sum((c.total_len_h.tolist() for c in small), [])
    assert big.state_len_h.tolist() == sum((c.state_len_h.tolist() for c in small), [])
    S = int(big.state_len_h.max())
    for f in FIELDS:
        parts = torch.cat([getattr(c.memory, f)[:, :S] for c in small])
        for s, rows in enumerate(big.state_len_h.tolist()):
            assert torch.equal(getattr(big.memory, f)[s * h:(s + 1) * h, :rows], parts[s * h:(s + 1) * h, :rows]), f
    for f in ("ring_k", "ring_v", "ring_gate"):
        assert torch.equal(getattr(big, f), torch.cat([getattr(c, f) for c in small])), f


def _close(got, want):
    # rows are cut between CTAs at other chunks: probabilities are rounded to bf16 (2^-8 of themselves) against another
    # running maximum, the result once; values stay below 6
    diff = (got.float() - want.float()).abs()
    assert float(diff.max()) <= 2.0 ** -7 * max(1.0, float(want.float().abs().max())) + 2.0 ** -8 * 6
    assert float(diff.mean()) <= 2.0 ** -8 * float(want.float().abs().mean())


@pytest.mark.parametrize("B", [_lib.UPDATE_LIST_MAX + 1, 300])
def test_many_sequences_update_at_one_token(B):
    """All sequences stand at a boundary together and their memories grow; the plain tokens behind it append nothing."""
    spec = gh.bf16_spec(SPEC)
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(B)
    T, n = 3 * C, 2 * C + 3
    prompt = tuple(t[:, :, :, 0].transpose(1, 2) for t in _inputs(gen, B, T))
    (big,), small = _caches(params, spec, prompt, B), _caches(params, spec, prompt, 50)
    before = int(big.state_len_h[0])
    for _ in range(n):
        x = _inputs(gen, B)
        got = big.step(*x)
        want = torch.cat([c.step(*(t[i * 50:(i + 1) * 50] for t in x)) for i, c in enumerate(small)])
        _close(got, want)
    assert int(big.state_len_h[0]) > before and big.update_count == 3 * B
    _same_state(big, small)


# sequences of one length, tokens behind the prompt: more at a boundary than one span launch updates (the others wait for the
# next), more tokens than one piece (a token's place in it is a byte), more sequences than a launch over spans takes
@pytest.mark.parametrize("B,n", [(_lib.UPDATE_LIST_MAX + 6, 3 * C), (3, 2 * 128 + 9), (_lib.SPAN_BATCH_MAX + 5, C + 3)])
def test_runs_of_many_sequences_or_tokens(B, n):
    spec = gh.bf16_spec(SPEC)
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(B + n)
    T, size = 3 * C, 60
    prompt = tuple(t[:, :, :, 0].transpose(1, 2) for t in _inputs(gen, B, T))
    (big,), small = _caches(params, spec, prompt, B), _caches(params, spec, prompt, size)
    x = _inputs(gen, n, B)
    got = big.run(*x)
    want = torch.stack([torch.cat([c.step(*(t[j, i * size:(i + 1) * size] for t in x)) for i, c in enumerate(small)]) for j in range(n)])
    assert got.shape == (n, B, H * D)
    _close(got, want.view(n, B, -1))
    assert big.update_count == sum(c.update_count for c in small) > 0
    _same_state(big, small)


def test_captured_token_reads_the_devices_lengths():
    """A token captured once and replayed goes on from the lengths on the device, like tokens issued one by one."""
    spec = gh.bf16_spec(SPEC)
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(8)
    B, T, n = 5, 3 * C + 2, 9  # (no boundary on the way)
    prompt = tuple(t[:, :, :, 0].transpose(1, 2) for t in _inputs(gen, B, T))
    (a,), (b,) = _caches(params, spec, prompt, B), _caches(params, spec, prompt, B)
    x = _inputs(gen, B)
    for c in (a, b):  # (also: kernels loaded, attributes set)
        c.step(*x)
    fixed = tuple(t.clone() for t in x)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = a.step(*fixed)
    for i in range(n):
        x = _inputs(gen, B)
        for dst, src in zip(fixed, x):
            dst.copy_(src)
        graph.replay()
        _close(y, b.step(*x))
    a.total_len_h += n - 1  # (the capture itself counted one token on the host)
    a.commit_lengths()
    x = _inputs(gen, B)
    _close(a.step(*x), b.step(*x))
    _same_state(a, [b])


@pytest.mark.parametrize("B,h", [(255, 5), (255, 12), (290, 9)])
def test_many_rows_end_in_one_cta(B, h):
    """About eight, twenty and seventeen kv rows per CTA: the new tokens of the first eight are waited for by themselves, those
    of all others together; lengths from the host and from the device."""
    import dataclasses

    spec = gh.bf16_spec(dataclasses.replace(SPEC, num_attention_heads=h, num_key_value_heads=h))
    params = gh.layer_params(spec)
    gen = torch.Generator(device="cuda").manual_seed(h)
    T, n, size = C + 5, 2 * C, 16
    prompt = tuple(t[:, :, :, 0].transpose(1, 2) for t in _inputs(gen, B, T, h=h))
    (big,), small = _caches(params, spec, prompt, B), _caches(params, spec, prompt, size)
    for _ in range(n):
        x = _inputs(gen, B, h=h)
        got = big.step(*x)
        _close(got, torch.cat([c.step(*(t[i * size:(i + 1) * size] for t in x)) for i, c in enumerate(small)]))
    _same_state(big, small, h)
