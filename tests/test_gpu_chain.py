"""The tensor-core chain kernels against the general chain kernel on the same inputs: every routing decision, the carried
sums, the attention view of the final memory.  Cases: the ways an update can go (no appended row, one, a few, more than
the logits-first order takes, the whole block), more touched rows than one scatter pass holds, clusters of 1 to 8 CTAs."""

import pytest
import torch

from kvm_paper_b200 import _lib, ops
from oracle import kvm_oracle as ko
from tests import gpu_helpers as gh
from tests.helpers import assert_close_bf16

pytestmark = pytest.mark.gpu

# block, tokens, heads, batch, rows appended by update u (the last entry repeats), capacity in blocks
CASES = {
    "merges_only": (128, 128 * 9 + 5, 4, 1, [0], 1),
    "one_row_c256": (256, 256 * 9, 8, 2, [1], 2),
    "few_rows": (128, 128 * 10, 3, 1, [2, 3, 7, 9, 16, 0, 1], 2),
    "few_rows_c256": (256, 256 * 8, 20, 1, [16, 5, 0, 8], 2),
    "many_rows": (128, 128 * 9, 2, 2, [17, 127, 1, 40, 0], 4),
    "whole_blocks": (128, 128 * 8 + 2, 8, 2, [128, 0, 128, 3], 4),
    "whole_blocks_c256": (256, 256 * 8, 16, 2, [256, 256, 0], 4),
    "two_scatter_passes": (256, 256 * 7, 40, 4, [0], 1),  # 160 kv rows: one CTA per row, more than 128 touched rows
    "initial_rows_are_sinks": (128, 128 * 7, 2, 1, [1], 2),  # only appended rows take merges
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tensor_core_chain_equals_the_general_chain(name):
    _chains_agree(name, gate_appends=0)


@pytest.mark.parametrize("name", ["few_rows", "many_rows", "whole_blocks", "whole_blocks_c256"])
def test_gated_appends_take_the_gated_keys_of_their_own_block(name):
    """With gated appends the new rows come from the buffer that the next block's gated keys are copied into."""
    _chains_agree(name, gate_appends=1)


def _chains_agree(name, gate_appends):
    C, T, H, B, appends, blocks = CASES[name]
    torch.manual_seed(5)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    sink = C if name == "initial_rows_are_sinks" else 1
    spec = gh.bf16_spec(ko.KvmSpec(H, H, 128, 128, 64, C, 2, blocks, sink, "fixed", state_min_len=C,
                                   kvm_apply_merge_gate_to_appends=gate_appends,
                                   ln_weight=1.0 + 0.1 * torch.randn(128), ln_bias=0.05 * torch.randn(128)))
    params = gh.layer_params(spec)
    step = iter(appends + [appends[-1]] * 1000)
    plan = ops.build_prefill_plan(T, C, 2, lambda ctx, avail, cur: cur + next(step))
    q, v = rnd(B, H, T, 128).bfloat16(), rnd(B, H, T, 128).bfloat16()
    k = torch.nn.functional.layer_norm(rnd(B, H, T, 128), (128,)).bfloat16()
    g = (1 + torch.nn.functional.elu(rnd(B, H, T, 1))).bfloat16()
    runs = []
    for phases in (3, 3 | _lib.PREFILL_LEGACY_CHAIN):
        r = ops.PrefillRunner(params, B, plan, want_route=True)
        r.run(q, k, v, g, phases=phases)
        r.check_status()
        runs.append(r)
    a, b = runs
    S = plan.final_state_len
    assert torch.equal(a.route[:, 1:], b.route[:, 1:])
    for field in ("k_sum", "v_sum"):
        assert torch.equal(getattr(a.memory, field)[:, :S], getattr(b.memory, field)[:, :S]), field
    # a norm of 128 squares: two orders of an fp32 sum differ by at most 2 x 127 x 2^-24 relative, its root by half of that
    assert torch.allclose(a.memory.vlen[:, :S], b.memory.vlen[:, :S], rtol=127 * 2.0 ** -24, atol=0)
    # The two kernels add a row's terms in different orders: mean and variance differ by up to 127 x 2^-24 relative, an element
    # x * w + b of the view (|x| below 8 here) by up to 8 x 127 x 2^-24 < 1e-4 before it is rounded, and then by the
    # neighbouring bf16 number
    for field in ("k_attn", "v_attn"):
        x, y = getattr(a.memory, field)[:, :S].float(), getattr(b.memory, field)[:, :S].float()
        assert bool(((x - y).abs() <= 2.0 ** -7 * torch.maximum(x.abs(), y.abs()) + 1e-4).all()), field
    assert float((a.out.float() - b.out.float()).abs().max()) <= 2e-2


# The routing scan of blocks that are not staged in shared memory (head_dim 128, whole accumulators of 128 tokens): block,
# tokens, heads, rows appended by update u, capacity in blocks, directions the keys are drawn around.  One and two passes of
# up to 256 tokens, tiles of 128 memory rows with and without a remainder, tokens of one warp and of several warps with one
# target, no appended row, one, many, a whole block; 40 heads: clusters of two CTAs, 160: one CTA per kv row.
WIDE = {
    "c512_merges": (512, 512 * 7 + 9, 2, [0], 1, 0),
    "c512_appends": (512, 512 * 8, 3, [1, 130, 3, 512, 17, 0], 4, 0),
    "c512_one_target": (512, 512 * 7, 2, [0, 2, 0], 2, 2),
    "c384_two_passes": (384, 384 * 8, 2, [0, 70, 5], 3, 0),
    "c384_clusters_of_two": (384, 384 * 6, 40, [9, 0], 2, 4),
    "c512_single_ctas": (512, 512 * 5, 160, [33, 0], 2, 0),
}


@pytest.mark.parametrize("name", sorted(WIDE))
def test_wide_routing_scan_decides_like_exact_scores(name):
    """Every decision against float64 scores of the device's own keys and memory rows, the result against the oracle that
    follows these decisions."""
    C, T, H, appends, blocks, clusters = WIDE[name]
    torch.manual_seed(6)
    gen = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    spec = gh.bf16_spec(ko.KvmSpec(H, H, 128, 128, 64, C, 2, blocks, 1, "fixed", state_min_len=C,
                                   ln_weight=1.0 + 0.1 * torch.randn(128), ln_bias=0.05 * torch.randn(128)))
    params = gh.layer_params(spec)
    step = iter(appends + [appends[-1]] * 1000)
    plan = ops.build_prefill_plan(T, C, 2, lambda ctx, avail, cur: cur + next(step))
    k = rnd(1, H, T, 128)
    if clusters:
        k = 0.3 * k + rnd(clusters, 128)[torch.randint(0, clusters, (1, H, T), generator=gen, device="cuda")]
    k = torch.nn.functional.layer_norm(k, (128,)).bfloat16()
    q, v, g = rnd(1, H, T, 128).bfloat16(), rnd(1, H, T, 128).bfloat16(), (1 + torch.nn.functional.elu(rnd(1, H, T, 1))).bfloat16()
    r = ops.PrefillRunner(params, 1, plan, want_route=True)
    r.run(q, k, v, g)
    r.check_status()
    counts = gh.exact_routing_check(spec, ops.PrefillResult(r.out, r.memory, plan, r.route, r), g)
    assert counts["merge_beyond_fp32_noise"] == 0 and counts["append_rows_illegal"] == 0, counts
    heads = slice(0, 2)  # (the oracle runs on the CPU: the first heads)
    small = gh.bf16_spec(ko.KvmSpec(2, 2, 128, 128, 64, C, 2, blocks, 1, "fixed", state_min_len=C, ln_weight=spec.ln_weight, ln_bias=spec.ln_bias))
    small_k, small_v, small_g, small_q = (t[:, heads].cpu() for t in (k, v, g, q))
    step = iter(appends + [appends[-1]] * 1000)
    forced = [gh.decisions_from_route(r.route[heads, u], 1, 2) for u in range(1, plan.n_updates + 1)]
    old, ko.desired_state_len = ko.desired_state_len, lambda spec, ctx, avail, cur: cur + next(step)
    try:
        with torch.no_grad():
            y, state = ko.prefill(small, small_q, small_k, small_v, small_g, forced=forced)
    finally:
        ko.desired_state_len = old
    assert_close_bf16(r.out[:, :, :256].cpu(), y, name)
    S = plan.final_state_len
    for field, want in (("k_sum", state["kvm_s_k"]), ("v_sum", state["kvm_s_v"])):
        scale = max(1.0, float(want.float().abs().max()))
        assert_close_bf16(getattr(r.memory, field)[heads, :S].cpu().view(want.shape), want, f"{name} {field}", max_abs_tol=2e-2 * scale)
