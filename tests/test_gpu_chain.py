"""The tensor-core chain kernels against the general chain kernel on the same inputs: every routing decision, the carried
sums, the attention view of the final memory.  Cases: the ways an update can go (no appended row, one, a few, more than
the logits-first order takes, the whole block), more touched rows than one scatter pass holds, clusters of 1 to 8 CTAs."""

import pytest
import torch

from kvm_paper_b200 import _lib, ops
from oracle import kvm_oracle as ko
from tests import gpu_helpers as gh

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
    C, T, H, B, appends, blocks = CASES[name]
    torch.manual_seed(5)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    sink = C if name == "initial_rows_are_sinks" else 1
    spec = gh.bf16_spec(ko.KvmSpec(H, H, 128, 128, 64, C, 2, blocks, sink, "fixed", state_min_len=C,
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
