"""The sum of a token's partial rows where the copy engine brings them (128-column shards, from twenty tokens a CTA on) and just
below: the output is the fp32 sum of the partial rows that the launch left, slot by slot, times the scale, with the shared
expert's row and the residual on top, rounded once. Scales are powers of two, so a product rounds nothing and the bits have to be
the same."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, synth, variant_path
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
STAGES = 20 * 148   # tokens from which the copy engine brings them
# tokens; shared expert; residual
CASES = [(7, False, False), (STAGES - 1, True, True), (STAGES, False, False), (STAGES + 1, True, False), (5003, True, True), (30000, False, False)]


@pytest.mark.parametrize("T,shared,residual", CASES)
def test_output_is_the_sum_of_the_partial_rows(T, shared, residual):
    variant, spec, width = "qwen_tp4", synth.QWEN, 128
    mk = MonoKernel(variant_path(variant))
    layer = synth.make_layer(spec, seed=3, device=DEV, inter_slice=(0, width), with_shared=shared)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=0.5)
    kw, scale = {}, 2.0 if shared or residual else 1.0
    if shared:
        sh, n, nb = layer["shared"], spec.shared_inter, spec.shared_inter // 128
        a, b = slice(0, width), slice(0, width // 128)
        kw["shared"] = prepare_shared_expert(torch.cat([sh["w13"].view(torch.uint8)[:n][a], sh["w13"].view(torch.uint8)[n:][a]]),
                                             torch.cat([sh["w13_scale"][:nb][b], sh["w13_scale"][nb:][b]]),
                                             sh["w2"].view(torch.uint8)[:, a], sh["w2_scale"][:, b], sh["gate"])
    if residual:
        kw["residual"] = torch.randn(T, spec.hidden, device=DEV).to(torch.bfloat16)
    if scale != 1.0:
        kw["out_scale"] = scale
    sc = mk._allocate_scratch(T, DEV)
    sc["partial"].fill_(float("nan"))
    out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
    mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                    layer["bias"], out, scratch=sc, check=True, **kw)
    rows = sc["partial"][:T * 8].view(T, 8, spec.hidden)
    want = torch.zeros(T, spec.hidden, device=DEV)
    for r in range(8):
        want += rows[:, r].float()
    base = torch.zeros_like(want)
    if shared:
        base += sc["partial"][T * 8:T * 9].float()
    if residual:
        base += kw["residual"].float()
    assert not torch.isnan(out).any()
    assert torch.equal(out, (want * scale + base).to(torch.bfloat16))
