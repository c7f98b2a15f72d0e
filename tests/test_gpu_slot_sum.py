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
WHOLE, COPIES = 0, 3   # prefill_wgmma_launched_form
# tokens; shared expert: this rank's part of its tiles, of how many; residual; tokens with fewer than eight experts
CASES = [(7, None, False, False), (STAGES - 1, (0, 1), True, False), (STAGES, None, False, False), (STAGES + 1, (0, 1), False, False),
         (5003, (0, 1), True, False), (30000, None, False, False)]
CASES += [(STAGES + 2, None, True, False), (3333, (1, 3), False, False), (4001, (2, 3), True, True), (3001, None, False, True)]


@pytest.mark.parametrize("T,part,residual,few", CASES)
def test_output_is_the_sum_of_the_partial_rows(T, part, residual, few):
    shared = part is not None
    variant, spec, width = "qwen_tp4", synth.QWEN, 128
    mk = MonoKernel(variant_path(variant))
    layer = synth.make_layer(spec, seed=3, device=DEV, inter_slice=(0, width), with_shared=shared)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=0.5)
    if few:   # tokens at both ends of the batch; their other slots have no row
        for t, n in ((0, 3), (1, 0), (147, 7), (148, 0), (T - 2, 0), (T - 1, 1)):
            batch["logits"][t, torch.randperm(256, device=DEV)[n:]] = -torch.inf
    kw, scale = {}, 2.0 if shared or residual else 1.0
    if shared:
        sh, n, nb = layer["shared"], spec.shared_inter, spec.shared_inter // 128
        a, b = slice(0, width), slice(0, width // 128)
        kw["shared"] = prepare_shared_expert(torch.cat([sh["w13"].view(torch.uint8)[:n][a], sh["w13"].view(torch.uint8)[n:][a]]),
                                             torch.cat([sh["w13_scale"][:nb][b], sh["w13_scale"][nb:][b]]),
                                             sh["w2"].view(torch.uint8)[:, a], sh["w2_scale"][:, b], sh["gate"])
        kw["shared_part"] = part
    if residual:
        kw["residual"] = torch.randn(T, spec.hidden, device=DEV).to(torch.bfloat16)
        if not shared:
            kw["tp"] = (0, 0, 0, 0, 1, 1, 0)   # the entry that folds it, its collective switched off
    if scale != 1.0:
        kw["out_scale"] = scale
    sc = mk._allocate_scratch(T, DEV)
    sc["partial"].fill_(float("nan"))
    out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
    mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                    layer["bias"], out, scratch=sc, check=True, **kw)
    assert mk._int_symbol("launched_form") == (COPIES if T >= STAGES else WHOLE)
    assert bool((sc["topk_ids"] < 0).any()) == few
    rows = sc["partial"][:T * 8].view(T, 8, spec.hidden)
    want = torch.zeros(T, spec.hidden, device=DEV)
    for r in range(8):
        want += rows[:, r].float()
    base = torch.zeros_like(want)
    if shared:
        here = torch.arange(T, device=DEV) // 128 % part[1] == part[0]
        base[here] += sc["partial"][T * 8:T * 9][here].float()
    if residual:
        base += kw["residual"].float()
    assert not torch.isnan(out).any()
    assert torch.equal(out, (want * scale + base).to(torch.bfloat16))
