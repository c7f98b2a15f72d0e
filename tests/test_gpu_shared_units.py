"""Units given to several CTAs (128-column shards: few units, or few behind the full rounds): a token's output has the bits that
it has in a batch whose units each stay with one CTA, and meets the oracle's bound."""
import pytest
import torch

from unimonomoe_b200 import synth
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu


# one to eight CTAs a unit; behind one round and several; the shared expert's tiles among the units
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("T", [1, 2, 3, 7, 9, 33, 5000, 8192])
def test_shared_units_give_the_bits_of_whole_units(T, shared):
    from oracle import cpu_oracle as O
    from tests import gpu_util as gu
    mk = gu.kernel("qwen_tp4")
    layer = synth.make_layer(synth.QWEN, seed=6, device=gu.DEV, inter_slice=(128, 256), with_shared=shared)
    kw = {}
    if shared:
        sh = layer["shared"]
        n, a, b = synth.QWEN.shared_inter, slice(0, 128), slice(0, 1)
        kw["shared"] = prepare_shared_expert(
            torch.cat([sh["w13"].view(torch.uint8)[:n][a], sh["w13"].view(torch.uint8)[n:][a]]),
            torch.cat([sh["w13_scale"][:n // 128][b], sh["w13_scale"][n // 128:][b]]),
            sh["w2"].view(torch.uint8)[:, a], sh["w2_scale"][:, b], sh["gate"])
    batch = synth.make_batch(synth.QWEN, layer, T, seed=T, device=gu.DEV, skew=0.5 if T < 4096 else 0.0)

    def run(hs, logits):
        sc = mk._allocate_scratch(len(hs), gu.DEV)
        sc["partial"].fill_(float("nan"))
        out = torch.full((len(hs), 2048), float("nan"), dtype=torch.bfloat16, device=gu.DEV)
        mk.prefill_impl(hs, logits, layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True, None, out,
                        scratch=sc, check=True, **kw)
        return out, sc, mk.workspace_view(sc["workspace"])["total_tiles"] + (-(-len(hs) // 128) if shared else 0)

    out, sc, units = run(batch["hs"], batch["logits"])
    assert bool(torch.isfinite(out.float()).all())
    # the same tokens among others, 300 at a time: too many units behind the full rounds to be shared
    gen = torch.Generator().manual_seed(1)
    some = torch.sort(torch.randperm(T, generator=gen)[:100]).values.to(gu.DEV)
    other = synth.make_batch(synth.QWEN, layer, 300 - len(some), seed=77, device=gu.DEV)
    whole, _, n = run(torch.cat([batch["hs"][some], other["hs"]]), torch.cat([batch["logits"][some], other["logits"]]))
    assert 2 * (n % 148) > 148
    assert torch.equal(out[some].view(torch.int16), whole[:len(some)].view(torch.int16))
    if not shared:
        toks = some[:16].cpu().numpy().astype("int32")
        q, s = O.quant_act(batch["hs"])
        ids, w, _ = O.route(batch["logits"], mode=0)
        gu.check_output(O, out, toks, q, s, ids, w, layer)
