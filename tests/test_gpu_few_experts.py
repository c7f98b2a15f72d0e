"""Tokens for which fewer than eight experts can be selected: their other slots have no row, and a launch adds nothing for them,
whatever an earlier one left in the scratch, in every form of the expert phase and both orders of the partial rows."""
import pytest
import torch

from unimonomoe_b200 import synth

pytestmark = pytest.mark.gpu

# one token for every CTA to route itself, units in passes, whole units, the largest batch in slot order and the smallest in
# sorted order; 128-column shards, pairs of tiles; where the bias alone decides (the grouped router), for all tokens alike
CASES = [("qwen_w1", T) for T in (1, 5, 64, 300, 4095, 4096)] + [("qwen_tp4", 5), ("qwen_tp4", 300), ("qwen_w1_pair", 300)]
CASES += [("ds_tp8", T) for T in (3, 64, 4096)] + [("ds_tp2", 64)]
SHAPE = {"qwen_w1": (synth.QWEN, 512), "qwen_tp4": (synth.QWEN, 128), "qwen_w1_pair": (synth.QWEN, 512),
         "ds_tp8": (synth.DEEPSEEK, 256), "ds_tp2": (synth.DEEPSEEK, 1024)}


@pytest.mark.parametrize("variant,T", CASES)
def test_slots_without_an_expert_add_nothing(variant, T):
    from oracle import cpu_oracle as O
    from tests import gpu_util as gu
    mk, (spec, width) = gu.kernel(variant), SHAPE[variant]
    layer = synth.make_layer(spec, seed=8, device=gu.DEV, inter_slice=(0, width) if width != spec.inter else None, with_shared=False)
    batch = synth.make_batch(spec, layer, T, seed=T, device=gu.DEV)
    mode = spec.router_mode
    few = [3, 0, 7, 0, 1][:T]   # selectable experts of the first tokens
    if mode == 0:
        for t, n in enumerate(few):
            batch["logits"][t, torch.randperm(256, device=gu.DEV)[n:]] = -torch.inf
        layer["bias"] = None
    else:
        bias = torch.full_like(layer["bias"], -torch.inf)   # six selectable ones, two in each of three groups
        bias[[5, 9, 69, 73, 133, 137]] = layer["bias"][[5, 9, 69, 73, 133, 137]]
        layer["bias"] = bias
    ran = gu.launch(mk, layer, batch)   # the partial rows are NaN before it
    ids, w, _ = O.route(batch["logits"], mode=mode, bias=layer["bias"])
    assert ((ids >= 0).sum(1)[:len(few)] == (few if mode == 0 else 6)).all()
    assert (ran["ids"] == ids).all()
    assert bool(torch.isfinite(ran["out"].float()).all())
    if mode == 0:
        assert not ran["out"][[t for t, n in enumerate(few) if n == 0]].any()
    toks = gu.sample_tokens(T, 8)
    toks = torch.unique(torch.cat([torch.arange(len(few)), torch.from_numpy(toks).long()])).numpy().astype("int32")
    q, s = O.quant_act(batch["hs"])
    gu.check_output(O, ran["out"], toks, q, s, ids, w, layer)
