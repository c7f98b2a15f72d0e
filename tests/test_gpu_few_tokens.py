"""Batches of a few tokens, which have an instance of the kernel without whole units: at its last size and behind it the bits of
whole units, and on a rank that owns none of the experts that the batch reaches, zeros. Whole units with a third weight stage, in both
instances that have them: the bits of two."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, synth, variant_path

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WHOLE, SHORT, SOLO, FEW = 0, 1, 4, 5   # prefill_wgmma_launched_form


@pytest.mark.parametrize("variant,spec,width,local", [("qwen_w1", synth.QWEN, 512, 256), ("ds_ep8", synth.DEEPSEEK, 2048, 32)])
@pytest.mark.parametrize("T", [1, 7, 8, 9])
def test_bits_of_whole_units(variant, spec, width, local, T):
    mk = MonoKernel(variant_path(variant))
    layer = synth.make_layer(spec, seed=1, device=DEV, expert_slice=(0, local) if local != 256 else None, with_shared=False)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=0.5)
    emap = synth.expert_map(spec, 0, 256 // local, device=DEV) if local != 256 else None
    got, ran = [], []
    for size in (None, mk._int_symbol("workspace_min_bytes")):   # without room behind the needed part units stay whole
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        sc["workspace"] = sc["workspace"][:size]
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                        layer["bias"], out, scratch=sc, check=True, expert_map=emap)
        got.append(out)
        ran.append(mk._int_symbol("launched_form"))
    assert ran == [SOLO if T <= 8 else SHORT, WHOLE if variant == "qwen_w1" else FEW]
    assert not torch.isnan(got[0]).any()
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("T", [1, 8])
def test_no_expert_of_this_rank(T):
    spec = synth.QWEN
    mk = MonoKernel(variant_path("qwen_ep8"))
    layer = synth.make_layer(spec, seed=2, device=DEV, expert_slice=(0, 32), with_shared=False)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV)
    logits = batch["logits"].clone()
    logits[:, :32] -= 100.0
    out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
    mk.prefill_impl(batch["hs"], logits, layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True, layer["bias"], out,
                    scratch=mk._allocate_scratch(T, DEV), check=True, expert_map=synth.expert_map(spec, 0, 8, device=DEV))
    assert mk._int_symbol("launched_form") == SOLO
    assert torch.equal(out, torch.zeros_like(out))


@pytest.mark.parametrize("T,form", [(9, SHORT), (300, FEW), (2048, FEW), (2049, WHOLE)])
def test_scales_from_global_memory(T, form):
    """K = 7168 beside an intermediate of 512 columns: a token's output is the same bits with the activation scales in shared memory
    (from 2049 tokens on) and loaded from global memory (below)."""
    spec, first = synth.DEEPSEEK, 2100
    mk = MonoKernel(variant_path("ds_ep8"))
    layer = synth.make_layer(spec, seed=4, device=DEV, expert_slice=(0, 32), with_shared=False)
    batch = synth.make_batch(spec, layer, first, seed=4, device=DEV)
    emap = synth.expert_map(spec, 0, 8, device=DEV)
    out, ran = {}, {}
    for n in (T, first):   # a token's output does not depend on the batch that it is in
        out[n] = torch.full((n, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"][:n], batch["logits"][:n], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                        layer["bias"], out[n], scratch=mk._allocate_scratch(n, DEV), check=True, expert_map=emap)
        ran[n] = mk._int_symbol("launched_form")
    assert ran == {T: form, first: WHOLE}
    assert torch.equal(out[T], out[first][:T])


@pytest.mark.parametrize("T,skew", [(3100, 1.0), (3400, 1.0), (3700, 0.5)])
def test_whole_units_of_a_batch_expected_to_be_split(T, skew):
    """A rank with a part of the experts, a second round of units that even routing would leave nearly empty: with uneven routing there
    are more, and the instance for short batches computes whole units, its scales from global memory and tiles that are full. Without
    room for the split form it is the ordinary instance: the same bits."""
    spec = synth.DEEPSEEK
    mk = MonoKernel(variant_path("ds_ep8"))
    layer = synth.make_layer(spec, seed=6, device=DEV, expert_slice=(0, 32), with_shared=False)
    emap = synth.expert_map(spec, 0, 8, device=DEV)
    for seed in range(20):
        batch = synth.make_batch(spec, layer, T, seed=seed, device=DEV, skew=skew)
        got = []
        for size in (None, mk._int_symbol("workspace_min_bytes")):
            sc = mk._allocate_scratch(T, DEV)
            sc["partial"].fill_(float("nan"))
            sc["workspace"] = sc["workspace"][:size]
            out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
            mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                            layer["bias"], out, scratch=sc, check=True, expert_map=emap)
            got.append((mk._int_symbol("launched_form"), int(mk.workspace_view(sc["workspace"])["phase_ns"][6]) != 0, out))
        (form, split, a), (plain, no_split, b) = got
        assert (form, plain) == (SHORT, WHOLE) and not no_split
        assert not torch.isnan(a).any() and torch.equal(a, b)
        if not split:
            return
    pytest.fail("no batch whose units stay whole")
