"""Batches of a few tokens, which have an instance of the kernel without whole units: at its last size and behind it the bits of
whole units, and on a rank that owns none of the experts that the batch reaches, zeros."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, synth, variant_path

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("variant,spec,width,local", [("qwen_w1", synth.QWEN, 512, 256), ("ds_ep8", synth.DEEPSEEK, 2048, 32)])
@pytest.mark.parametrize("T", [1, 7, 8, 9])
def test_bits_of_whole_units(variant, spec, width, local, T):
    mk = MonoKernel(variant_path(variant))
    layer = synth.make_layer(spec, seed=1, device=DEV, expert_slice=(0, local) if local != 256 else None, with_shared=False)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=0.5)
    emap = synth.expert_map(spec, 0, 256 // local, device=DEV) if local != 256 else None
    got = []
    for size in (None, mk._int_symbol("workspace_min_bytes")):   # without room behind the needed part units stay whole
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        sc["workspace"] = sc["workspace"][:size]
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                        layer["bias"], out, scratch=sc, check=True, expert_map=emap)
        got.append(out)
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
    assert torch.equal(out, torch.zeros_like(out))


@pytest.mark.parametrize("T", [9, 300, 2048, 2049])
def test_scales_from_global_memory(T):
    """K = 7168 beside an intermediate of 512 columns: a token's output is the same bits with the activation scales in shared memory
    (from 2049 tokens on) and loaded from global memory (below)."""
    spec, first = synth.DEEPSEEK, 2049
    mk = MonoKernel(variant_path("ds_ep8"))
    layer = synth.make_layer(spec, seed=4, device=DEV, expert_slice=(0, 32), with_shared=False)
    batch = synth.make_batch(spec, layer, first, seed=4, device=DEV)
    emap = synth.expert_map(spec, 0, 8, device=DEV)
    out = {}
    for n in (T, first):   # a token's output does not depend on the batch that it is in
        out[n] = torch.full((n, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"][:n], batch["logits"][:n], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                        layer["bias"], out[n], scratch=mk._allocate_scratch(n, DEV), check=True, expert_map=emap)
    assert torch.equal(out[T], out[first][:T])
