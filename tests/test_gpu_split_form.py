"""The split form of the expert phase (units cut into passes, dealt over all SMs in two halves) against whole units (the
same launch with a workspace that has no room for the split intermediate): the outputs have to be the same bits,
because every row sees the same operations in the same order."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, build as kbuild, synth, variant_path
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# (build, layer, intermediate columns, local experts, shared expert), tokens: fewer passes than SMs, about one and two
# rounds of units, one column pass per unit, ragged and full tiles, the shared expert's tiles, units in chunks
CASES = [(("qwen_w1", synth.QWEN, 512, 256, False), T) for T in (1, 2, 9, 32)]
CASES += [(("qwen_tp2", synth.QWEN, 256, 256, False), T) for T in (1, 3)]
CASES += [(("qwen_ep4", synth.QWEN, 512, 64, False), T) for T in (9, 257)]
CASES += [(("qwen_w1", synth.QWEN, 512, 256, True), T) for T in (3, 32)]
CASES += [(("ds_tp8", synth.DEEPSEEK, 256, 256, False), T) for T in (1, 4)]
CASES += [(("ds_ep8", synth.DEEPSEEK, 2048, 32, True), T) for T in (8, 20)]
# more than 64 K slabs: a lane holds the weight scales of three of them
WIDE = synth.LayerSpec("wide", hidden=9216, inter=256)
CASES += [(("wide_ep8", WIDE, 256, 32, False), T) for T in (3, 16)]
# every token on this rank's experts: 65536 rows, several waves of units through the intermediate
CASES += [(("qwen_ep4", synth.QWEN, 512, 64, False), 8192)]
_layers = {}


def _layer(build):
    if build not in _layers:
        _layers.clear()   # one layer on the GPU at a time
        variant, spec, width, local, shared = build
        _layers[build] = synth.make_layer(
            spec, seed=21, device=DEV, inter_slice=(0, width) if width != spec.inter else None,
            expert_slice=(0, local) if local != 256 else None, with_shared=shared)
    return _layers[build]


@pytest.mark.parametrize("build,T", CASES, ids=[f"{b[0]}{'-shared' if b[4] else ''}-{T}" for b, T in CASES])
def test_split_units_give_the_bits_of_whole_units(build, T):
    variant, spec, width, local, shared = build
    path = kbuild.build_variant(variant) if variant in kbuild.DEV_VARIANTS else variant_path(variant)
    layer, mk = _layer(build), MonoKernel(path)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=0.5)
    emap = synth.expert_map(spec, 0, 256 // local, device=DEV) if local != 256 else None
    if T == 8192:
        batch["logits"][:, :local] += 50.0
    kw = {}
    if shared:
        sh = layer["shared"]
        kw = {"shared": prepare_shared_expert(sh["w13"], sh["w13_scale"], sh["w2"], sh["w2_scale"], sh["gate"]),
              "shared_part": (0, 256 // local), "out_scale": spec.routed_scaling}
    needed = mk._int_symbol("prof_offset") + 148 * 64 * 8
    ns = mk._int_symbol("phase_ns_offset") + 6 * 8        # time stamp between the halves of the split form
    outs, ran = [], []
    for small in (False, True):
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        if small:
            sc["workspace"] = sc["workspace"][:needed]
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8,
                        True, layer["bias"], out, expert_map=emap, scratch=sc, check=True, **kw)
        outs.append(out.view(torch.int16))
        ran.append(int(sc["workspace"][ns:ns + 8].view(torch.int64)[0]) != 0)
    assert ran == [True, False]
    assert torch.equal(outs[0], outs[1])
    assert bool(torch.isfinite(outs[0].view(torch.bfloat16).float()).all())
