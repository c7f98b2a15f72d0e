"""The split form of the expert phase (units cut into passes, dealt over all SMs in two halves) against whole units (the
same launch with a workspace that has no room for the split intermediate): the outputs have to be the same bits,
because every row sees the same operations in the same order. And which of the two a batch gets: the units decide that
there are, not those that even routing of as many tokens would give."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, build as kbuild, synth, variant_path
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# more than 64 K slabs: a lane holds the weight scales of three of them
WIDE = synth.LayerSpec("wide", hidden=9216, inter=256)

# build: (binary, layer, intermediate columns, local experts, shared expert). A case: build, tokens, skew, where the
# tokens go (None: as the router says; "apart": each to eight experts of its own; otherwise
# (n, the experts of the first n tokens, the experts of the others)).
# Fewer passes than SMs, about one round of units and (even routing) somewhat more than one, ragged and full tiles, the
# shared expert's tiles, units in chunks
W1, SHARED = ("qwen_w1", synth.QWEN, 512, 256, False), ("qwen_w1", synth.QWEN, 512, 256, True)
CASES = [(W1, T, 0.5, None) for T in (1, 2, 9)] + [(W1, 32, 0.0, None)]
CASES += [(("qwen_tp2", synth.QWEN, 256, 256, False), T, 0.5, None) for T in (1, 3)]
CASES += [(("qwen_ep4", synth.QWEN, 512, 64, False), T, 0.5, None) for T in (9, 257)]
CASES += [(SHARED, 3, 0.5, None), (SHARED, 32, 0.0, None)]
CASES += [(("ds_tp8", synth.DEEPSEEK, 256, 256, False), T, 0.5, None) for T in (1, 4)]
CASES += [(("ds_ep8", synth.DEEPSEEK, 2048, 32, True), T, 0.5, None) for T in (8, 20)]
CASES += [(("wide_ep8", WIDE, 256, 32, False), T, 0.5, None) for T in (3, 16)]
# from 4096 tokens on: whole units, and those behind the full round of 148 split, the shared expert's among them
CASES += [(("qwen_ep8", synth.QWEN, 512, 32, True), 18000, 0.0, None)]
# two waves of units through the intermediate: more rows than it holds. 2600 of the tokens on eight local experts: 168 units
# with 20800 of the 18944 rows that it has room for, and the shared expert's 13 units at the end of the second wave; and units
# in chunks (2600 of the tokens on two local experts: 42 tiles)
CASES += [(("qwen_ep2", synth.QWEN, 512, 128, True), 3300, 0.0,
           (2600, (1, 17, 40, 41, 77, 78, 100, 101), (130, 150, 170, 190, 200, 210, 220, 230)))]
CASES += [(("ds_ep8", synth.DEEPSEEK, 2048, 32, False), 3200, 0.0,
           (2600, (3, 17, 40, 41, 77, 78, 100, 101), (40, 41, 77, 78, 100, 101, 130, 131)))]
_layers = {}


def _layer(build):
    if build not in _layers:
        _layers.clear()   # one layer on the GPU at a time
        variant, spec, width, local, shared = build
        _layers[build] = synth.make_layer(
            spec, seed=21, device=DEV, inter_slice=(0, width) if width != spec.inter else None,
            expert_slice=(0, local) if local != 256 else None, with_shared=shared)
    return _layers[build]


def _run(build, T, skew, experts=None):
    """One launch with the intermediate and one without room for it: (output bits, split?, units) each."""
    variant, spec, width, local, shared = build
    path = kbuild.build_variant(variant) if variant in kbuild.DEV_VARIANTS else variant_path(variant)
    layer, mk = _layer(build), MonoKernel(path)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=skew)
    if experts is not None:
        batch["logits"] -= 50.0
        if experts == "apart":
            for t in range(T):
                batch["logits"][t, 8 * t:8 * t + 8] += 100.0
    if isinstance(experts, tuple):
        n, first, others = experts
        batch["logits"][:n, list(first)] += 100.0
        batch["logits"][n:, list(others)] += 100.0
    emap = synth.expert_map(spec, 0, 256 // local, device=DEV) if local != 256 else None
    kw = {}
    if shared:
        sh = layer["shared"]
        kw = {"shared": prepare_shared_expert(sh["w13"], sh["w13_scale"], sh["w2"], sh["w2_scale"], sh["gate"]),
              "shared_part": (0, 256 // local), "out_scale": spec.routed_scaling}
    needed = mk._int_symbol("workspace_min_bytes")
    ns = mk._int_symbol("phase_ns_offset") + 6 * 8        # time stamp between the halves of the split form
    got = []
    for small in (False, True):
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        if small:
            sc["workspace"] = sc["workspace"][:needed]
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8,
                        True, layer["bias"], out, expert_map=emap, scratch=sc, check=True, **kw)
        got.append((out.view(torch.int16), int(sc["workspace"][ns:ns + 8].view(torch.int64)[0]) != 0,
                    mk.workspace_view(sc["workspace"])["total_tiles"]))
    return got


@pytest.mark.parametrize("build,T,skew,experts", CASES, ids=[f"{b[0]}{'-shared' if b[4] else ''}-{T}" for b, T, _, _ in CASES])
def test_split_units_give_the_bits_of_whole_units(build, T, skew, experts):
    (a, a_split, units), (b, b_split, _) = _run(build, T, skew, experts)
    assert (a_split, b_split) == (True, False)
    assert not isinstance(experts, tuple) or units > 148
    assert torch.equal(a, b)
    assert bool(torch.isfinite(a.view(torch.bfloat16).float()).all())


def test_the_time_stamp_tells_which_form_ran():
    """Two launches on one workspace: the second computes whole units and must not keep the first one's time stamp."""
    layer, mk = _layer(W1), MonoKernel(variant_path("qwen_w1"))
    sc = mk._allocate_scratch(16, DEV)
    seen = []
    for T in (1, 16, 1):
        batch = synth.make_batch(synth.QWEN, layer, T, seed=T, device=DEV)
        out = torch.empty(T, 2048, dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8,
                        True, None, out, scratch=sc, check=True)
        seen.append(int(mk.workspace_view(sc["workspace"])["phase_ns"][6]) != 0)
    assert seen == [True, False, True]


# 148 units fill one round of whole units, in which splitting does not pay from about 75 on (where a unit is long, H =
# 7168 and 512 columns, from 112 on, and with a few rows a tile it pays throughout): up to there, and from 149 to about 203,
# the split form. 32 tokens reach 169 experts at even routing, 124 at skew 0.5, 69 at skew 1.0. From 4096 tokens on whole
# units fill the round, and up to 37 behind it are split: 149 to 185.
EP2, EP4, TP4 = ("qwen_ep2", synth.QWEN, 512, 128, False), ("qwen_ep4", synth.QWEN, 512, 64, False), ("ds_tp4", synth.DEEPSEEK, 512, 256, False)
CHOICES = [(W1, 32, 0.0, None, (149, 203), True), (W1, 32, 0.5, None, (76, 148), False), (W1, 32, 1.0, None, (1, 74), True),
           (W1, 16, 0.0, None, (76, 148), False), (EP4, 7500, 0.0, None, (76, 148), False),
           (EP2, 3850, 0.0, None, (149, 203), True), (EP4, 8192, 0.0, None, (149, 185), True),
           (EP4, 10200, 0.0, None, (186, 203), False), (TP4, 12, 0.0, "apart", (96, 96), True),
           (TP4, 28, 0.5, None, (112, 148), True), (W1, 9, 0.0, "apart", (72, 72), True)]


@pytest.mark.parametrize("build,T,skew,experts,between,splits", CHOICES, ids=[f"{c[0][0]}-{c[1]}-{c[3] or c[2]}" for c in CHOICES])
def test_the_units_of_the_batch_decide(build, T, skew, experts, between, splits):
    (a, a_split, units), (b, b_split, _) = _run(build, T, skew, experts)
    assert between[0] <= units <= between[1]
    assert (a_split, b_split) == (splits, False)
    assert torch.equal(a, b)
