"""Partial rows in sorted order (large batches) against slot order (the same launch with a workspace that has no room for the
slots' positions): the outputs have to be the same bits, and the positions the inverse of the sort. And the units that are
left behind the full rounds: split where every CTA gets one pass of the up projection at most."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, build as kbuild, loader, synth, variant_path
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# (binary, layer, intermediate columns, local experts, shared expert), tokens, skew, residual: the smallest batch that has
# sorted rows and the largest that has not, ragged tiles, ranks that own a part of the experts, three and four blocks a box,
# intermediates too small for the last pass's box, units in chunks, the shared expert's rows behind the routed ones
CASES = [(("qwen_w1", synth.QWEN, 512, 256, False), T, skew, False) for T, skew in ((4095, 0.0), (4096, 0.0), (5003, 1.0))]
CASES += [(("qwen_w1", synth.QWEN, 512, 256, True), 4157, 0.5, True), (("qwen_tp2", synth.QWEN, 256, 256, False), 4111, 0.5, False),
          (("qwen_ep4", synth.QWEN, 512, 64, False), 11003, 1.0, False), (("ds_tp8", synth.DEEPSEEK, 256, 256, False), 4099, 0.5, False),
          (("ds_tp4", synth.DEEPSEEK, 512, 256, False), 4096, 1.0, False), (("ds_ep8", synth.DEEPSEEK, 2048, 32, True), 4133, 0.5, False)]
# a few units left behind one round or several, the shared expert's among them, chunks, more than are split, none, less than one round
CASES += [(("qwen_ep4", synth.QWEN, 512, 64, False), 8192, 0.5, False), (("qwen_ep4", synth.QWEN, 512, 64, False), 7500, 0.0, False),
          (("qwen_ep8", synth.QWEN, 512, 32, True), 18000, 0.0, False), (("qwen_ep8", synth.QWEN, 512, 32, False), 6000, 0.0, False),
          (("qwen_w1", synth.QWEN, 512, 256, False), 10000, 0.0, False), (("ds_tp8", synth.DEEPSEEK, 256, 256, False), 8192, 0.0, False),
          (("ds_ep8", synth.DEEPSEEK, 2048, 32, False), 8000, 0.0, False)]
# the most tokens that the C entries take (the Python entries have a cap of their own): 31 full rounds, and no room in the
# CTAs' lists for a part of the units behind them
CASES += [(("qwen_w1", synth.QWEN, 512, 256, False), 71680, 0.0, False)]
PASSES = {"qwen_w1": 4, "qwen_ep4": 4, "qwen_ep8": 4, "ds_tp8": 2, "ds_tp4": 4, "ds_ep8": 4}   # of a unit's up projection, where units are long


@pytest.mark.parametrize("build,T,skew,residual", CASES, ids=[f"{b[0]}{'-shared' if b[4] else ''}-{T}" for b, T, _, _ in CASES])
def test_sorted_rows_give_the_bits_of_slot_order(build, T, skew, residual, monkeypatch):
    variant, spec, width, local, shared = build
    monkeypatch.setattr(loader, "MOE_MONOKERNEL_PREFILL_MAX_TOKENS", max(T, loader.MOE_MONOKERNEL_PREFILL_MAX_TOKENS))
    mk = MonoKernel(variant_path(variant))
    layer = synth.make_layer(spec, seed=5, device=DEV, inter_slice=(0, width) if width != spec.inter else None,
                             expert_slice=(0, local) if local != 256 else None, with_shared=shared)
    batch = synth.make_batch(spec, layer, T, seed=T, device=DEV, skew=skew)
    kw = {"expert_map": synth.expert_map(spec, 0, 256 // local, device=DEV) if local != 256 else None}
    if shared:
        sh = layer["shared"]
        kw.update(shared=prepare_shared_expert(sh["w13"], sh["w13_scale"], sh["w2"], sh["w2_scale"], sh["gate"]),
                  shared_part=(0, 256 // local), out_scale=spec.routed_scaling)
    if residual:
        kw["residual"] = torch.randn(T, spec.hidden, device=DEV).to(torch.bfloat16)
    needed = mk._int_symbol("workspace_min_bytes")
    behind = -(-needed // 256) * 256
    got = []
    for small in (False, True):
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        sc["sorted_ids"].fill_(-1)
        if small:
            sc["workspace"] = sc["workspace"][:needed]
        else:
            sc["workspace"][behind:behind + T * 32].fill_(0xEE)
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8,
                        True, layer["bias"], out, scratch=sc, check=True, **kw)
        got.append((out.view(torch.int16), sc))
    (a, sc), (b, flat) = got
    assert torch.equal(a, b)
    assert bool(torch.isfinite(a.view(torch.bfloat16).float()).all())
    pos = sc["workspace"][behind:behind + T * 32].view(torch.int32)
    if T < 4096:
        assert bool((pos.view(torch.uint8) == 0xEE).all())
        return
    rows = int((sc["topk_ids"] >= 0).sum())
    here = sc["topk_ids"].flatten() >= 0
    assert bool((pos[~here] == -1).all())
    assert torch.equal(sc["sorted_ids"][pos[here].long()], here.nonzero()[:, 0].int())
    assert int(pos.max()) == rows - 1
    # units behind the full rounds: split or not
    view, chunks = mk.workspace_view(sc["workspace"]), max(width // 512, 1)
    units = view["total_tiles"] + (-(-(-(-T // 128)) // (256 // local)) * chunks if shared else 0)
    left = units % 148 if units > 148 else 0
    split = int(view["phase_ns"][6]) != 0
    if units > 148:
        room = units // 148 + 2 <= mk._int_symbol("max_tiles") // 148
        assert split == (variant in PASSES and 0 < left <= 148 // PASSES[variant] // chunks * chunks and room)
    assert int(mk.workspace_view(flat["workspace"])["phase_ns"][6]) == 0


def test_the_build_without_row_stores_measures_the_sorted_form():
    """The development build that leaves the row stores out: large batches run the sorted form there as well (the positions
    are written), and none of its row stores."""
    mk, T = MonoKernel(kbuild.build_variant("qwen_w1_abl4")), 4096
    layer = synth.make_layer(synth.QWEN, seed=5, device=DEV, with_shared=False)
    batch = synth.make_batch(synth.QWEN, layer, T, seed=T, device=DEV)
    sc = mk._allocate_scratch(T, DEV)
    behind = -(-mk._int_symbol("workspace_min_bytes") // 256) * 256
    sc["partial"].fill_(float("nan"))
    sc["workspace"][behind:].fill_(0xEE)
    out = torch.empty(T, 2048, dtype=torch.bfloat16, device=DEV)
    mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True, None,
                    out, scratch=sc, check=True)
    pos = sc["workspace"][behind:behind + T * 32].view(torch.int32)
    assert torch.equal(torch.sort(pos).values, torch.arange(T * 8, dtype=torch.int32, device=DEV))
    assert bool(sc["partial"].isnan().all())
