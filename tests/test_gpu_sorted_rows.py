"""Partial rows in sorted order (large batches) against slot order (the same launch with a workspace that has no room for the
slots' positions): the outputs have to be the same bits, and the positions the inverse of the sort. And the units that are
left behind the full rounds: split where every CTA gets one pass of the up projection at most, a batch of less than one round
where the busiest CTA's steps are few enough, and neither where the workspace holds the positions alone."""
import pytest
import torch

from unimonomoe_b200 import MonoKernel, build as kbuild, loader, synth, variant_path
from unimonomoe_b200.loader import prepare_shared_expert

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# (binary, layer, intermediate columns, local experts, shared expert), tokens, skew, residual, units behind the full rounds
# split?: the smallest batch that has sorted rows and the largest that has not, ragged tiles, ranks that own a part of the
# experts, three and four blocks a box, intermediates too small for the last pass's box, units in chunks, the shared expert's
# rows behind the routed ones
CASES = [(("qwen_w1", synth.QWEN, 512, 256, False), 4095, 0.0, False, False), (("qwen_w1", synth.QWEN, 512, 256, False), 4096, 0.0, False, False),
         (("qwen_w1", synth.QWEN, 512, 256, False), 5003, 1.0, False, False), (("qwen_w1", synth.QWEN, 512, 256, True), 4157, 0.5, True, False),
         (("qwen_tp2", synth.QWEN, 256, 256, False), 4111, 0.5, False, False), (("qwen_ep4", synth.QWEN, 512, 64, False), 11003, 1.0, False, False),
         (("ds_tp8", synth.DEEPSEEK, 256, 256, False), 4099, 0.5, False, False), (("ds_tp4", synth.DEEPSEEK, 512, 256, False), 4096, 1.0, False, False),
         (("ds_ep8", synth.DEEPSEEK, 2048, 32, True), 4133, 0.5, False, False)]
# more units left behind one round than are split, less than one round, likewise, a few left, the shared expert's among them;
# few in less than one round, behind several, in chunks
CASES += [(("qwen_ep4", synth.QWEN, 512, 64, False), 8192, 0.5, False, False), (("qwen_ep4", synth.QWEN, 512, 64, False), 7500, 0.0, False, False),
          (("qwen_ep8", synth.QWEN, 512, 32, True), 18000, 0.0, False, True), (("qwen_ep8", synth.QWEN, 512, 32, False), 6000, 0.0, False, True),
          (("qwen_w1", synth.QWEN, 512, 256, False), 10000, 0.0, False, True), (("ds_tp8", synth.DEEPSEEK, 256, 256, False), 8192, 0.0, False, True),
          (("ds_ep8", synth.DEEPSEEK, 2048, 32, False), 8000, 0.0, False, True)]
# the most tokens that the C entries take (the Python entries have a cap of their own): 31 full rounds, and no room in the
# CTAs' lists for a part of the units behind them
CASES += [(("qwen_w1", synth.QWEN, 512, 256, False), 71680, 0.0, False, False)]
PASSES = {"qwen_w1": 4, "qwen_ep4": 4, "qwen_ep8": 4, "ds_tp8": 2, "ds_tp4": 4, "ds_ep8": 4}   # of a unit's up projection, where units are long
MOST = {"qwen_w1": 74, "qwen_ep4": 74, "qwen_ep8": 74, "ds_tp8": 74, "ds_tp4": 111, "ds_ep8": 111}   # of less than a round that are split


@pytest.mark.parametrize("build,T,skew,residual,splits", CASES, ids=[f"{c[0][0]}{'-shared' if c[0][4] else ''}-{c[1]}" for c in CASES])
def test_sorted_rows_give_the_bits_of_slot_order(build, T, skew, residual, splits, monkeypatch):
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
    positions = -(-T * 32 // 256) * 256
    got = []
    for size in (None, behind + positions, needed):   # all of it, the positions alone, neither
        sc = mk._allocate_scratch(T, DEV)
        sc["partial"].fill_(float("nan"))
        sc["sorted_ids"].fill_(-1)
        sc["workspace"][behind:behind + positions].fill_(0xEE)
        sc["workspace"] = sc["workspace"][:size]
        out = torch.full((T, spec.hidden), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8,
                        True, layer["bias"], out, scratch=sc, check=True, **kw)
        view = mk.workspace_view(sc["workspace"])
        got.append((out.view(torch.int16), sc, view["total_tiles"], int(view["phase_ns"][6]) != 0))
        sc["partial"] = None
    (a, sc, units, split), (b, some, _, some_split), (c, _, _, no_split) = got
    assert torch.equal(a, b) and torch.equal(a, c)
    assert bool(torch.isfinite(a.view(torch.bfloat16).float()).all())
    assert not no_split
    if T < 4096:
        assert all(bool((x["workspace"][behind:behind + T * 32] == 0xEE).all()) for x in (sc, some))
        return
    here = sc["topk_ids"].flatten() >= 0
    for x in (sc, some):
        pos = x["workspace"][behind:behind + T * 32].view(torch.int32)
        assert bool((pos[~here] == -1).all())
        assert torch.equal(x["sorted_ids"][pos[here].long()], here.nonzero()[:, 0].int())
        assert int(pos.max()) == int(here.sum()) - 1
    # units behind the full rounds: split or not
    chunks = max(width // 512, 1)
    units += -(-(-(-T // 128)) // (256 // local)) * chunks if shared else 0
    most = 0 if variant not in PASSES else MOST[variant] if units < 148 else 148 // PASSES[variant] // chunks * chunks
    room = units // 148 + 2 <= mk._int_symbol("max_tiles") // 148
    assert split == splits == (0 < units % 148 <= most and room)
    assert not some_split


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


def test_the_largest_batch_in_pairs_of_tiles(monkeypatch):
    """More than 32 pairs for a cluster: one ragged pair per expert behind the full ones. Same bits as the build that deals tiles."""
    T = 71680
    monkeypatch.setattr(loader, "MOE_MONOKERNEL_PREFILL_MAX_TOKENS", T)
    layer = synth.make_layer(synth.QWEN, seed=5, device=DEV, with_shared=False)
    for seed in range(40):
        batch = synth.make_batch(synth.QWEN, layer, T, seed=seed, device=DEV)
        pairs = int((torch.bincount(batch["logits"].topk(8, dim=-1).indices.flatten(), minlength=256) + 255).div(256, rounding_mode="floor").sum())
        if pairs > 32 * 74:
            break
    got = []
    for variant in ("qwen_w1_pair", "qwen_w1"):
        mk = MonoKernel(variant_path(variant))
        sc = mk._allocate_scratch(T, DEV)
        out = torch.full((T, 2048), float("nan"), dtype=torch.bfloat16, device=DEV)
        mk.prefill_impl(batch["hs"], batch["logits"], layer["w13"], layer["w13_scale"], layer["w2"], layer["w2_scale"], 8, True,
                        None, out, scratch=sc, check=True)
        got.append((out.view(torch.int16), mk.workspace_view(sc["workspace"])["total_tiles"]))
    assert got[0][1] == pairs > 32 * 74
    assert torch.equal(got[0][0], got[1][0])
    assert bool(torch.isfinite(got[0][0].view(torch.bfloat16).float()).all())
