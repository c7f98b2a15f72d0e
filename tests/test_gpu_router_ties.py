"""Routing where scores tie inside a lane's experts, between lanes and between groups, with zeros of both signs and masked
experts, and activation scales of tokens whose columns are zero, subnormal or huge: the same bits as the oracle, in every router
mode, on both sides of eight tokens (up to which every CTA routes and sorts the whole batch for itself)."""
import pytest
import torch

from unimonomoe_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,spec,width,local,mode", [("qwen_ep8", synth.QWEN, 512, 32, 0), ("qwen_sig_w1", synth.QWEN, 512, 256, 1),
                                                           ("ds_tp8", synth.DEEPSEEK, 256, 256, 2)])
@pytest.mark.parametrize("T", [1, 8, 9, 149, 300])
def test_ties_and_extremes_are_exact(variant, spec, width, local, mode, T):
    from oracle import cpu_oracle as O
    from tests import gpu_util as gu
    mk, g = gu.kernel(variant), torch.Generator().manual_seed(T)
    layer = synth.make_layer(spec, seed=4, device=gu.DEV, inter_slice=(0, width) if width != spec.inter else None,
                             expert_slice=(0, local) if local != 256 else None, with_shared=False)
    emap = synth.expert_map(spec, 0, 256 // local, device=gu.DEV) if local != 256 else None
    logits = torch.randint(-3, 4, (T, 256), generator=g).float() * 0.5     # seven values: about 36 experts carry each
    logits[logits == 0] *= torch.where(torch.rand(int((logits == 0).sum()), generator=g) < 0.5, -1.0, 1.0)
    logits[::3] = torch.where(torch.rand(logits[::3].shape, generator=g) < 0.7, -torch.inf, logits[::3])
    logits[::3, ::16] = 2.0                                                # at least 16 selectable, two in every group
    hs = torch.randn(T, spec.hidden, generator=g).to(torch.bfloat16)
    hs[0, :128], hs[0, 128:256], hs[0, 256:384] = 0.0, 1e-39, 3e38
    hs[-1, -128:] = -0.0
    layer["bias"] = None if mode == 0 else (torch.randint(0, 3, (256,), generator=g).float() * 0.25).to(gu.DEV)
    batch = {"hs": hs.to(gu.DEV), "logits": logits.to(gu.DEV)}
    res = gu.launch(mk, layer, batch, expert_map=emap)
    gu.check_routing(O, res, batch, mode, layer["bias"], local, expert_map=emap)
    gu.check_act_quant(O, res, batch)
