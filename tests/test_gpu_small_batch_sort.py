"""Counts, offsets and the stable sort on both sides of the batch size up to which every CTA counts the expert ids itself,
with ids that belong to other ranks among them."""
import pytest

from unimonomoe_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 13, 255, 256, 257])
def test_sort_is_exact_around_the_direct_count(T):
    from oracle import cpu_oracle as O
    from tests import gpu_util as gu
    mk = gu.kernel("qwen_ep4")
    layer = synth.make_layer(synth.QWEN, seed=2, device=gu.DEV, expert_slice=(64, 128), with_shared=False)
    emap = synth.expert_map(synth.QWEN, 1, 4, device=gu.DEV)
    batch = synth.make_batch(synth.QWEN, layer, T, seed=T, device=gu.DEV, skew=0.5)
    res = gu.launch(mk, layer, batch, expert_map=emap)
    gu.check_routing(O, res, batch, 0, None, 64, expert_map=emap)
