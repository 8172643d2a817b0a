"""GPU: the two orders in which the forward walks its items, on both sides of the rule that chooses between them (more than
four query tiles; K and V of a (b,h) below 40 MB), with short row groups, a ragged last tile and several heads and batches."""
import pytest
import torch

from helpers import REL_TOL
from oracle import evo_oracle as oc
from test_parity_gpu import DEV, _lib, rand_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    (2, 5, 512, 3, 32), (2, 5, 513, 3, 32), (1, 7, 700, 2, 8), (3, 2, 640, 1, 64), (1, 1, 900, 2, 16),
    (1, 255, 641, 1, 64), (1, 257, 641, 1, 64)], ids=lambda c: "B%dS%dR%dH%dD%d" % c)
@pytest.mark.parametrize("bias", [True, False], ids=["bias", "none"])
def test_forward(cfg, bias):
    import evoformer_triton_b200 as evo
    from evoformer_triton_b200 import attention
    x = rand_inputs(*cfg, torch.bfloat16, seed=cfg[2], mask="bool", bias=bias)
    dev = [None if x[n] is None else x[n].to(DEV) for n in ("Q", "K", "V", "res_mask", "pair_bias")]
    with torch.no_grad():
        out = evo.EvoformerAttention.apply(*dev)
    assert attention.last_path["fwd"] == _lib().PATH_TCGEN05
    evo.check_device_status()
    exact = oc.attention(*(None if x[n] is None else x[n].float() if x[n].is_floating_point() else x[n]
                           for n in ("Q", "K", "V", "res_mask", "pair_bias")))
    assert oc.rel_err(out, exact) <= REL_TOL[torch.bfloat16]
