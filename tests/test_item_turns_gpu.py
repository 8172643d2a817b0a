"""GPU: the backward over several items a CTA, whose dK and dV leave while the next item is under way: a partial last key
tile together with a partial last row group, in the forms with and without a d(pair_bias)."""
import pytest
import torch

from test_parity_gpu import _lib, check, rand_inputs, run_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [True, False], ids=["bias", "none"])
@pytest.mark.parametrize("D,S", [(8, 141), (24, 70), (32, 71), (40, 37)])
def test_partial_tiles_and_groups(D, S, bias):
    x = rand_inputs(1, S, 200, 8, D, torch.bfloat16, seed=D, mask="bool", bias=bias)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    check(got, x, label=f"D={D} ")
