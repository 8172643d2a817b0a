"""GPU: the backward above a head dimension of 32, where d(pair_bias) comes from a kernel of its own and dK and dV
leave by bulk stores: edges of the 128 x 128 tiles, one row and rows cut into uneven runs, a query tile and a key tile
that hold a single residue, masks of each kind, rows without a key."""
import pytest
import torch

from test_parity_gpu import DEV, _lib, check, rand_inputs, run_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    (1, 1, 129, 1, 64), (2, 3, 127, 2, 40), (1, 2, 128, 3, 48), (1, 149, 64, 1, 64), (1, 21, 257, 2, 64),
    (3, 7, 66, 1, 56)], ids=lambda c: "B%dS%dR%dH%dD%d" % c)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("mask", ["bool", "add32", "none"])
def test_d64_backward_tiles(cfg, dtype, mask):
    B, S, R, H, D = cfg
    x = rand_inputs(B, S, R, H, D, dtype, seed=R + D, mask=mask, bias=True)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    check(got, x, label=f"{cfg} {mask} ")


@pytest.mark.parametrize("D", [40, 64])
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
def test_rows_without_a_key_and_a_16_bit_bias(D, bias_dtype):
    x = rand_inputs(1, 6, 200, 2, D, torch.bfloat16, seed=D, mask="bool", bias=True)
    x["res_mask"][:, 2] = False
    x["pair_bias"] = x["pair_bias"].to(bias_dtype)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    check(got, x, label=f"D={D} ")


def test_d64_outputs_that_are_not_accumulated_are_reproducible():
    """Long items, several of them a CTA: O, dK and dV have the same bits every time, and d(pair_bias) and dQ, which are
    sums of atomics, agree to the order of fp32 sums (S terms: sqrt(S) 2^-24 of their size)."""
    x = rand_inputs(1, 150, 300, 2, 64, torch.bfloat16, seed=5, mask="bool", bias=True)
    first, second = run_op(x)[0], run_op(x)[0]
    for i in (0, 2, 3):
        assert torch.equal(first[i], second[i])
    d = (first[4].double() - second[4].double()).norm() / first[4].double().norm()
    assert d < 150 ** 0.5 * 2.0 ** -22
