"""GPU: above a head dimension of 32 d(pair_bias) comes from the kernel that gives dQ, dK and dV where there are few MSA
rows or at most two tiles of residues, and from a kernel of its own above: both sides of the rule, at the edges of the
tiles, with items that follow one another in a CTA, each type of bias, each layout of its gradient."""
import pytest
import torch

from oracle import evo_oracle as oc
from test_parity_gpu import DEV, _lib, check, rand_inputs, run_op

pytestmark = pytest.mark.gpu

FEW, MANY = 3, 4  # launches of a backward: first pass, kernel, (d(pair_bias),) dQ store


@pytest.mark.parametrize("cfg,launches", [
    ((1, 1, 64, 1, 64), FEW), ((4, 1, 300, 3, 64), FEW), ((1, 3, 516, 2, 40), FEW), ((1, 150, 256, 1, 64), FEW),
    ((1, 63, 260, 1, 64), FEW), ((1, 64, 260, 1, 64), MANY), ((2, 65, 388, 1, 48), MANY), ((1, 39, 516, 1, 56), MANY)],
    ids=lambda c: "B%dS%dR%dH%dD%d" % c if isinstance(c, tuple) else str(c))
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("mask", ["bool", "add32"])
def test_both_sides_of_the_rule(cfg, launches, bias_dtype, mask):
    from evoformer_triton_b200 import attention
    B, S, R, H, D = cfg
    x = rand_inputs(B, S, R, H, D, torch.bfloat16, seed=S + R, mask=mask, bias=True)
    x["pair_bias"] = x["pair_bias"].to(bias_dtype)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    assert attention.launches["bwd"] == launches + (bias_dtype != torch.float32)  # (the conversion)
    check(got, x, chunk=32, label=f"{cfg} ")


@pytest.mark.parametrize("cfg", [(1, 2, 203, 2, 64), (1, 66, 261, 1, 64)], ids=["few", "many"])
def test_heads_last_in_16_bits_at_an_odd_length(cfg):
    import evoformer_triton_b200 as evo
    B, S, R, H, D = cfg
    x = rand_inputs(B, S, R, H, D, torch.bfloat16, seed=R, mask="bool", bias=True)
    brrh = x["pair_bias"].reshape(B, H, R, R).permute(0, 2, 3, 1).contiguous().bfloat16()
    want = oc.extended_attention_fwd_bwd(x["Q"], x["K"], x["V"], x["res_mask"], brrh, x["dO"], pair_bias_layout="brrh",
                                         upcast=torch.float32)
    q, k, v, b = (t.to(DEV).requires_grad_() for t in (x["Q"], x["K"], x["V"], brrh))
    out = evo.evoformer_attention(q, k, v, [x["res_mask"].to(DEV), b], layout="reinterpret", pair_bias_layout="brrh")
    out.backward(x["dO"].to(DEV))
    evo.check_device_status()
    for name, g, e in zip("O dQ dK dV d_pair_bias".split(), (out, q.grad, k.grad, v.grad, b.grad), want):
        assert oc.rel_err(g, e) <= 1e-2, name


def test_tiles_that_follow_one_another_in_a_cta():
    """180 tiles of d(pair_bias) and 33 rows in uneven runs, several items for every SM.  Run twice, d(pair_bias) and dQ, sums
    of atomics, agree to the order of fp32 sums (sqrt(terms) 2^-24 of their size), dQ to that and its rounding to bf16."""
    x = rand_inputs(1, 33, 650, 5, 64, torch.bfloat16, seed=7, mask="bool", bias=True)
    (o, dq, dk, dv, db), _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    _, dq2, dk2, dv2, db2 = run_op(x)[0]
    check((o, dq, dk, dv, db), x, chunk=11, label="180 tiles ")
    assert torch.equal(dk, dk2) and torch.equal(dv, dv2)
    assert (db.double() - db2.double()).norm() <= 33 ** 0.5 * 2.0 ** -22 * db.double().norm()
    a, b = dq.float(), dq2.float()
    assert ((a - b).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), b.abs()) + 2.0 ** -18 * a.abs().max()).all()
