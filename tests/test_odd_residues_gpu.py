"""GPU: any number of residues on the tensor-core path.  A pair bias whose rows are not whole 16-byte
pieces is read from a padded copy and its gradient is summed in one; the sizes are the edges of the
128-wide tiles and every remainder of a 16-byte row."""
import pytest
import torch

from test_parity_gpu import DEV, _lib, check, rand_inputs, run_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias_dtype", ["fp32", "same"])
@pytest.mark.parametrize("cfg", [
    (2, 5, 127, 2, 32, torch.bfloat16, "bool"), (1, 7, 129, 3, 32, torch.float16, "add32"),
    (1, 4, 203, 2, 32, torch.bfloat16, "bool"), (1, 3, 257, 1, 64, torch.bfloat16, "addsame"),
    (2, 1, 302, 4, 64, torch.bfloat16, "none"), (1, 9, 70, 4, 8, torch.float16, "bool"),
    (8192, 1, 5, 9, 8, torch.bfloat16, "none")],  # more (b, h) than a grid has rows
    ids=lambda c: "B%dS%dR%dH%dD%d-%s-%s" % (*c[:5], str(c[5]).split(".")[-1], c[6]))
def test_any_number_of_residues(cfg, bias_dtype):
    B, S, R, H, D, dtype, mask = cfg
    x = rand_inputs(B, S, R, H, D, dtype, seed=R + D, mask=mask)
    if bias_dtype == "same":
        x["pair_bias"] = x["pair_bias"].to(dtype)
    got, paths = run_op(x)
    assert paths == (_lib().PATH_TCGEN05, _lib().PATH_TCGEN05)
    check(got, x, label=f"{cfg} {bias_dtype} ")


def test_heads_last_bias_of_odd_length():
    import evoformer_triton_b200 as evo
    from oracle import evo_oracle as oc
    B, S, R, H, D = 1, 3, 141, 4, 32
    x = rand_inputs(B, S, R, H, D, torch.bfloat16, seed=5)
    brrh = x["pair_bias"].reshape(B, H, R, R).permute(0, 2, 3, 1).contiguous().bfloat16()
    want = oc.extended_attention_fwd_bwd(x["Q"], x["K"], x["V"], x["res_mask"], brrh, x["dO"], pair_bias_layout="brrh",
                                         upcast=torch.float32)
    q, k, v, b = (t.to(DEV).requires_grad_() for t in (x["Q"], x["K"], x["V"], brrh))
    out = evo.evoformer_attention(q, k, v, [x["res_mask"].to(DEV), b], layout="reinterpret", pair_bias_layout="brrh")
    out.backward(x["dO"].to(DEV))
    torch.cuda.synchronize()
    evo.check_device_status()
    for g, e in zip((out, q.grad, k.grad, v.grad, b.grad), want):
        assert oc.rel_err(g, e) < 1e-2
