"""GPU: an MSA row whose keys are all dropped keeps what it holds to itself.

Padding rows may hold anything: memory that was never written, an overflow.  Their scores are replaced by constants, so
dS of such a row is zero whatever its Q, K, V and dO are, and d(pair_bias), which all rows of a (b,h) share, and the
gradients of the other rows do not see it.  The fp64 oracle says which values stay finite; the tolerance is that of the
parity tests.
"""
import pytest
import torch

from helpers import NAMES, REL_TOL
from oracle import evo_oracle as oc
from test_parity_gpu import _lib, rand_inputs, run_op

pytestmark = pytest.mark.gpu

ROWS = (1, 4)  # of five: a whole row group of three, a short one, and items of one row


def poisoned(D, name, value, frozen=False, R=203, S=5):
    x = rand_inputs(1, S, R, 2, D, torch.bfloat16, seed=D + R, mask="bool", bias=True)
    if frozen:
        x["pair_bias"] = None
    for s in ROWS:
        x["res_mask"][:, s] = False
        rows = oc.kernel_view(x[name])[:, :, s]
        if value == "nan":
            rows.fill_(float("nan"))
        else:  # one value of the first, of a middle and of the last residue
            rows[..., [0, R // 2, R - 1], D - 1] = float("inf")
    return x


def finite_values_agree(got, x):
    exact = oc.attention_fwd_bwd_explicit(x["Q"], x["K"], x["V"], x["res_mask"], x["pair_bias"], x["dO"])
    for name, g, e in zip(NAMES, got, exact):
        if e is None:
            continue
        known = torch.isfinite(e)
        assert torch.isfinite(g[known]).all(), f"{name}: not finite where the exact value is"
        err = (g.double() - e)[known].abs().max() / e[known].abs().max()
        assert err <= REL_TOL[torch.bfloat16], f"{name}: {err:.2e}"
    assert exact[4] is None or torch.isfinite(exact[4]).all()


@pytest.mark.parametrize("value", ["nan", "inf"])
@pytest.mark.parametrize("name", ["Q", "K", "V", "dO"])
@pytest.mark.parametrize("D", [8, 24, 32, 64])
def test_with_a_pair_bias_gradient(D, name, value):
    x = poisoned(D, name, value)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    finite_values_agree(got, x)


@pytest.mark.parametrize("name", ["Q", "K", "V", "dO"])
@pytest.mark.parametrize("D", [16, 32, 64])
def test_without_a_pair_bias(D, name):
    x = poisoned(D, name, "nan", frozen=True, R=264)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    finite_values_agree(got, x)


@pytest.mark.parametrize("name", ["Q", "K", "V", "dO"])
def test_many_rows_above_a_head_dimension_of_32(name):
    x = poisoned(64, name, "nan", R=261, S=64)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    finite_values_agree(got, x)
