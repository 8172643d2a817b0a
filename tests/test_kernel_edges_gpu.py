"""GPU: the places where the kernels' tiling, splitting and dispatch can go wrong, against the oracle:
edges of the CUDA-core tiles and of the runs of MSA rows that share a partial d(pair_bias), the forward's
rescaling of an output that is accumulated in tensor memory, key tiles that skip the mask arithmetic, and
d(pair_bias) leaving in each type and layout."""
import pytest
import torch

from oracle import evo_oracle as oc
from test_parity_gpu import DEV, _lib, check, rand_inputs, run_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [
    (1, 1, 1, 1, 8), (2, 3, 63, 2, 16), (1, 2, 64, 2, 32), (1, 37, 65, 2, 32), (1, 5, 129, 1, 64),
    (1, 3, 130, 2, 100), (1, 2, 70, 1, 128), (1, 700, 40, 1, 7)], ids=lambda c: "B%dS%dR%dH%dD%d" % c)
@pytest.mark.parametrize("mask,bias", [("bool", True), ("add32", True), ("none", False)])
def test_cuda_core_tiles_fp32(cfg, mask, bias):
    B, S, R, H, D = cfg
    x = rand_inputs(B, S, R, H, D, torch.float32, seed=R + D, mask=mask, bias=bias)
    got, paths = run_op(x)
    assert paths == (_lib().PATH_GENERIC, _lib().PATH_GENERIC)
    if R == 1:  # one key: P = 1, every score gradient is rounding noise around 0
        assert torch.equal(got[0], x["V"]) or not x["res_mask"].any()
        return
    check(got, x, label=f"{cfg} {mask} ")


def test_cuda_core_backward_is_reproducible_over_runs_of_rows():
    x = rand_inputs(1, 90, 72, 2, 24, torch.float32, seed=2)
    a, b = run_op(x)[0], run_op(x)[0]
    assert all(torch.equal(u, v) for u, v in zip(a, b))


@pytest.mark.parametrize("D,dtype,S", [(8, torch.float16, 3), (32, torch.bfloat16, 2), (64, torch.bfloat16, 1)])
def test_running_maximum_that_keeps_growing(D, dtype, S):
    """Scores that rise from key tile to key tile by far more than the forward lets the running maximum lag,
    by less than that, and that fall again; the rows start with a tile whose keys are all dropped."""
    R = 448
    x = rand_inputs(1, S, R, 2, D, dtype, seed=D, keep_p=0.9)
    ramp = torch.cat([torch.full((64,), float(v)) for v in (0, 3, 7, 30, 31, 60, 10)])
    x["pair_bias"] = x["pair_bias"] * 0.5 + ramp
    x["res_mask"][..., :64] = False
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    check(got, x, label=f"ramp D={D} ")


@pytest.mark.parametrize("S", [1, 3])
@pytest.mark.parametrize("D", [8, 32, 64])
@pytest.mark.parametrize("dtype,bits", [(torch.float16, 8.5), (torch.float16, 9.5), (torch.float16, 14), (torch.float16, 17),
                                        (torch.bfloat16, 25.5), (torch.bfloat16, 33), (torch.bfloat16, 140)])
def test_maximum_that_lags_as_far_as_it_may(dtype, bits, D, S):
    """Key tiles whose scores lie just below and just beyond what the exponentials against the maximum of the tiles
    before can take (2^15 and 2^32 in a tile's sum), one such rise after another, then a level stretch; in one query of
    32, and in all.  The bound is what rounding P and O to the storage type gives (twice eps / 2)."""
    from evoformer_triton_b200 import attention, check_device_status
    B, H, R = 1, 2, 640
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v = (torch.randn((B, H, S, R, D), generator=g, device=DEV).to(dtype) * 0.25 for _ in range(3))
    steps = torch.tensor([0, 1, 2, 2, 2, 3, 1, 4, 4, 5.]) * bits * 0.6931472
    bias = torch.randn((B, H, R, R), generator=g, device=DEV) * 0.1
    bias[:, :, :256] += steps.repeat_interleave(64).to(DEV)
    bias[:, :, 256::32] += steps.repeat_interleave(64).to(DEV)
    o, lse = attention.attention_forward(q, k, v, None, bias, D ** -0.5)
    torch.cuda.synchronize()
    check_device_status()
    assert attention.last_path["fwd"] == _lib().PATH_TCGEN05
    x = (q.double() @ k.double().transpose(-1, -2)) * D ** -0.5 + bias.double()[:, :, None]
    want = x.softmax(-1) @ v.double()
    assert (o.double() - want).norm() <= torch.finfo(dtype).eps * want.norm()
    want_lse = x.logsumexp(-1)  # (scores up to 490: half a unit in the last place of such a float is 1.5e-5)
    assert ((lse.double() - want_lse).abs() <= 1e-5 + 2.0 ** -23 * want_lse.abs()).all()


@pytest.mark.parametrize("S,D,dtype", [(64, 64, torch.bfloat16), (64, 64, torch.float16), (128, 32, torch.bfloat16)])
@pytest.mark.parametrize("kind", ["rises", "jumps", "dropped rows"])
def test_forward_takes_drifting_scores_in_its_stride(kind, S, D, dtype):
    """A bias that rises along the keys by 8 bits, one that jumps by 7 once, and rows that the mask drops whole cost
    what independent scores cost: 1.00 to 1.05 as measured, 1.5 to 2 where every tile pays for a second pass."""
    from evoformer_triton_b200 import attention, check_device_status
    B, H, R = 1, 8, 768
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v = (torch.randn((B, H, S, R, D), generator=g, device=DEV).to(dtype) * 0.5 for _ in range(3))
    flat = torch.randn((B, H, R, R), generator=g, device=DEV)
    j = torch.arange(R, device=DEV)
    drift = {"rises": flat + j / R * 8 * 0.6931472, "jumps": flat + (j > 76) * 7 * 0.6931472, "dropped rows": flat}[kind]
    mask = torch.zeros((B, S, R), device=DEV)
    mask[:, :, 700:] = -1e9
    other = mask.clone()
    if kind == "dropped rows":
        other[:, ::4] = -1e9

    def time(bias, m):
        best = float("inf")
        for _ in range(9):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(5):
                attention.attention_forward(q, k, v, m, bias, D ** -0.5)
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]))
        return best

    base, got = time(flat, mask), time(drift, other)
    check_device_status()
    assert got < 1.25 * base, (base, got)


@pytest.mark.parametrize("S", [1, 5])
@pytest.mark.parametrize("D", [8, 32, 64])
@pytest.mark.parametrize("dtype,drop", [(torch.float16, -1e9), (torch.float16, -6e4), (torch.float16, -3e38), (torch.bfloat16, -1e9),
                                        (torch.bfloat16, -2e9), (torch.bfloat16, -1e30)])
def test_rows_that_an_additive_mask_drops_whole(dtype, drop, D, S):
    """Scores near the mask's value, where a float has no bits left for the rest: those that come out equal have equal
    probabilities, as a softmax in fp32 gives them, and a row whose first keys are dropped so goes on to its others.
    The bound is what rounding P and O to the storage type gives (twice eps / 2)."""
    from evoformer_triton_b200 import attention, check_device_status
    B, H, R = 2, 2, 200
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v = (torch.randn((B, H, S, R, D), generator=g, device=DEV).to(dtype) for _ in range(3))
    bias = torch.randn((B, H, R, R), generator=g, device=DEV)
    mask = torch.zeros((B, S, R), device=DEV)
    mask[0, 0] = drop
    mask[1, S - 1, :150] = drop
    o, lse = attention.attention_forward(q, k, v, mask, bias, D ** -0.5)
    torch.cuda.synchronize()
    check_device_status()
    assert attention.last_path["fwd"] == _lib().PATH_TCGEN05
    x = (q.double() @ k.double().transpose(-1, -2)) * D ** -0.5 + bias.double()[:, :, None]
    x = (x.float() + mask[:, None, :, None, :]).double()  # (the sum with the mask is rounded to a float, the rest is not)
    want = x.softmax(-1) @ v.double()
    for b, s in ((0, 0), (1, S - 1)):
        w = want[b, :, s]
        assert (o[b, :, s].double() - w).norm() <= torch.finfo(dtype).eps * w.norm(), (b, s)
    assert (o.double() - want).norm() <= torch.finfo(dtype).eps * want.norm()


@pytest.mark.parametrize("S", [1, 5])
@pytest.mark.parametrize("D", [8, 32, 64])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mask", ["none", "bool", "add32"])
def test_queries_whose_bias_lies_far_out(mask, dtype, D, S):
    """The same for a pair bias that drops (or lifts) all keys of some queries, next to ordinary ones, ones whose first
    keys only are so, and ones at the lowest float, which count as dropped."""
    from evoformer_triton_b200 import attention, check_device_status
    B, H, R = 1, 2, 200
    g = torch.Generator(device=DEV).manual_seed(D)
    q, k, v = (torch.randn((B, H, S, R, D), generator=g, device=DEV).to(dtype) for _ in range(3))
    bias = torch.randn((B, H, R, R), generator=g, device=DEV)
    lowest = torch.finfo(torch.float32).min
    for i, far in ((3, -1e9), (4, lowest), (70, 1e9), (71, -2e9), (130, -1e30), (199, -1e9)):
        bias[:, :, i] = far
    bias[:, :, 140, :100] = -1e9
    bias[:, :, 141, 64:] = 3e9
    keep = torch.rand((B, S, R), generator=g, device=DEV) < 0.9
    m = {"none": None, "bool": keep, "add32": torch.where(keep, 0.0, -1e9)}[mask]
    o, lse = attention.attention_forward(q, k, v, m, bias, D ** -0.5)
    torch.cuda.synchronize()
    check_device_status()
    assert attention.last_path["fwd"] == _lib().PATH_TCGEN05
    x = ((q.double() @ k.double().transpose(-1, -2)) * D ** -0.5 + bias.double()[:, :, None]).float()
    if mask == "bool":
        x = torch.where(m[:, None, :, None, :], x, lowest)
    elif mask == "add32":
        x = x + m[:, None, :, None, :]
    want = x.clamp(min=lowest).double().softmax(-1) @ v.double()
    assert (o.double() - want).norm() <= torch.finfo(dtype).eps * want.norm()
    for i in (3, 4, 70, 71, 130, 140, 141, 199):
        assert (o[:, :, :, i].double() - want[:, :, :, i]).norm() <= torch.finfo(dtype).eps * want[:, :, :, i].norm(), i


@pytest.mark.parametrize("mask", ["bool", "add32", "addsame"])
@pytest.mark.parametrize("D", [16, 32, 64])
def test_mask_that_touches_some_key_tiles(mask, D):
    x = rand_inputs(1, 3, 328, 2, D, torch.bfloat16, seed=D, mask=mask, keep_p=1.1)
    drop = torch.tensor([70, 71, 319])
    if mask == "bool":
        x["res_mask"][..., drop] = False
    else:
        x["res_mask"][..., drop] = torch.tensor([-1e9, 1.5, -2.0]).to(x["res_mask"].dtype)
    got, _ = run_op(x, want_path=_lib().PATH_TCGEN05)
    check(got, x, label=f"{mask} D={D} ")


@pytest.mark.parametrize("layout", ["b1hrr", "brrh"])
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16, torch.float64])
@pytest.mark.parametrize("R", [96, 130])
def test_pair_bias_gradient_in_its_type_and_layout(layout, bias_dtype, R):
    import evoformer_triton_b200 as evo
    B, S, H, D = 2, 4, 3, 32
    x = rand_inputs(B, S, R, H, D, torch.bfloat16, seed=R)
    x["pair_bias"] = x["pair_bias"].bfloat16().float()
    want = oc.attention_fwd_bwd(x["Q"], x["K"], x["V"], x["res_mask"], x["pair_bias"], x["dO"], upcast=torch.float32)[4]
    bias = x["pair_bias"].to(bias_dtype)
    if layout == "brrh":
        bias = bias.reshape(B, H, R, R).permute(0, 2, 3, 1).contiguous()
    q, k, v, b = (t.to(DEV).requires_grad_() for t in (x["Q"], x["K"], x["V"], bias))
    out = evo.evoformer_attention(q, k, v, [x["res_mask"].to(DEV), b], layout="reinterpret", pair_bias_layout=layout)
    out.backward(x["dO"].to(DEV))
    torch.cuda.synchronize()
    evo.check_device_status()
    assert b.grad.dtype == bias_dtype and b.grad.shape == bias.shape
    got = b.grad if layout == "b1hrr" else b.grad.permute(0, 3, 1, 2).reshape(B, 1, H, R, R)
    assert oc.rel_err(got, want) < 1e-2


@pytest.mark.parametrize("cfg", [
    (1, 63, 200, 8, 8, torch.bfloat16, "bool", "fp32", False), (1, 60, 200, 8, 16, torch.float16, "add32", "same", False),
    (2, 14, 400, 8, 8, torch.bfloat16, "addsame", "none", False), (2, 13, 397, 8, 16, torch.bfloat16, "bool", "same", True),
    (1, 120, 130, 8, 16, torch.float16, "none", "fp32", False)],
    ids=lambda c: "B%dS%dR%dH%dD%d-%s-%s-%s%s" % (*c[:5], str(c[5]).split(".")[-1], c[6], c[7], "-gate" if c[8] else ""))
def test_items_of_seven_rows(cfg):
    """Head dimensions up to 16 with enough MSA rows for work items of seven: types, masks, biases, a gate, row groups
    that are not full, residues that do not fill a tile, one and two items to a block."""
    import evoformer_triton_b200 as evo
    from evoformer_triton_b200 import attention
    B, S, R, H, D, dtype, mask, bias, gated = cfg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    steps = lambda G: -(-B * H * -(-R // 128) * -(-S // G) // sms) * G  # noqa: E731
    assert 25 * steps(7) <= 26 * steps(3)  # the launcher's condition: these sizes do take seven rows
    x = rand_inputs(B, S, R, H, D, dtype, seed=S + R, mask=mask, bias=bias != "none", keep_p=0.85)
    if bias == "same":
        x["pair_bias"] = x["pair_bias"].to(dtype)
    gate = torch.randn(x["Q"].shape, generator=torch.Generator().manual_seed(1)).to(dtype) if gated else None
    want = oc.extended_attention_fwd_bwd(x["Q"], x["K"], x["V"], x["res_mask"], x["pair_bias"], x["dO"], gate=gate,
                                         upcast=torch.float32)
    t = {n: None if v is None else v.to(DEV) for n, v in dict(x, gate=gate).items()}
    wrt = [t[n].requires_grad_() for n in ("Q", "K", "V", "pair_bias", "gate") if t[n] is not None]
    out = evo.evoformer_attention(t["Q"], t["K"], t["V"], [t["res_mask"], t["pair_bias"]], layout="reinterpret", gate=t["gate"])
    grads = torch.autograd.grad(out, wrt, t["dO"])
    torch.cuda.synchronize()
    evo.check_device_status()
    assert attention.last_path["bwd"] == _lib().PATH_TCGEN05
    want = [w for w, n in zip(want[1:6], ("Q", "K", "V", "pair_bias", "gate")) if t[n] is not None]
    for g, w in zip(grads, want):
        assert oc.rel_err(g, w) < 1e-2


def test_pair_bias_gradient_of_64_gib():
    """d(pair_bias) of 2^34 values: its clearing in the backward's first pass counts beyond 32 bits.  The buffer
    holds a marker before the call; a (b, h) slab that was not cleared would keep it."""
    from evoformer_triton_b200 import attention, check_device_status
    B, H, S, R, D = 512, 8, 1, 2048, 8
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 110 << 30:
        pytest.skip("needs 64 GiB for the gradient and 32 GiB for the bias")
    g = torch.Generator(device=DEV).manual_seed(8)
    q, k, v, d_o = (torch.randn((B, H, S, R, D), generator=g, device=DEV).bfloat16() for _ in range(4))
    q *= 0.25  # (no probability comes near 1, so no score gradient comes near the marker)
    bias = torch.zeros((B, H, R, R), dtype=torch.bfloat16, device=DEV)
    dbias = torch.full((B, H, R, R), 7.0, device=DEV)
    o, lse = attention.attention_forward(q, k, v, None, bias, D ** -0.5)
    attention.attention_backward(q, k, v, o, lse, None, bias, D ** -0.5, d_o, dbias_out=dbias)
    torch.cuda.synchronize()
    check_device_status()
    assert attention.last_path["bwd"] == _lib().PATH_TCGEN05
    for b, h in ((0, 0), (171, 3), (B - 1, H - 1)):
        one = [t[b:b + 1, h:h + 1].contiguous() for t in (q, k, v, o, lse, bias, d_o)]
        want = attention.attention_backward(*one[:5], None, one[5], D ** -0.5, one[6])[3]
        assert torch.equal(dbias[b, h], want[0, 0]), (b, h)  # (one row: one addition to each element)
    low, high = torch.aminmax(dbias)
    assert -3.5 < low.item() and high.item() < 3.5  # no marker left anywhere
    del bias, dbias
    torch.cuda.empty_cache()


@pytest.mark.parametrize("cfg", [
    # rows in an item (0: query pairs), B, S, R, H, D, dtype, mask, bias
    (4, 1, 594, 72, 8, 32, torch.bfloat16, "bool", "fp32"), (4, 1, 595, 40, 8, 8, torch.float16, "add32", "same"),
    (4, 2, 296, 65, 8, 16, torch.bfloat16, "none", "none"), (3, 1, 100, 136, 4, 32, torch.float16, "addsame", "same"),
    (3, 1, 592, 64, 8, 64, torch.bfloat16, "bool", "fp32"), (3, 1, 590, 40, 8, 48, torch.bfloat16, "add32", "same"),
    (2, 1, 5, 200, 3, 32, torch.bfloat16, "bool", "same"), (2, 3, 1, 100, 2, 64, torch.float16, "none", "fp32"),
    (0, 2, 1, 272, 3, 32, torch.bfloat16, "addsame", "fp32"), (0, 2, 1, 520, 2, 64, torch.float16, "bool", "same"),
    (0, 2, 1, 264, 3, 16, torch.float16, "bool", "fp32"), (0, 1, 1, 2048, 3, 32, torch.bfloat16, "add32", "fp32"),
    (0, 2, 1, 1476, 3, 64, torch.float16, "bool", "fp32"), (0, 1, 1, 2048, 80, 64, torch.bfloat16, "add32", "fp32")],
    ids=lambda c: "rows%d-B%dS%dR%dH%dD%d-%s-%s-%s" % (*c[:6], str(c[6]).split(".")[-1], c[7], c[8]))
def test_forward_items_of_each_size(cfg):
    """Forward items of two, three and four MSA rows and of two query tiles: row groups and query pairs that are not
    full, one and several items to a block, scores whose maximum lies beyond the first key tile, a row whose keys
    are all dropped.  Against float64; the bound is what rounding P and O to the storage type gives (twice eps / 2),
    and the log-sum-exp has fp32's."""
    from evoformer_triton_b200 import attention, check_device_status
    rows, B, S, R, H, D, dtype, mask, bias = cfg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148 and rows:  # the launcher's rule: these sizes do take items of `rows` rows
        cost = {2: 100, 3: 137 if D > 32 else 130, 4: 158}
        busiest = {n: -(-B * H * -(-R // 128) * -(-S // n) // sms) * c for n, c in cost.items() if n < 4 or D <= 32}
        assert min(busiest, key=lambda n: (busiest[n], n)) == rows
    x = rand_inputs(B, S, R, H, D, dtype, seed=S + R, mask=mask, bias=bias != "none", keep_p=0.8)
    x["Q"][..., R // 2:, :, :] *= 6  # (some rows' scores spread far enough for the running maximum to move)
    if mask == "bool":
        x["res_mask"][0, 0] = False
    q, k, v = (x[n].to(DEV).reshape(B, H, S, R, D) for n in ("Q", "K", "V"))
    b = None if bias == "none" else x["pair_bias"].reshape(B, H, R, R).to(DEV).to(torch.float32 if bias == "fp32" else dtype)
    m = None if mask == "none" else x["res_mask"].reshape(B, S, R).to(DEV)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        o, lse = attention.attention_forward(q, k, v, m, b, D ** -0.5)
        torch.cuda.synchronize()
    check_device_status()
    assert attention.last_path["fwd"] == _lib().PATH_TCGEN05
    ran = [e.name for e in prof.events() if "evo_fwd_sm100_kernel" in e.name]
    if sms == 148 or not rows:  # template arguments: type, padded head dimension, mask, bias, warpgroups, query pairs
        assert len(ran) == 1 and ran[0].split(">")[0].endswith(f"{rows or 2}, {'false' if rows else 'true'}"), ran
    p = (q.double() @ k.double().transpose(-1, -2)) * D ** -0.5
    if b is not None:
        p += b.double()[:, :, None]
    if mask == "bool":
        p.masked_fill_(~m[:, None, :, None, :], -1e300)
    elif m is not None:
        p += m.double()[:, None, :, None, :]
    want_lse = p.logsumexp(-1)
    want = p.softmax(-1) @ v.double()
    assert (o.double() - want).norm() <= torch.finfo(dtype).eps * want.norm()
    live = want_lse > -1e30
    assert (lse.double() - want_lse)[live].abs().max().item() < 2e-5
    if mask == "bool":
        assert (lse[~live] == torch.finfo(torch.float32).min).all()


@pytest.mark.parametrize("cfg", [
    # B, S, R, H, D, dtype, mask, bias
    (1, 5, 200, 2, 32, torch.bfloat16, "bool", "none"), (1, 70, 264, 8, 32, torch.float16, "addsame", "same"),
    (2, 61, 132, 8, 24, torch.bfloat16, "bool", "fp32"), (1, 64, 130, 8, 8, torch.float16, "add32", "none"),
    (1, 63, 200, 8, 16, torch.bfloat16, "bool", "same"), (1, 40, 300, 8, 64, torch.bfloat16, "bool", "none"),
    (2, 1, 520, 4, 48, torch.float16, "addsame", "same"), (1, 3, 64, 1, 64, torch.bfloat16, "none", "fp32"),
    (1, 1, 1, 1, 32, torch.bfloat16, "none", "none")],
    ids=lambda c: "B%dS%dR%dH%dD%d-%s-%s-%s" % (*c[:5], str(c[5]).split(".")[-1], c[6], c[7]))
def test_backward_without_pair_bias_gradient(cfg):
    """The backward kernel that has no d(pair_bias) to sum, against float64: one and several items to a block, row
    groups that are not full, one step in all, a row whose keys are all dropped.  P, dS and the results are rounded to
    the storage type, eps / 2 each, and no more."""
    from evoformer_triton_b200 import attention, check_device_status
    B, S, R, H, D, dtype, mask, bias = cfg
    x = rand_inputs(B, S, R, H, D, dtype, seed=S + R, mask=mask, bias=bias != "none", keep_p=0.8)
    if mask == "bool":
        x["res_mask"][0, 0] = False
    q, k, v, d_o = (x[n].to(DEV).reshape(B, H, S, R, D) for n in ("Q", "K", "V", "dO"))
    b = None if bias == "none" else x["pair_bias"].reshape(B, H, R, R).to(DEV).to(torch.float32 if bias == "fp32" else dtype)
    m = None if mask == "none" else x["res_mask"].reshape(B, S, R).to(DEV)
    o, lse = attention.attention_forward(q, k, v, m, b, D ** -0.5)
    dq, dk, dv, none = attention.attention_backward(q, k, v, o, lse, m, b, D ** -0.5, d_o, want_dbias=False)
    torch.cuda.synchronize()
    check_device_status()
    assert none is None and attention.last_path["bwd"] == _lib().PATH_TCGEN05
    Q, K, V, G = (t.double().requires_grad_() for t in (q, k, v, d_o))
    p = (Q @ K.transpose(-1, -2)) * D ** -0.5
    if b is not None:
        p = p + b.double()[:, :, None]
    if mask == "bool":
        p = p.masked_fill(~m[:, None, :, None, :], -1e300)
    elif m is not None:
        p = p + m.double()[:, None, :, None, :]
    want = torch.autograd.grad(p.softmax(-1) @ V, (Q, K, V), G)
    for name, got, w in zip(("dQ", "dK", "dV"), (dq, dk, dv), want):
        scale = max(w.norm().item(), torch.finfo(dtype).eps * G.norm().item())  # (one key: no gradient but rounding)
        assert (got.double() - w).norm().item() <= 1.5 * torch.finfo(dtype).eps * scale, name
