"""The calls whose speed matters to a user of this package, as cases that can be timed one by one.

A case is one call of the attention op: forward only (inference) or forward and backward (training),
through ``EvoformerAttention.apply`` or the list-style ``evoformer_attention``.  Sizes are those of the
package's workloads C1..C5, of the sweep B=4, H=32, D=64 with a single MSA row, and generic ones; the
number of residues of a protein or a crop is any whole number, so odd ones belong to the range.
"""
import math

import torch

from evoformer_triton_b200 import EvoformerAttention, evoformer_attention

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, call, train, B, S, R, H, D, dtype, mask, bias, bias_grad=True, gate=False, brrh=False, std=0.5):
    """One case.  ``call``: "apply" (reinterpreting layout) or "list" (true head layout); ``mask``: "none",
    "pad" / "random" (bool keep-mask), "add_f32" / "add_same" (additive); ``bias``: "none", "fp32" or "same"
    (the type of Q); ``brrh``: the bias comes as [B, R, R, H], as a linear layer emits it."""
    c = dict(call=call, train=train, B=B, S=S, R=R, H=H, D=D, dtype=dtype, mask=mask, bias=bias,
             bias_grad=bool(train and bias_grad and bias != "none"), gate=gate, brrh=brrh, std=std)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a single short row, forward only: latency, launches and host work are all there is
        _case("short row, inference", "list", False, 4, 1, 32, 32, 64, "bf16", "add_same", "same"),
        # unit-test and debugging size in single precision, forward and backward (C1)
        _case("tiny fp32, training", "apply", True, 1, 16, 64, 4, 32, "fp32", "random", "fp32", std=1.0),
        # MSA row attention of a training crop (C2)
        _case("msa row, training", "apply", True, 1, 128, 384, 8, 32, "bf16", "pad", "fp32"),
        # triangle attention of a training crop (C3), as a pair stack calls it: true head layout, gated,
        # the bias straight from its linear layer
        _case("triangle gated, training", "list", True, 1, 384, 384, 4, 32, "bf16", "add_same", "same", gate=True, brrh=True),
        # extra-MSA stack: many rows, head dimension 8 (C4)
        _case("extra msa, training", "apply", True, 1, 1024, 384, 8, 8, "fp16", "random", "fp32"),
        # large crop, head dimension 64 (C5): the largest
        _case("large crop, training", "apply", True, 2, 512, 768, 8, 64, "bf16", "pad", "fp32"),
        # the single-row sweep: its long end, and one of its lengths that is not a multiple of the tile
        _case("sweep 2048, training", "list", True, 4, 1, 2048, 32, 64, "bf16", "add_same", "same", bias_grad=False),
        _case("sweep 300, training", "list", True, 4, 1, 300, 32, 64, "bf16", "add_same", "same", bias_grad=False),
        # a protein of some odd length, whole, forward only
        _case("odd length, inference", "list", False, 1, 128, 437, 8, 32, "bf16", "add_f32", "same", gate=True, brrh=True),
        # a protein shorter than the crop size: triangle attention on its odd number of residues
        _case("odd triangle, training", "apply", True, 1, 203, 203, 4, 32, "bf16", "random", "fp32"),
        # a long protein or complex: triangle attention, forward only
        _case("long triangle, inference", "apply", False, 1, 1024, 1024, 4, 32, "bf16", "pad", "same"),
        # single precision throughout at a training-like size
        _case("fp32 crop, training", "apply", True, 1, 32, 256, 8, 32, "fp32", "pad", "fp32"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    train = rng.random() < 0.6
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    call = rng.choice(["apply", "list"])
    H, D = rng.choice([(8, 32), (4, 32), (8, 8), (8, 64), (32, 64), (16, 48), (4, 16), (12, 24)])
    R = _log_int(rng, 32, 2048)
    if rng.random() < 0.5:  # half of the lengths are crop sizes, the others are whatever a protein has
        R = max(32, R // 32 * 32)
    B = rng.choice([1, 1, 2, 4])
    # as many rows as a budget of arithmetic allows; a tenth of the calls have a single row
    budget = (2e10 if dtype == "fp32" or R % 8 else 4e11) / (3.5 if train else 1.0)
    while R > 64 and 4.0 * B * H * R * R * D > 2 * budget:
        R = R * 2 // 3
    most = int(budget / (4.0 * B * H * R * R * D))
    S = 1 if most < 2 or rng.random() < 0.1 else _log_int(rng, 1, min(1024, most))
    mask = rng.choice(["pad", "random", "none"] if call == "apply" else ["add_f32", "add_same", "none"])
    bias = "fp32" if dtype == "fp32" else rng.choice(["fp32", "same", "same", "none"])
    gated = call == "list" and rng.random() < 0.5
    return _case(None, call, train, B, S, R, H, D, dtype, mask, bias, bias_grad=rng.random() < 0.8,
                 gate=gated, brrh=gated and bias != "none")


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed))
    B, S, R, H, D = (case[k] for k in "BSRHD")
    dtype = DTYPES[case["dtype"]]
    train = case["train"]

    def normal(shape, std, dt, grad):
        t = torch.empty(shape, dtype=dt, device=dev).normal_(0.0, std, generator=g)
        return t.requires_grad_() if grad else t

    q, k, v = (normal((B, S, R, H, D), case["std"], dtype, train) for _ in range(3))
    mask = None
    if case["mask"] != "none":
        if case["mask"] == "random":
            keep = torch.rand((B, S, R), generator=g, device=dev) < 0.95
        else:  # trailing padding, another amount in every batch entry
            pad = (torch.rand((B, 1, 1), generator=g, device=dev) * (0.15 * R)).floor()
            keep = (torch.arange(R, device=dev) < R - pad).expand(B, S, R)
        keep = keep.reshape(B, S, 1, 1, R).contiguous()
        if case["mask"] in ("pad", "random"):
            mask = keep
        else:
            mt = torch.float32 if case["mask"] == "add_f32" else dtype
            mask = torch.zeros(keep.shape, dtype=mt, device=dev).masked_fill_(~keep, -3e4 if mt == torch.float16 else -1e9)
    bias = None
    if case["bias"] != "none":
        shape = (B, R, R, H) if case["brrh"] else (B, 1, H, R, R)
        bias = normal(shape, 1.0, torch.float32 if case["bias"] == "fp32" else dtype, case["bias_grad"])
    gate = normal((B, S, R, H, D), 1.0, dtype, train) if case["gate"] else None
    d_out = normal((B, S, R, H, D), 1.0, dtype, False) if train else None
    return dict(case=case, q=q, k=k, v=v, mask=mask, bias=bias, gate=gate, d_out=d_out)


def _forward(st):
    case = st["case"]
    if case["call"] == "apply":
        return EvoformerAttention.apply(st["q"], st["k"], st["v"], st["mask"], st["bias"])
    return evoformer_attention(st["q"], st["k"], st["v"], [st["mask"], st["bias"]],
                               pair_bias_layout="brrh" if case["brrh"] else "b1hrr", gate=st["gate"])


def run(st):
    case = st["case"]
    if not case["train"]:
        with torch.no_grad():
            return [_forward(st)]
    out = _forward(st)
    wrt = [st["q"], st["k"], st["v"]]
    if case["bias_grad"]:
        wrt.append(st["bias"])
    if case["gate"]:
        wrt.append(st["gate"])
    return [out.detach(), *torch.autograd.grad(out, wrt, st["d_out"])]


def work(case):
    B, S, R, H, D = (case[k] for k in "BSRHD")
    es = 4 if case["dtype"] == "fp32" else 2
    rows = B * S * R * H * D * es
    bias = 0 if case["bias"] == "none" else B * H * R * R * (4 if case["bias"] == "fp32" else es)
    mask = B * S * R * {"none": 0, "pad": 1, "random": 1, "add_f32": 4, "add_same": es}[case["mask"]]
    tensors = 4 + (1 if case["gate"] else 0)          # Q, K, V, O, gate
    if case["train"]:
        tensors += 4 + (1 if case["gate"] else 0)     # dO, dQ, dK, dV, d(gate)
    nbytes = tensors * rows + mask + bias * (2 if case["bias_grad"] else 1)
    # two matrix products forward, five backward, 2*R*R*D each for every row and head
    return {"bytes": nbytes, "flops": 2.0 * B * H * S * R * R * D * (7 if case["train"] else 2)}


def tolerance(case):
    # probabilities and score gradients are rounded to the storage type before the second products
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
