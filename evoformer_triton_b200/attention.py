"""Host side of the Evoformer attention op: the reference's autograd boundary.

``EvoformerAttention`` mirrors dsevoformer-triton/evoformer.py:633-862: same class
name, same ``apply(Q, K, V, res_mask, pair_bias)`` call on ``[B, N_seq, N_res, H, D]``
tensors, same reinterpretation of those tensors as ``[B, H, N_seq, N_res, D]``
(evoformer.py:648-650), same ``(dQ, dK, dV, None, d_pair_bias)`` gradients.  The device
work is done by libevoattn.so through its C ABI; torch is used for memory and streams.
A call goes through the native boundary (csrc/host.cpp); the raw forward and backward below are the
same steps in Python, for the N_seq-sharded op and for callers that hold attention-view tensors.
"""
from __future__ import annotations

import collections.abc
import contextlib
import ctypes as C
import os
import threading
from typing import Optional, Sequence

import torch

from . import _lib

_DTYPES = {torch.bfloat16: _lib.BF16, torch.float16: _lib.FP16, torch.float32: _lib.FP32}


class _LastCall(collections.abc.Mapping):
    """What the most recent forward and backward call of the process reported."""

    def __init__(self, read):
        self._read = read

    def __getitem__(self, key):
        return dict(zip(("fwd", "bwd"), self._read(_lib.host())))[key]

    def __iter__(self):
        return iter(("fwd", "bwd"))

    def __len__(self):
        return 2

    def __repr__(self):
        return repr(dict(self))


# Launch counters the benchmark reads (kernels of this library only), and which kernel family ran.
launches = _LastCall(lambda h: h.launch_counts())
last_path = _LastCall(lambda h: h.paths())
_force_generic = False


def force_generic(on: bool) -> None:
    """Route every call to the CUDA-core kernels: slower, with P and dS of 16-bit calls in fp32 where the tensor
    cores take them in the storage type (errors about 1.4 times smaller)."""
    global _force_generic
    _force_generic = bool(on)
    _lib.host().force_generic(_force_generic)


if int(os.environ.get("EVOATTN_FORCE_GENERIC", "0")):
    force_generic(True)


def _status_word(device: torch.device) -> torch.Tensor:
    """One int32 per device that kernels set when they give up a bounded wait."""
    return _lib.host().status_word(torch.cuda.current_device() if device.index is None else device.index)


def check_device_status(device=None) -> None:
    """Synchronise and raise if any kernel reported a timed-out wait."""
    for t in _lib.host().status_words():
        if device is not None and torch.device(device) != t.device:
            continue
        v = int(t.item())
        if v != 0:
            t.zero_()
            raise RuntimeError(f"evoattn kernel on {t.device} gave up a bounded wait (device status {v})")


def _strides4(t: torch.Tensor):
    st = t.stride()
    return (C.c_int64 * 4)(st[0], st[1], st[2], st[3])


def _fill_fwd(p: "_lib.FwdParams", q, k, v, o, lse, mask, bias, scale, gate=None):
    B, H, S, R, D = q.shape
    p.dtype = _DTYPES[q.dtype]
    p.B, p.H, p.S, p.R, p.D = B, H, S, R, D
    p.scale = float(scale)
    p.flags = _lib.FLAG_FORCE_GENERIC if _force_generic else 0
    p.q, p.k, p.v, p.o, p.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr()
    p.q_stride, p.k_stride, p.v_stride, p.o_stride = _strides4(q), _strides4(k), _strides4(v), _strides4(o)
    if mask is None:
        p.mask, p.mask_kind = None, _lib.MASK_NONE
    else:
        p.mask = mask.data_ptr()
        if mask.dtype == torch.bool:
            p.mask_kind = _lib.MASK_BOOL
        elif mask.dtype == torch.float32:
            p.mask_kind = _lib.MASK_ADD_F32
        elif mask.dtype == q.dtype:
            p.mask_kind = _lib.MASK_ADD_SAME
        else:
            raise TypeError(f"res_mask dtype {mask.dtype} not supported (bool, float32 or the q/k/v dtype)")
        ms = mask.stride()
        p.mask_stride = (C.c_int64 * 3)(ms[0], ms[1], ms[2])
    if bias is None:
        p.bias = None
    else:
        if bias.dtype != torch.float32 and bias.dtype != q.dtype:
            raise TypeError("pair bias must be float32 or of the q/k/v dtype")
        p.bias = bias.data_ptr()
        p.bias_dtype = _lib.BIAS_F32 if bias.dtype == torch.float32 else _lib.BIAS_SAME
        bs = bias.stride()
        p.bias_stride = (C.c_int64 * 3)(bs[0], bs[1], bs[2])
    p.status = _status_word(q.device).data_ptr()
    if gate is None:
        p.gate = None
    else:
        p.gate = gate.data_ptr()
        p.gate_stride = _strides4(gate)


def _view_dims(x: torch.Tensor, layout: str) -> torch.Tensor:
    """[B,S,R,H,D] -> the [B,H,S,R,D] attention view (no copy for contiguous input)."""
    B, S, R, H, D = x.shape
    if layout == "reinterpret":
        return x.reshape(B, H, S, R, D)  # evoformer.py:648-650
    return x.permute(0, 3, 1, 2, 4)


def _unview(x: torch.Tensor, layout: str) -> torch.Tensor:
    B, H, S, R, D = x.shape
    if layout == "reinterpret":
        return x.reshape(B, S, R, H, D)  # evoformer.py:735
    return x.permute(0, 2, 3, 1, 4)


def _prep_operand(x: torch.Tensor) -> torch.Tensor:
    if x.stride(-1) != 1:
        x = x.contiguous()
    return x


def attention_forward(q, k, v, mask, bias, scale, gate=None):
    """Raw forward on attention-view tensors.  Returns (o, lse); with ``gate`` (attention view,
    same dtype) ``o`` is ``sigmoid(gate) * attention``, multiplied in the kernel's epilogue."""
    lib = _lib.load()
    B, H, S, R, D = q.shape
    o = torch.empty((B, H, S, R, D), dtype=q.dtype, device=q.device)
    lse = torch.empty((B, H, S, R), dtype=torch.float32, device=q.device)
    p = _lib.FwdParams()
    _fill_fwd(p, q, k, v, o, lse, mask, bias, scale, gate)
    stream = torch.cuda.current_stream(q.device).cuda_stream
    with torch.cuda.device(q.device):
        _lib.check(lib.evoattn_fwd(C.byref(p), C.c_void_p(stream)), "evoattn_fwd")
    _lib.host().note_fwd(lib.evoattn_last_launch_count(), lib.evoattn_last_path())
    return o, lse


def attention_backward(q, k, v, o, lse, mask, bias, scale, d_o, want_dbias=True, dbias_out=None, gate=None,
                       want_dmask=False, exchange=None):
    """Raw backward on attention-view tensors.  Returns (dq, dk, dv, dbias fp32 or None), plus
    ``dgate`` when ``gate`` is given (``o`` and ``d_o`` are then the gated output and its
    gradient) and the fp32 ``[B,S,R]`` gradient of an additive mask when ``want_dmask``.
    ``want_dbias=False`` skips d(pair_bias) (its reductions are the backward's largest stream
    of writes; speed_benchmark.py:68 builds the bias without ``requires_grad``).  ``exchange``
    (a ``PeerAllReduceParams`` whose own buffer is ``dbias_out``) makes the call sum d(pair_bias)
    over the node's GPUs itself, next to its last kernel."""
    lib = _lib.load()
    B, H, S, R, D = q.shape
    dq = torch.empty((B, H, S, R, D), dtype=q.dtype, device=q.device)
    dk = torch.empty_like(dq)
    dv = torch.empty_like(dq)
    dbias = None
    if bias is not None and want_dbias:
        # (``dbias_out``: caller-provided fp32 storage, e.g. a buffer peers can reach)
        dbias = dbias_out.view(B, H, R, R) if dbias_out is not None else \
            torch.empty((B, H, R, R), dtype=torch.float32, device=q.device)
    p = _lib.BwdParams()
    _fill_fwd(p.fwd, q, k, v, o, lse, mask, bias, scale, gate)
    dgate = dmask = None
    if gate is not None:
        dgate = torch.empty((B, H, S, R, D), dtype=q.dtype, device=q.device)
        p.dgate, p.dgate_stride = dgate.data_ptr(), _strides4(dgate)
    if want_dmask:
        dmask = torch.empty((B, S, R), dtype=torch.float32, device=q.device)
        p.dmask = dmask.data_ptr()
    p.d_o, p.dq, p.dk, p.dv = d_o.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr()
    p.dbias = None if dbias is None else dbias.data_ptr()
    if exchange is not None:
        if dbias is None or dbias_out is None:
            raise ValueError("the in-call exchange sums d(pair_bias) in the caller's exchange buffer")
        p.exchange = C.pointer(exchange)
    p.do_stride, p.dq_stride, p.dk_stride, p.dv_stride = _strides4(d_o), _strides4(dq), _strides4(dk), _strides4(dv)
    need = lib.evoattn_bwd_workspace_bytes(C.byref(p))
    ws = torch.empty(max(int(need), 1), dtype=torch.uint8, device=q.device)
    p.workspace, p.workspace_bytes = ws.data_ptr(), int(need)
    stream = torch.cuda.current_stream(q.device).cuda_stream
    with torch.cuda.device(q.device):
        _lib.check(lib.evoattn_bwd(C.byref(p), C.c_void_p(stream)), "evoattn_bwd")
    _lib.host().note_bwd(lib.evoattn_last_launch_count(), lib.evoattn_last_path())
    if gate is None and not want_dmask:
        return dq, dk, dv, dbias
    return dq, dk, dv, dbias, dgate, dmask


def _rows_of_16_bytes(R: int, dtype: torch.dtype) -> int:
    """``R`` rounded up so that a row of that many elements is a whole number of 16-byte pieces."""
    per = 16 // dtype.itemsize
    return (R + per - 1) // per * per


def pad_bias_rows(bias: torch.Tensor) -> torch.Tensor:
    """A ``[B, H, R, R]`` pair bias whose rows a tensor map cannot read (their stride is not a multiple
    of 16 bytes, as for most odd ``R``) copied into padded rows; any other bias as it is.  One pass
    over the bias, which the MSA rows share, instead of the CUDA-core kernels for the whole call."""
    es = bias.element_size()
    if bias.data_ptr() % 16 == 0 and all(st * es % 16 == 0 for st in bias.stride()[:3]):
        return bias
    lib = _lib.load()
    B, H, R, _ = bias.shape
    ld = _rows_of_16_bytes(R, bias.dtype)
    dst = torch.empty((B, H, R, ld), dtype=bias.dtype, device=bias.device)
    stream = torch.cuda.current_stream(bias.device).cuda_stream
    with torch.cuda.device(bias.device):
        _lib.check(lib.evoattn_bias_pad_rows(bias.data_ptr(), (C.c_int64 * 3)(*bias.stride()[:3]), dst.data_ptr(),
                                             _DTYPES[bias.dtype], B, H, R, ld, C.c_void_p(stream)), "evoattn_bias_pad_rows")
    return dst[..., :R]


def bias_to_heads_first(bias_brrh: torch.Tensor) -> torch.Tensor:
    """``[B, R, R, H]`` (as a linear layer emits a pair bias) -> ``[B, H, R, R]``, same dtype, one
    device pass (the reference's layout, evoformer.py:638,652, makes its caller permute and copy);
    rows padded to whole 16-byte pieces."""
    lib = _lib.load()
    B, R, R2, H = bias_brrh.shape
    src = bias_brrh.contiguous()
    ld = _rows_of_16_bytes(R, src.dtype)
    dst = torch.empty((B, H, R, ld), dtype=src.dtype, device=src.device)
    stream = torch.cuda.current_stream(src.device).cuda_stream
    with torch.cuda.device(src.device):
        _lib.check(lib.evoattn_bias_to_heads_first_ld(src.data_ptr(), dst.data_ptr(), _DTYPES[src.dtype], B, H, R, ld,
                                                      C.c_void_p(stream)), "evoattn_bias_to_heads_first_ld")
    return dst[..., :R]


def dbias_to_heads_last(dbias_bhrr: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """fp32 ``[B, H, R, R]`` gradient -> ``[B, R, R, H]`` in ``dtype``: the layout change and the one
    cast of the gradient in a single device pass."""
    lib = _lib.load()
    B, H, R, _ = dbias_bhrr.shape
    dst = torch.empty((B, R, R, H), dtype=dtype, device=dbias_bhrr.device)
    stream = torch.cuda.current_stream(dst.device).cuda_stream
    with torch.cuda.device(dst.device):
        _lib.check(lib.evoattn_dbias_to_heads_last(dbias_bhrr.data_ptr(), dst.data_ptr(), _DTYPES[dtype], B, H, R,
                                                   C.c_void_p(stream)), "evoattn_dbias_to_heads_last")
    return dst


_pending = threading.local()


@contextlib.contextmanager
def pair_bias_grad_summed_over(group, peer_reducer=None):
    """Calls of the op made inside this context sum their d(pair_bias) over the ranks of
    ``group`` (``None`` = the default process group) in backward: the fp32 sum over the local
    MSA rows is all-reduced as it leaves the kernel, before the single cast to the bias dtype.
    With ``peer_reducer`` (:class:`evoformer_triton_b200.sharding.PeerReducer`) the kernel writes
    into peer-mapped memory and the sum runs over NVLink in this package's own kernel instead of
    NCCL.  Used by :func:`evoformer_triton_b200.sharding.sharded_evoformer_attention`."""
    prev = getattr(_pending, "group", None)
    _pending.group = (group, peer_reducer)
    try:
        yield
    finally:
        _pending.group = prev


class _EvoformerAttentionBase(torch.autograd.Function):
    """What the public classes share.  A call goes to the native boundary (csrc/host.cpp); inside
    :func:`pair_bias_grad_summed_over` it is this Function itself, whose backward sums d(pair_bias)
    over the ranks, and so it is where a tracer wants one node (:func:`_python_boundary`).  ``layout`` (how heads are found in Q/K/V) and ``bias_layout``
    (``"b1hrr"``: the reference's ``[B, 1, H, R, R]``; ``"brrh"``: ``[B, R, R, H]`` as a linear
    layer emits it) are fixed by the public subclasses."""

    layout = "reinterpret"
    bias_layout = "b1hrr"

    @classmethod
    def apply(cls, Q, K, V, res_mask=None, pair_bias=None):
        return cls._call(Q, K, V, res_mask, pair_bias)

    @classmethod
    def _call(cls, Q, K, V, res_mask, pair_bias, *gate):
        if getattr(_pending, "group", None) is not None:
            return cls._function(Q, K, V, res_mask, pair_bias, *gate)
        return _lib.host().attention(Q, K, V, res_mask, pair_bias, gate[0] if gate else None,
                                     cls.layout == "true", cls.bias_layout == "brrh")

    @classmethod
    def _function(cls, *args):
        return super().apply(*args)

    @classmethod
    def _forward(cls, ctx, Q, K, V, res_mask, pair_bias, gate=None):
        q, k, v, mask, bias, g = _lib.host().prepare_call(Q, K, V, res_mask, pair_bias, gate, cls.layout == "true",
                                                          cls.bias_layout == "brrh")
        B, S, R, H, D = Q.shape
        scale = D ** -0.5  # evoformer.py:646
        q, k, v = (_view_dims(t, cls.layout) for t in (q, k, v))
        g = None if g is None else _view_dims(g, cls.layout)
        mask = None if mask is None else mask.view(B, S, R)  # [B,S,1,1,R] in the reference (evoformer.py:651)
        if bias is not None:  # [B,1,H,R,R] (evoformer.py:652), or [B,H,R,>=R] where the rows had to be padded
            bias = (bias.squeeze(1) if bias.dim() == 5 else bias)[..., :R]
        o, lse = attention_forward(q, k, v, mask, bias, scale, g)
        ctx.save_for_backward(q, k, v, mask, bias, o, lse, g)  # evoformer.py:729
        ctx.softmax_scale = scale
        ctx.bias_meta = None if pair_bias is None else (pair_bias.dtype, tuple(pair_bias.shape))
        ctx.mask_meta = None if res_mask is None else (res_mask.dtype, tuple(res_mask.shape))
        ctx.reduce_group = getattr(_pending, "group", None)
        return _unview(o, cls.layout)

    @classmethod
    def _backward(cls, ctx, dO):
        q, k, v, mask, bias, o, lse, g = ctx.saved_tensors
        if cls.layout == "reinterpret":
            dO = dO.contiguous()  # the reference asserts contiguity instead (evoformer.py:747)
        d_o = _prep_operand(_view_dims(dO, cls.layout))
        if d_o.dtype != q.dtype:
            d_o = d_o.to(q.dtype)
        want_dbias = bias is not None and ctx.needs_input_grad[4]
        want_dmask = mask is not None and mask.is_floating_point() and ctx.needs_input_grad[3]
        if want_dmask and ctx.reduce_group is not None:
            raise RuntimeError("a mask gradient is not available in the N_seq-sharded op (the mask rows are sharded)")
        reducer = ctx.reduce_group[1] if want_dbias and ctx.reduce_group is not None else None
        dbias_out = reducer.buffer(bias.numel()) if reducer is not None else None
        # (with a peer reducer the call sums d(pair_bias) over the ranks itself, next to its last kernel)
        res = attention_backward(q, k, v, o, lse, mask, bias, ctx.softmax_scale, d_o, want_dbias=want_dbias,
                                 dbias_out=dbias_out, gate=g, want_dmask=want_dmask,
                                 exchange=None if reducer is None else reducer.exchange_params(bias.numel()))
        dq, dk, dv, dbias = res[:4]
        dgate, dmask = res[4:] if len(res) > 4 else (None, None)
        if dmask is not None:
            dtype, shape = ctx.mask_meta
            dmask = dmask.reshape(shape).to(dtype)
        d_pair_bias = None
        if dbias is not None:
            dtype, shape = ctx.bias_meta
            # N_seq is sharded: the other ranks' rows belong to the sum (with a reducer it was taken in the call)
            if ctx.reduce_group is not None and reducer is None:
                import torch.distributed as dist
                dist.all_reduce(dbias, op=dist.ReduceOp.SUM, group=ctx.reduce_group[0])
            # the sum over N_seq stays in fp32 until this single cast (evoformer.py:860 casts to dO's dtype)
            if cls.bias_layout == "brrh":
                d_pair_bias = dbias_to_heads_last(dbias, dtype if dtype in _DTYPES else torch.float32).to(dtype)
            else:
                d_pair_bias = dbias.reshape(shape).to(dtype)
                if reducer is not None and d_pair_bias.data_ptr() == dbias.data_ptr():
                    d_pair_bias = d_pair_bias.clone()  # the exchange buffer is reused by the next call
        grads = (_unview(dq, cls.layout), _unview(dk, cls.layout), _unview(dv, cls.layout), dmask, d_pair_bias)
        if g is not None:
            grads = grads + (_unview(dgate, cls.layout),)
        return grads


class EvoformerAttention(_EvoformerAttentionBase):
    """Drop-in for ``evoformer.EvoformerAttention`` (dsevoformer-triton/evoformer.py:633).

    ``EvoformerAttention.apply(Q, K, V, res_mask, pair_bias)`` with
    Q, K, V ``[B, N_seq, N_res, H, D]``; res_mask ``[B, N_seq, 1, 1, N_res]`` (bool keep-mask,
    or a floating tensor that is added to the scores); pair_bias ``[B, 1, H, N_res, N_res]``.
    Like the reference, the head axis is obtained by *reinterpreting* the buffer as
    ``[B, H, N_seq, N_res, D]``.  Unlike the reference, ``None`` works for the mask and the bias.
    """

    layout = "reinterpret"

    @staticmethod
    def forward(ctx, Q, K, V, res_mask=None, pair_bias=None):
        return EvoformerAttention._forward(ctx, Q, K, V, res_mask, pair_bias)

    @staticmethod
    def backward(ctx, dO):
        return EvoformerAttention._backward(ctx, dO)


class EvoformerAttentionTrueLayout(_EvoformerAttentionBase):
    """Same op with genuine head semantics: head h of Q is ``Q[:, :, :, h, :]``
    (what ``DS4Sci_EvoformerAttention`` computes).  The kernels read the strided view
    in place through their tensor maps; nothing is transposed in memory."""

    layout = "true"

    @staticmethod
    def forward(ctx, Q, K, V, res_mask=None, pair_bias=None):
        return EvoformerAttentionTrueLayout._forward(ctx, Q, K, V, res_mask, pair_bias)

    @staticmethod
    def backward(ctx, dO):
        return EvoformerAttentionTrueLayout._backward(ctx, dO)


class GatedEvoformerAttention(_EvoformerAttentionBase):
    """``apply(Q, K, V, res_mask, pair_bias, gate)``: the attention of :class:`EvoformerAttention`
    followed by the sigmoid gate of a gated-attention block, ``sigmoid(gate) * O`` with ``gate`` of
    the shape of Q, multiplied in the forward kernel's epilogue; backward returns a gradient for the
    gate as well.  Not in the reference, whose op ends at O."""

    layout = "reinterpret"

    @classmethod
    def apply(cls, Q, K, V, res_mask, pair_bias, gate):
        return cls._call(Q, K, V, res_mask, pair_bias, gate)

    @staticmethod
    def forward(ctx, Q, K, V, res_mask, pair_bias, gate):
        return GatedEvoformerAttention._forward(ctx, Q, K, V, res_mask, pair_bias, gate)

    @staticmethod
    def backward(ctx, dO):
        return GatedEvoformerAttention._backward(ctx, dO)


def _variant(layout: str, bias_layout: str, gated: bool):
    """The autograd.Function for a combination of head layout, bias layout and gating."""
    key = (layout, bias_layout, gated)
    fn = _VARIANTS.get(key)
    if fn is None:
        def apply(cls, Q, K, V, res_mask=None, pair_bias=None, gate=None):  # (what a traced node calls)
            return cls._call(Q, K, V, res_mask, pair_bias, gate)

        def forward(ctx, Q, K, V, res_mask=None, pair_bias=None, gate=None):
            return fn._forward(ctx, Q, K, V, res_mask, pair_bias, gate)

        def backward(ctx, dO):
            grads = fn._backward(ctx, dO)
            return grads if len(grads) == 6 else grads + (None,)

        fn = type(f"EvoformerAttention_{layout}_{bias_layout}{'_gated' if gated else ''}", (_EvoformerAttentionBase,),
                  {"layout": layout, "bias_layout": bias_layout, "apply": classmethod(apply),
                   "forward": staticmethod(forward), "backward": staticmethod(backward)})
        _VARIANTS[key] = fn
    return fn


_VARIANTS = {}


def _python_boundary(Q, K, V, res_mask, pair_bias, gate, true_layout, heads_last):
    """A call as a Python autograd.Function: what ``torch.jit.trace`` records as one node that runs the op."""
    fn = _variant("true" if true_layout else "reinterpret", "brrh" if heads_last else "b1hrr", gate is not None)
    return fn._function(Q, K, V, res_mask, pair_bias, gate)


def evoformer_attention(Q, K, V, biases: Optional[Sequence[Optional[torch.Tensor]]] = None, *, layout="true",
                        pair_bias_layout="b1hrr", gate=None):
    """List-style call ``attn(Q, K, V, [res_mask_bias, pair_bias])`` of
    ``DS4Sci_EvoformerAttention`` (used at dsevoformer-triton/speed_benchmark.py:24,84).

    ``biases[0]`` is the residue mask ``[B, N_seq, 1, 1, N_res]`` (additive when floating,
    keep-mask when bool); ``biases[1]`` the pair bias ``[B, 1, H, N_res, N_res]``.
    ``layout="true"`` (default) takes heads from axis 3 as DS4Sci does;
    ``layout="reinterpret"`` matches ``EvoformerAttention``.
    ``pair_bias_layout="brrh"`` takes the pair bias as ``[B, N_res, N_res, H]``, the way a linear
    layer on the pair representation emits it, and returns its gradient in that layout.
    ``gate`` (shape of Q) multiplies the output by ``sigmoid(gate)`` inside the kernel.
    A floating ``res_mask_bias`` that requires a gradient gets one, as in DS4Sci.
    """
    biases = list(biases or [])
    while len(biases) < 2:
        biases.append(None)
    if getattr(_pending, "group", None) is None:
        return _lib.host().attention(Q, K, V, biases[0], biases[1], gate, layout == "true", pair_bias_layout == "brrh")
    fn = _variant("true" if layout == "true" else "reinterpret", pair_bias_layout, gate is not None)
    return fn._call(Q, K, V, biases[0], biases[1], gate)
