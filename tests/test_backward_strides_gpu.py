"""GPU: gradients written with negative strides through the C ABI (rows from the last residue to the first)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D,with_bias", [(32, True), (32, False), (64, True)])
def test_dk_and_dv_from_the_last_row_to_the_first(D, with_bias):
    from evoformer_triton_b200 import _lib, attention
    lib = _lib.load()
    B, H, S, R = 1, 2, 3, 136
    g = torch.Generator(device=DEV).manual_seed(D)
    mk = lambda *s, dt=torch.bfloat16: torch.randn(s, generator=g, device=DEV).to(dt)  # noqa: E731
    q, k, v, d_o = (mk(B, H, S, R, D) for _ in range(4))
    bias = mk(B, H, R, R, dt=torch.float32) if with_bias else None
    scale = D ** -0.5
    o, lse = attention.attention_forward(q, k, v, None, bias, scale)
    want = attention.attention_backward(q, k, v, o, lse, None, bias, scale, d_o)
    p = _lib.BwdParams()
    attention._fill_fwd(p.fwd, q, k, v, o, lse, None, bias, scale)
    dq, dk, dv = (torch.full_like(q, 7.0) for _ in range(3))
    dbias = None if bias is None else torch.full_like(bias, 7.0)
    p.d_o, p.dq, p.dbias = d_o.data_ptr(), dq.data_ptr(), None if bias is None else dbias.data_ptr()
    last = (R - 1) * D * q.element_size()
    p.dk, p.dv = dk.data_ptr() + last, dv.data_ptr() + last
    p.do_stride, p.dq_stride = attention._strides4(d_o), attention._strides4(dq)
    back = (C.c_int64 * 4)(*dk.stride()[:3], -D)
    p.dk_stride, p.dv_stride = back, back
    need = int(lib.evoattn_bwd_workspace_bytes(C.byref(p)))
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device=DEV)
    p.workspace, p.workspace_bytes = ws.data_ptr(), need
    assert lib.evoattn_bwd(C.byref(p), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    attention.check_device_status()
    for name, a, b in zip(("dq", "dk", "dv", "dbias"), (dq, dk.flip(3), dv.flip(3), dbias), want):
        if b is not None:  # (one or the other kernel: a 16-bit rounding of P, dS and the result apart)
            assert (a.double() - b.double()).abs().max() <= 1e-2 * b.double().abs().max(), name
