"""Suffix attention with pointers that its kernels' vector accesses do not take: refused on the host, or sent to the kernel that takes them."""
import ctypes as C

import pytest
import torch

from miinfer_b200 import kv
from miinfer_b200._lib import View, lib


# byte offsets of q (fp16 or fp32), gate and output behind a 16-byte boundary
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("q,gate,out", [(2, 0, 0), (4, 0, 0), (8, 0, 0), (0, 4, 0), (0, 12, 0), (0, 0, 4)])
def test_refused(dtype, q, gate, out):
    """(Nothing is launched: the addresses are the library's to look at only.)"""
    view = View(key_q8=16, key_scales=16, value_q8=16, value_scales=16, capacity=8, kv_heads=1, head_dim=128, qblock=32, quant_mode=3)
    rc = lib.b200kv_prefill_attn(C.byref(view), 4096 + q, dtype, 4096 + gate if gate else None, 4096 + out, 1, 0, 1, 1.0, None, None, 0, None)
    assert rc == lib.b200kv_prefill_attn(C.byref(view), None, dtype, None, 4096, 1, 0, 1, 1.0, None, None, 0, None) != 0


@pytest.mark.gpu
@pytest.mark.parametrize("d,H,G", [(128, 2, 4), (256, 2, 6)])
@pytest.mark.parametrize("gate_off,out_off", [(0, 0), (2, 0), (0, 2), (2, 2)])      # in floats
def test_two_floats(cuda, d, H, G, gate_off, out_off):
    P, T, Hq = 150, 9, H * G
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    st = kv.AttentionLayerKvCacheStorage(P + T, kv.KvCacheQuantMode.kFp16Fp16, kv_heads=H, head_dim=d, qblock=32)
    k, v = rand(P + T, H, d).half(), rand(P + T, H, d).half()
    kv.launch_kv_store_quant(st.view(), k.view(P + T, -1), v.view(P + T, -1), None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    q, n = rand(T, Hq, d).half(), T * Hq * d
    gate = rand(n + 4)[gate_off:gate_off + n].view(T, Hq, d)
    out = torch.full((n + 4,), 7.0, device="cuda")
    kv.launch_suffix_attention_quant(st.view(), q, gate, out[out_off:out_off + n].view(T, Hq, d), kv.prefill_workspace(P + T, H, d, token_count=T, query_heads=Hq), T, P,
                                     query_heads=Hq, scale=d ** -0.5)
    torch.cuda.synchronize()
    s = torch.einsum("thgd,lhd->thgl", q.double().view(T, H, G, d), k.double()) * d ** -0.5
    seen = torch.arange(P + T, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgl,lhd->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), v.double()).flatten(1, 2) * gate.double().sigmoid()
    got = out[out_off:out_off + n].view(T, Hq, d).double()
    # operands and weights enter the MMAs as fp16: 2^-11 each, a few 1e-4 of the result's norm; the gate of the other tests of these kernels
    assert ((got - ref).norm() / ref.norm()).item() <= 1e-3
    assert (out[:out_off] == 7.0).all() and (out[out_off + n:] == 7.0).all()
