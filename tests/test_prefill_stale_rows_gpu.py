"""Suffix attention with the position on the device: cache rows past the visible ones count for nothing, whatever they hold (a session before this one, memory that was never
written), at the edges of the KV tiles, against float64."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


# two row tiles a CTA with 148 heads; the visible rows end in a tile, with one and at the capacity
@pytest.mark.parametrize("d,H,G", [(128, 2, 4), (256, 2, 6), (128, 148, 1)])
@pytest.mark.parametrize("mode,qblock", [(kv.KvCacheQuantMode.kFp16Fp16, 32), (kv.KvCacheQuantMode.kQ8Q8, 32), (kv.KvCacheQuantMode.kQ8Q8, 0)])
@pytest.mark.parametrize("P,T", [(0, 1), (60, 3), (62, 2), (63, 2), (100, 29), (191, 1), (130, 159), (300, 5)])
def test_rows_past_the_visible_ones(cuda, d, H, G, mode, qblock, P, T):
    if H == 148:
        P, T = P + T % 2, T + 128     # a second row tile
    g = torch.Generator(device="cuda")
    g.manual_seed(P + T)
    n, Hq, bound = P + T, H * G, T + 3
    st = kv.AttentionLayerKvCacheStorage(max(n, 500 if n % 2 else n + 1), mode, kv_heads=H, head_dim=d, qblock=qblock or d)
    k, v = (torch.randn(n, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, n, 0, rope_mode=kv.RopeMode.NONE)
    planes = []
    for f16, q8, scales in ((st.key_cache, st.key_cache_q8, st.key_scales), (st.value_cache, st.value_cache_q8, st.value_scales)):
        stale = f16 if f16 is not None else scales
        stale.view(H, st.capacity, -1)[:, n:] = float("nan")
        x = f16.view(H, -1, d) if f16 is not None else (q8.float().view(*scales.shape, -1) * scales.float().unsqueeze(-1)).flatten(2)
        planes.append(x[:, :n].double())
    q, gate = torch.randn(bound, Hq, d, generator=g, device="cuda"), torch.randn(bound, Hq, d, generator=g, device="cuda")
    out = torch.empty(bound, Hq, d, device="cuda")
    ws = kv.prefill_workspace(st.capacity, H, d)
    kv.launch_suffix_attention_quant(st.view(), q, gate, out, ws, bound, 0, query_heads=Hq, scale=d ** -0.5, prefill_state=kv.make_prefill_state(P, T))
    torch.cuda.synchronize()
    s = torch.einsum("thgd,hld->thgl", q[:T].double().view(T, H, G, d), planes[0]) * d ** -0.5
    seen = torch.arange(n, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgl,hld->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), planes[1]).flatten(1, 2) * gate[:T].double().sigmoid()
    assert (out[T:] == 0).all()       # tokens past the device's count
    # operands and weights enter the MMAs as fp16: 2^-11 each, a few 1e-4 of the result's norm; the gate of the other tests of this kernel
    assert ((out[:T].double() - ref).norm() / ref.norm()).item() <= 1e-3
