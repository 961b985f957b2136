"""Suffix attention with two 128-row tiles per CTA (head_dim 128, enough rows for a CTA on every SM) and with KV splits, at the
edges of the row tiles, against the same attention in float64 over the dequantised cache."""
import pytest
import torch

from gpu_util import captured_node_types
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


def expected(st, q, gate, P, T, Hq, scale):
    deq = lambda data, scales: (data.double().view(*scales.shape, -1) * scales.double().unsqueeze(-1)).flatten(2)
    k, v = (deq(d, s)[:, :P + T] for d, s in ((st.key_cache_q8, st.key_scales), (st.value_cache_q8, st.value_scales)))
    G = Hq // k.shape[0]
    s = torch.einsum("thgd,hld->thgl", q.double().view(T, k.shape[0], G, -1), k) * scale
    seen = torch.arange(P + T, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    o = torch.einsum("thgl,hld->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), v).flatten(1, 2)
    return o if gate is None else o * gate.double().sigmoid()


# one row per token and kv head (G = 1) with 148 kv heads: two row tiles per CTA from the second token tile on;
# 2 x 4 heads: the same launch below the line; 40 heads x G = 2: the line itself (ceil(tiles / 2) x 40 >= 148 from 7 tiles on)
@pytest.mark.parametrize("H,G,P,T", [(148, 1, 0, 1), (148, 1, 70, 128), (148, 1, 0, 129), (148, 1, 65, 255), (148, 1, 3, 257), (148, 1, 600, 130),
                                     (148, 2, 64, 193), (8, 4, 100, 33), (40, 2, 130, 384), (40, 2, 130, 385), (37, 1, 1100, 513),
                                     (2, 4, 3001, 33), (1, 1, 4000, 5)])   # few rows over a long prefix: up to 16 splits
@pytest.mark.parametrize("act", [torch.float16, torch.float32])
def test_row_tiles(cuda, H, G, P, T, act):
    g = torch.Generator(device="cuda")
    g.manual_seed(P * 1000 + T)
    d, Hq = 128, H * G
    st = kv.AttentionLayerKvCacheStorage(P + T + 7, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(P + T, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    q = torch.randn(T, Hq, d, generator=g, device="cuda").to(act)
    gate = torch.randn(T, Hq, d, generator=g, device="cuda") if act == torch.float32 else None
    ws = kv.prefill_workspace(P + T, H, d, token_count=T, query_heads=Hq)
    guard = torch.full((T * Hq * d + 4096,), 7.0, device="cuda")
    out = guard[:T * Hq * d].view(T, Hq, d)
    kv.launch_suffix_attention_quant(st.view(), q, gate, out, ws, T, P, query_heads=Hq, scale=d ** -0.5)
    torch.cuda.synchronize()
    ref = expected(st, q, gate, P, T, Hq, d ** -0.5)
    # Operands and weights enter the MMAs as fp16: 2^-11 each on scores of about unit size and on the weights, i.e. a few 1e-4
    # of the result's norm; 1e-3 is the gate the other tests of this kernel use
    assert torch.isfinite(out).all() and (guard[T * Hq * d:] == 7.0).all()
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3


# whether the KV range is split (a merge kernel follows) goes by the prefix, with no step where the chunk grows longer than it
@pytest.mark.parametrize("P,T,kernels", [(0, 2048, 2), (100, 2048, 2), (2047, 2048, 3), (2048, 2048, 3), (2049, 2048, 3), (1100, 1300, 3)])
def test_kv_split_of_a_chunk_about_as_long_as_its_prefix(cuda, P, T, kernels):
    g = torch.Generator(device="cuda")
    g.manual_seed(P)
    d, H, Hq = 128, 1, 4
    st = kv.AttentionLayerKvCacheStorage(P + T, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(P + T, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    q, out = torch.randn(T, Hq, d, generator=g, device="cuda").half(), torch.empty(T, Hq, d, device="cuda")
    ws = kv.prefill_workspace(P + T, H, d, token_count=T, query_heads=Hq)
    go = lambda _: kv.launch_suffix_attention_quant(st.view(), q, None, out, ws, T, P, query_heads=Hq, scale=d ** -0.5)
    go(None)
    ref = expected(st, q, None, P, T, Hq, d ** -0.5)
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3   # fp16 operands, as above
    assert captured_node_types(go) == [0] * kernels
