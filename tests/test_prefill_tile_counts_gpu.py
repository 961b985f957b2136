"""Suffix attention at the edges of its KV tiles (64 positions, in pairs, stages reused from the third on), unsplit and split, against float64."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


# the last one: two row tiles per CTA (every SM still gets a CTA), of which the second holds rows only with more than 128 of them
@pytest.mark.parametrize("d,H,G,T", [(128, 2, 4, 1), (128, 2, 4, 33), (256, 2, 6, 1), (256, 2, 6, 22), (128, 148, 1, 129)])
@pytest.mark.parametrize("positions", [1, 63, 64, 65, 128, 129, 192, 193, 256, 257, 320, 577])
@pytest.mark.parametrize("room", [False, True])      # for the partials of a split launch
@pytest.mark.parametrize("act", [torch.float16, torch.float32])
def test_tile_edges(cuda, d, H, G, T, positions, room, act):
    if positions < T:
        pytest.skip("a chunk is no longer than what it sees")
    P, Hq = positions - T, H * G
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * positions + T)
    st = kv.AttentionLayerKvCacheStorage(positions + 3, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(positions, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, positions, 0, rope_mode=kv.RopeMode.NONE)
    k, v = ((x.double().view(H, -1, d // 32, 32) * s.double().unsqueeze(-1)).flatten(2)[:, :positions]
            for x, s in ((st.key_cache_q8, st.key_scales), (st.value_cache_q8, st.value_scales)))
    q, gate = torch.randn(T, Hq, d, generator=g, device="cuda").to(act), torch.randn(T, Hq, d, generator=g, device="cuda")
    ws = kv.prefill_workspace(positions, H, d, **(dict(token_count=T, query_heads=Hq) if room else {}))
    out = torch.empty(T, Hq, d, device="cuda")
    kv.launch_suffix_attention_quant(st.view(), q, gate, out, ws, T, P, query_heads=Hq, scale=d ** -0.5)
    torch.cuda.synchronize()
    s = torch.einsum("thgd,hld->thgl", q.double().view(T, H, G, d), k) * d ** -0.5
    seen = torch.arange(positions, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgl,hld->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), v).flatten(1, 2) * gate.double().sigmoid()
    # operands and weights enter the MMAs as fp16: 2^-11 each, a few 1e-4 of the result's norm; the gate of the other tests of this kernel
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3
