"""Few rows over a long prefix in 1 to 16 KV splits (the workspace has room for no more): the merge's variants for up to 4, 8, 12 and 16, against float64."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [1, 2, 4, 5, 8, 9, 12, 13, 16])
@pytest.mark.parametrize("d,G", [(128, 4), (256, 6)])
@pytest.mark.parametrize("gated", [False, True])
def test_splits(cuda, splits, d, G, gated):
    P, T, H = 3300, 5, 1
    g = torch.Generator(device="cuda")
    g.manual_seed(splits)
    st = kv.AttentionLayerKvCacheStorage(P + T, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(P + T, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    k, v = ((x.double().view(H, -1, d // 32, 32) * s.double().unsqueeze(-1)).flatten(2)[0] for x, s in ((st.key_cache_q8, st.key_scales), (st.value_cache_q8, st.value_scales)))
    q = torch.randn(T, G, d, generator=g, device="cuda").half()
    gate = torch.randn(T, G, d, generator=g, device="cuda") if gated else None
    room = kv.prefill_workspace(P + T, H, d).numel() + 1024 + splits * H * 128 * (d + 2) * 4
    ws, out = torch.full((room,), 0xFF, dtype=torch.uint8, device="cuda"), torch.empty(T, G, d, device="cuda")
    kv.launch_suffix_attention_quant(st.view(), q, gate, out, ws, T, P, query_heads=G, scale=d ** -0.5)
    torch.cuda.synchronize()
    s = torch.einsum("tgd,ld->tgl", q.double(), k) * d ** -0.5
    seen = torch.arange(P + T, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("tgl,ld->tgd", s.masked_fill(~seen[:, None], float("-inf")).softmax(-1), v) * (gate.double().sigmoid() if gated else 1.0)
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3   # operands and weights as fp16, the gate of the other tests of this kernel
