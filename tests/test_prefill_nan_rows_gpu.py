"""A query row of NaN is its own affair: the other rows of its warp come out as without it, on the unsplit, the split and the two-row-tile launch."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,H,G,P,T", [(256, 1, 6, 0, 40), (256, 1, 6, 3000, 40), (128, 1, 4, 0, 40), (128, 1, 4, 3000, 40), (128, 148, 1, 0, 200)])
def test_other_rows_keep_their_values(cuda, d, H, G, P, T):
    g = torch.Generator(device="cuda")
    g.manual_seed(T + P)
    Hq = H * G
    st = kv.AttentionLayerKvCacheStorage(P + T, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(P + T, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    q = torch.randn(T, Hq, d, generator=g, device="cuda").half()
    ws = kv.prefill_workspace(P + T, H, d, token_count=T, query_heads=Hq)
    outs = []
    for bad in (False, True):
        if bad:
            q[7, G - 1, 3] = float("nan")
        out = torch.empty(T, Hq, d, device="cuda")
        kv.launch_suffix_attention_quant(st.view(), q, None, out, ws, T, P, query_heads=Hq, scale=d ** -0.5)
        outs.append(out)
    torch.cuda.synchronize()
    assert outs[1][7, G - 1].isnan().all()
    outs[1][7, G - 1] = outs[0][7, G - 1]
    assert torch.equal(outs[0], outs[1])
