"""The merge inside a decode launch at the edges of its rounds (four groups of threads take ten splits each at a time), against float64."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 3, 5, 39, 40, 41, 79, 81, 128])
@pytest.mark.parametrize("d,H,G,mode,rel", [(128, 1, 4, 3, 2e-4),      # tcgen05 kernel: query and weights as 15 and 16 bits of fixed point
                                            (256, 1, 6, 0, 2e-6)])     # streaming kernel, fp16 cache: fp32 sums
def test_split_counts(cuda, splits, d, H, G, mode, rel):
    L, Hq = 128 * 128 + 77, H * G
    g = torch.Generator(device="cuda")
    g.manual_seed(splits)
    st = kv.AttentionLayerKvCacheStorage(L + 3, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=32 if mode else d)
    k, v = (torch.randn(L, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, L, 0, rope_mode=kv.RopeMode.NONE)
    if mode:
        k, v = ((x.double().view(H, -1, d // 32, 32) * s.double().unsqueeze(-1)).flatten(2)[:, :L]
                for x, s in ((st.key_cache_q8, st.key_scales), (st.value_cache_q8, st.value_scales)))
    else:
        k, v = (x.double()[:, :L] for x in (st.key_cache, st.value_cache))
    q, gate = torch.randn(Hq, d, generator=g, device="cuda"), torch.randn(Hq, d, generator=g, device="cuda")
    out, gated = torch.empty(Hq, d, device="cuda"), torch.empty(Hq, d, device="cuda")
    ws = kv.decode_workspace(Hq, d)

    def go():
        kv.launch_decode_attention_quant(st.view(), q, query_heads=Hq, scale=d ** -0.5, cache_length=L, output=out, gate=gate, gated_output=gated,
                                         workspace=ws, num_splits=splits)

    def check():
        torch.cuda.synchronize()
        p = (torch.einsum("hgd,hld->hgl", q.double().view(H, G, d), k) * d ** -0.5).softmax(-1)
        ref = torch.einsum("hgl,hld->hgd", p, v).flatten(0, 1)
        assert ((out.double() - ref).norm() / ref.norm()).item() <= rel
        ref = ref * gate.double().sigmoid()
        assert ((gated.double() - ref).norm() / ref.norm()).item() <= rel
        assert ws.count_nonzero().item() == 0      # what a merge reads it zeroes

    go()
    check()
    # replays of a captured launch share its tag: words that one left behind would pass for the next one's
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        go()
    for _ in range(3):
        q.copy_(torch.randn(Hq, d, generator=g, device="cuda"))
        out.fill_(float("nan"))
        gated.fill_(float("nan"))
        graph.replay()
        check()
