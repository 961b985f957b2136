"""Suffix attention over caches with an fp16 side, which the tcgen05 kernel reads where it lies: NaN in the rows past the visible ones (of this head and of the
next), at the edges of the KV tiles, split and whole, against float64."""
import pytest
import torch

from gpu_util import captured_grids
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [kv.KvCacheQuantMode.kFp16Fp16, kv.KvCacheQuantMode.kQ8Fp16, kv.KvCacheQuantMode.kFp16Q8])
@pytest.mark.parametrize("d,H,G", [(128, 3, 4), (256, 2, 6)])
@pytest.mark.parametrize("P,T", [(0, 1), (0, 70), (60, 5), (63, 1), (64, 1), (100, 29), (513, 40), (2048, 7)])
def test_planes(cuda, mode, d, H, G, P, T):
    g = torch.Generator(device="cuda")
    g.manual_seed(P + T)
    n, Hq = P + T, H * G
    st = kv.AttentionLayerKvCacheStorage(n + 37, mode, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(n, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, n, 0, rope_mode=kv.RopeMode.NONE)
    planes = []
    for f16, q8, scales in ((st.key_cache, st.key_cache_q8, st.key_scales), (st.value_cache, st.value_cache_q8, st.value_scales)):
        if f16 is not None:
            f16.view(H, -1, d)[:, n:] = float("nan")
            planes.append(f16.view(H, -1, d)[:, :n].double())
        else:
            planes.append((q8.double().view(H, -1, d // 32, 32) * scales.double().view(H, -1, d // 32, 1)).flatten(2)[:, :n])
    q = torch.randn(T, Hq, d, generator=g, device="cuda")
    ws = kv.prefill_workspace(n, H, d, token_count=T, query_heads=Hq)
    ws.view(torch.uint8).fill_(0xFF)
    out = torch.empty(T, Hq, d, device="cuda")
    go = lambda _: kv.launch_suffix_attention_quant(st.view(), q, None, out, ws, T, P, query_heads=Hq, scale=d ** -0.5)
    go(None)
    torch.cuda.synchronize()
    s = torch.einsum("thgd,hld->thgl", q.double().view(T, H, G, d), planes[0]) * d ** -0.5
    seen = torch.arange(n, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgl,hld->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), planes[1]).flatten(1, 2)
    # operands and weights enter the MMAs as fp16: 2^-11 each, a few 1e-4 of the result's norm; the gate of the other tests of this kernel
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-3
    # from the second tile on no pre-pass, or one of the int8 side alone
    assert captured_grids(go)[0][1:] == ((H, 2) if n <= 64 else (1, 1) if mode == kv.KvCacheQuantMode.kFp16Fp16 else (H, 1))
