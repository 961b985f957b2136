"""Launches that split their KV range: two row tiles per CTA (head_dim 128) and single ones at the edges of the KV tiles, against float64, and how many splits
a launch takes."""
import pytest
import torch

from gpu_util import captured_grids
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


def run(d, H, G, P, T, act, gated, rows_per_cta):
    """(KV splits of the launch, relative error of its output); the workspace holds NaN beforehand, and the output a guard behind it."""
    Hq, scale = H * G, d ** -0.5
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * P + T)
    st = kv.AttentionLayerKvCacheStorage(P + T + 5, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=32)
    k, v = (torch.randn(P + T, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, P + T, 0, rope_mode=kv.RopeMode.NONE)
    q = torch.randn(T, Hq, d, generator=g, device="cuda").to(act)
    gate = torch.randn(T, Hq, d, generator=g, device="cuda") if gated else None
    ws = kv.prefill_workspace(P + T, H, d, token_count=T, query_heads=Hq)
    ws.view(torch.uint8).fill_(0xFF)
    guard = torch.full((T * Hq * d + 4096,), 7.0, device="cuda")
    out = guard[:T * Hq * d].view(T, Hq, d)
    go = lambda _: kv.launch_suffix_attention_quant(st.view(), q, gate, out, ws, T, P, query_heads=Hq, scale=scale)
    go(None)
    torch.cuda.synchronize()
    assert torch.isfinite(out).all() and (guard[T * Hq * d:] == 7.0).all()
    k, v = ((x.double().view(H, -1, d // 32, 32) * s.double().unsqueeze(-1)).flatten(2)[:, :P + T]
            for x, s in ((st.key_cache_q8, st.key_scales), (st.value_cache_q8, st.value_scales)))
    num = den = 0.0
    for t0 in range(0, T, 128):
        t1 = min(T, t0 + 128)
        s = torch.einsum("thgd,hld->thgl", q[t0:t1].double().view(t1 - t0, H, G, d), k) * scale
        seen = torch.arange(P + T, device="cuda") <= P + torch.arange(t0, t1, device="cuda")[:, None]
        ref = torch.einsum("thgl,hld->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), v).flatten(1, 2)
        if gated:
            ref = ref * gate[t0:t1].double().sigmoid()
        num, den = num + (out[t0:t1].double() - ref).square().sum().item(), den + ref.square().sum().item()
    grids = captured_grids(go)      # pre-pass, attention, and the merge of a split launch
    splits = grids[1][0] // (-(-T * G // rows_per_cta) * H)
    assert grids[1][0] == splits * -(-T * G // rows_per_cta) * H and len(grids) == (3 if splits > 1 else 2)
    return splits, (num / den) ** 0.5


# operands and weights enter the MMAs as fp16: 2^-11 each, a few 1e-4 of the result's norm; the gate of the other tests of this kernel
GATE = 1e-3


# 8 x 4 heads as served; 152 heads, the second row tile with one row; G = 3, a last CTA whose second row tile holds no rows
@pytest.mark.parametrize("H,G,P,T,splits", [(8, 4, 4000, 1600, 1), (8, 4, 8192, 1200, 3), (8, 4, 4001, 1200, 2), (152, 1, 8000, 129, 2), (50, 3, 6010, 200, 2)])
@pytest.mark.parametrize("act,gated", [(torch.float16, False), (torch.float32, True)])
def test_two_row_tiles(cuda, H, G, P, T, splits, act, gated):
    taken, error = run(128, H, G, P, T, act, gated, 256)
    assert taken == splits and error <= GATE


@pytest.mark.parametrize("d,H,G,T", [(128, 2, 4, 33), (256, 2, 6, 22)])
@pytest.mark.parametrize("positions", [385, 447, 448, 449, 640, 641, 705, 1025])
@pytest.mark.parametrize("act,gated", [(torch.float16, True), (torch.float32, False)])
def test_edges_of_kv_tiles(cuda, d, H, G, T, positions, act, gated):
    taken, error = run(d, H, G, positions - T, T, act, gated, 128)
    assert taken > 1 and error <= GATE
