"""Suffix attention at head_dim 128 where a row's reference maximum moves, by more than the 2^8 up to which it may stay, at every tile number modulo four: the output in TMEM is
rescaled between tiles that are under way together.  One and two row tiles a CTA, split and whole, against float64."""
import pytest
import torch

from gpu_util import captured_grids
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu

TILE = 64


def levels(kind, tiles, first):
    """How far up each tile's scores lie, in steps of about 9 (log2).  `steps`: two steps, at tiles `first` and `first + 1`; `growing`: one at each tile."""
    at = torch.arange(tiles, device="cuda", dtype=torch.float32)
    return at if kind == "growing" else (at >= first).float() + (at >= first + 1).float()


# one row tile a CTA: 8 and 66 rows of 2 heads, 128 rows and one more; two: 148 heads of 256 rows and of 129 (the second tile a single row)
@pytest.mark.parametrize("H,G,T", [(2, 4, 2), (2, 3, 22), (1, 1, 129), (148, 1, 256), (148, 1, 129)])
@pytest.mark.parametrize("room", [False, True])      # for the partials of a split launch
@pytest.mark.parametrize("kind,first", [("steps", 1), ("steps", 2), ("steps", 3), ("steps", 4), ("steps", 8), ("growing", 0)])
def test_growing_maxima(cuda, H, G, T, room, kind, first):
    d, tiles, Hq = 128, 13, H * G
    n = tiles * TILE - 5
    P, scale = n - T, d ** -0.5
    g = torch.Generator(device="cuda")
    g.manual_seed(100 * T + first)
    rand = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    level = levels(kind, tiles, first).repeat_interleave(TILE)[:n, None, None]
    # a third of the rows has a maximum that grows by 0.5625 x 128 / sqrt(128) / ln 2 = 9.2 a step, a third one that falls, a third one that stays
    side = (torch.arange(T, device="cuda")[:, None] + torch.arange(Hq, device="cuda")) % 3 - 1.0
    q = (0.3 * rand(T, Hq, d) + side[..., None]).half()
    k = (0.3 * rand(n, H, d) + 0.5625 * level).half()
    # `steps`: values shrink as weights grow, so that tiles on either side of a step have as large a part in the output
    v = (rand(n, H, d) * (1.0 if kind == "growing" else torch.exp2(9.0 - 9.0 * level))).half()
    st = kv.AttentionLayerKvCacheStorage(n, kv.KvCacheQuantMode.kFp16Fp16, kv_heads=H, head_dim=d, qblock=32)
    kv.launch_kv_store_quant(st.view(), k.view(n, H * d), v.view(n, H * d), None, n, 0, rope_mode=kv.RopeMode.NONE)
    ws = kv.prefill_workspace(n, H, d, **(dict(token_count=T, query_heads=Hq) if room else {}))
    out = torch.empty(T, Hq, d, device="cuda")
    go = lambda _: kv.launch_suffix_attention_quant(st.view(), q, None, out, ws, T, P, query_heads=Hq, scale=scale)
    s = torch.einsum("thgd,lhd->thgl", q.double().view(T, H, G, d), k.double()) * scale
    seen = torch.arange(n, device="cuda") <= P + torch.arange(T, device="cuda")[:, None]
    ref = torch.einsum("thgl,lhd->thgd", s.masked_fill(~seen[:, None, None], float("-inf")).softmax(-1), v.double()).flatten(1, 2)
    for _ in range(5):
        out.fill_(float("nan"))
        go(None)
        torch.cuda.synchronize()
        # Row by row.  Queries, keys and values are fp16 as they come; weights are rounded to fp16, 2^-11 each at random, and the sum is of the rounded ones: a few 1e-4 of a row's norm.  A
        # tile whose weights are a step off takes a third of it and more.
        assert ((out.double() - ref).norm(dim=-1) / ref.norm(dim=-1)).max().item() <= 1e-3
    assert len(captured_grids(go)) == (2 if room and H < 148 else 1)      # attention, and the merge of a split launch
