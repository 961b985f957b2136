"""The tcgen05 decode kernels' softmax at its edges: maxima that grow with every tile or never, weights that are all one (the top of the fixed-point range), rows of zeros,
and one head of NaN, against float64."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,H,G", [(128, 2, 4), (256, 2, 6), (256, 1, 4)])
@pytest.mark.parametrize("qblock", [32, 0])
@pytest.mark.parametrize("kind", ["growing", "falling", "equal", "zeros", "nan", "one"])
@pytest.mark.parametrize("n", [1, 128, 129, 1400])
def test_weights(cuda, d, H, G, qblock, kind, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    st = kv.AttentionLayerKvCacheStorage((n + 63) // 64 * 64, kv.KvCacheQuantMode.kQ8Q8, kv_heads=H, head_dim=d, qblock=qblock or d)
    q = torch.randn(H * G, d, generator=g, device="cuda").half()
    k, v = (torch.randn(n, H, d, generator=g, device="cuda") for _ in range(2))
    towards = q.float().view(H, G, d)[:, 0] / d ** 0.5      # a key along the first head's query
    at = torch.arange(n, device="cuda", dtype=torch.float32)[:, None, None] / max(n - 1, 1)
    if kind == "growing":
        k = k * 0.1 + at * 6.0 * towards
    elif kind == "falling":
        k = k * 0.1 + (1.0 - at) * 6.0 * towards
    elif kind == "equal":
        k = k[:1].expand(n, H, d)
    elif kind == "zeros":
        k, v = torch.zeros_like(k), torch.cat([v[: n // 2], torch.zeros_like(v[n // 2:])])
    elif kind == "one":
        k = torch.cat([k[: n - 1] * 0.01 - towards, 40.0 * towards[None]])
    kv.launch_kv_store_quant(st.view(), k.reshape(n, H * d).contiguous(), v.reshape(n, H * d).contiguous(), None, n, 0, rope_mode=kv.RopeMode.NONE)
    if kind == "nan" and d == 256:
        pytest.skip("this kernel quantises a head of NaN as zeros")
    if kind == "nan":
        q[1] = float("nan")      # (a lone NaN among a head's elements is quantised as a zero)
    out = torch.empty(H * G, d, device="cuda")
    splits = min(3, -(-n // 128))       # a split count given: the tcgen05 kernels
    kv.launch_decode_attention_quant(st.view(), q, query_heads=H * G, scale=d ** -0.5, cache_length=n, output=out, workspace=kv.decode_workspace(H * G, d), num_splits=splits)
    torch.cuda.synchronize()
    deq = lambda x, s: (x.double().view(*s.shape, -1) * s.double().unsqueeze(-1)).flatten(2)[:, :n]
    kd, vd = deq(st.key_cache_q8, st.key_scales), deq(st.value_cache_q8, st.value_scales)
    w = (torch.einsum("hgd,hld->hgl", q.double().view(H, G, d), kd) * d ** -0.5).softmax(-1)
    ref = torch.einsum("hgl,hld->hgd", w, vd).flatten(0, 1)
    if kind == "nan":
        assert out[1].isnan().all() and out[torch.arange(H * G) != 1].isfinite().all()
        keep = torch.arange(H * G) != 1
        out, ref = out[keep], ref[keep]
    # Query elements are rounded by at most half of amax / 16319, so scores are off by 2^-15 amax times the sum of |k| times the scale (random signs: its root mean
    # square), here up to 1e-3, and weights by the same share; values enter at 2^-16 of the tile's largest.
    assert (out.double() - ref).norm().item() <= 1e-3 * ref.norm().item() + 1e-6
