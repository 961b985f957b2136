"""The pre-pass of the tcgen05 suffix attention: the fp16 copy of the visible cache rows in the workspace, bit for bit."""
import pytest
import torch

from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


def planes(st, rows):
    """fp16 rows [kv_head][row][d] of K and V: fp16 sides as they are, int8 times scale with the one rounding to fp16."""
    out = []
    for data, f16, scales in ((st.key_cache_q8, st.key_cache, st.key_scales), (st.value_cache_q8, st.value_cache, st.value_scales)):
        if f16 is not None:
            out.append(f16[:, :rows])
        else:
            x = (data.float().view(*scales.shape, -1) * scales.float().unsqueeze(-1)).half().flatten(2)   # 8 x 11 bits: the fp32 product is exact
            out.append(x[:, :rows])
    return torch.stack(out)


# a block converts 64 (head_dim 256) or 128 rows: one row, edges of that and of the 64-row tile, ahead of the chunk up to any row; odd capacities
@pytest.mark.parametrize("d,H", [(128, 3), (256, 2)])
@pytest.mark.parametrize("mode,blocks", [(3, True), (3, False), (0, False), (1, True), (2, False)])
@pytest.mark.parametrize("P,T,prepared", [(0, 1, 0), (63, 1, 63), (64, 1, 1), (127, 2, 100), (128, 65, 128), (1000, 37, 777)])
def test_fp16_copy(cuda, d, H, mode, blocks, P, T, prepared):
    rows, G = P + T, 2
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * P + 10 * T + mode)
    st = kv.AttentionLayerKvCacheStorage(rows + 5, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=32 if blocks else d)
    k, v = (torch.randn(rows, H * d, generator=g, device="cuda").half() for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k, v, None, rows, 0, rope_mode=kv.RopeMode.NONE)
    ws = kv.prefill_workspace(rows, H, d, token_count=T, query_heads=H * G)
    ws.view(torch.uint8).fill_(0xFF)      # 0xFFFF is a NaN in fp16
    scratch_rows = (rows + 63) // 64 * 64
    first = -ws.data_ptr() % 1024
    scratch = ws.view(torch.uint8)[first:first + 4 * H * scratch_rows * d].view(torch.float16).view(2, H, scratch_rows, d)
    want = planes(st, rows)
    kv.prepare_suffix_attention(st.view(), prepared, rows, ws)
    torch.cuda.synchronize()
    assert torch.equal(scratch[:, :, :prepared].view(torch.int16), want[:, :, :prepared].view(torch.int16))
    assert scratch[:, :, prepared:].isnan().all()
    q, out = torch.randn(T, H * G, d, generator=g, device="cuda"), torch.empty(T, H * G, d, device="cuda")
    kv.launch_suffix_attention_quant(st.view(), q, None, out, ws, T, P, query_heads=H * G, scale=d ** -0.5, prepared_rows=prepared)
    torch.cuda.synchronize()
    assert torch.equal(scratch[:, :, :rows].view(torch.int16), want.view(torch.int16))
    assert (scratch[:, :, rows:] == 0).all()
