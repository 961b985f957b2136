"""The store kernel where its launch shape changes (how many units a warp takes, and how many CTAs an SM) and with pointers that are aligned for elements only,
bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import kvoracle as ko
from gpu_util import assert_planes_equal, captured_grids, device_storage_like
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu


def run(d, H, qb, mode, rope, T, base, dtype, offset):
    rng = np.random.default_rng(T + d)
    k, v = (rng.standard_normal((T, H * d), dtype=np.float32).astype(dtype) for _ in range(2))
    w = (1.0 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    host = ko.HostCache(base + T, H, d, qb, mode)
    host.append(k.astype(np.float32), v.astype(np.float32), w, base, rope_mode=rope, trig_mode=1)
    st = device_storage_like(host)

    def place(x):   # `offset` elements behind a 16-byte boundary
        buf = torch.empty(x.size + offset, dtype=torch.from_numpy(x).dtype, device="cuda")
        buf[offset:] = torch.from_numpy(x).cuda().flatten()
        return buf[offset:]
    kd, vd, wd = place(k), place(v), place(w)
    go = lambda _: kv.launch_kv_store_quant(st.view(), kd, vd, wd, T, base, rope_mode=kv.RopeMode(rope))
    go(None)
    torch.cuda.synchronize()
    assert_planes_equal(st, host, f"d={d} H={H} T={T} offset={offset}")
    return captured_grids(go)[0][0]


# two units a token; the lines lie at 2 x 16, 2 x 20 and 4 x 16 warps' worth an SM
@pytest.mark.parametrize("d,H", [(128, 1), (256, 3)])
@pytest.mark.parametrize("units,ctas", [(2 * 16, 8), (2 * 16 + 1, 10), (2 * 20, 10), (2 * 20 + 1, 8), (4 * 16, 8), (4 * 16 + 1, 10)])
def test_launch_shapes(cuda, d, H, units, ctas):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T = (units // 4 * 4 * sms + 1) // 2 + (1 if units % 4 else 0)     # at the line, or one token past it
    assert run(d, H, 32, 3, 1 if d == 128 else 2, T, 3, np.float16, 0) == sms * ctas


@pytest.mark.parametrize("d,H,qb,mode,rope", [(128, 9, 32, 3, 1), (256, 5, 32, 3, 1), (256, 4, 256, 3, 2), (128, 3, 32, 1, 2), (256, 2, 256, 2, 1)])
@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("T", [1, 2, 75])
def test_alignment(cuda, d, H, qb, mode, rope, dtype, offset, T):
    run(d, H, qb, mode, rope, T, 11, dtype, offset)
