"""The decode kernel that serves every cache mode and shape (csrc/decode_stream.cu), at the edges of its tiles (16
positions), warps, splits and alignments: batched launches, and decode steps with the append fused in."""
import numpy as np
import pytest
import torch

import kvoracle as ko
from gpu_util import assert_planes_equal, captured_parameter_blocks, to_dev, upload
from miinfer_b200 import kv

pytestmark = pytest.mark.gpu
# fp32 sums of products exact to 2^-22 and ex2.approx (2^-22) weights: 1e-5 relative leaves room for a few thousand terms
REL = 1.0e-5


def _filled(rng, L, H, d, qb, mode, cap):
    host = ko.HostCache(cap, H, d, qb, mode)
    host.append(ko.normal_f16(rng, (L, H * d)).astype(np.float32), ko.normal_f16(rng, (L, H * d)).astype(np.float32), None, 0, rope_mode=0)
    return host


def _close(got, ref, what):
    rel = np.linalg.norm(got.astype(np.float64) - ref) / np.linalg.norm(ref)
    assert np.isfinite(got).all() and rel <= REL, (what, rel)


# odd capacities: 2-byte aligned row scales, 8-byte aligned block scales
@pytest.mark.parametrize("d,H,Hq,qb,mode", [(256, 4, 24, 32, 3), (256, 4, 24, 256, 3), (256, 2, 16, 256, 0), (256, 1, 3, 256, 1), (256, 2, 4, 32, 2),
                                            (128, 8, 32, 128, 0), (128, 2, 14, 32, 3), (128, 3, 3, 128, 2), (128, 2, 10, 128, 3), (128, 2, 8, 32, 1)])
def test_batched_lengths_at_tile_and_split_edges(cuda, d, H, Hq, qb, mode):
    rng = np.random.default_rng(d + H + qb + mode)
    lengths = [1, 15, 16, 17, 127, 129, 511, 700]
    hosts = [_filled(rng, n, H, d, qb, mode, n + 1 + n % 3) for n in lengths]
    q16 = ko.normal_f16(rng, (len(lengths), Hq, d), 2.0)
    gate = rng.standard_normal((len(lengths), Hq, d)).astype(np.float32)
    sts, table = [upload(h) for h in hosts], kv.view_table(len(lengths))
    lens, ws = torch.tensor(lengths, dtype=torch.int32, device="cuda"), kv.decode_workspace(Hq, d, len(lengths))
    for q in (to_dev(q16), to_dev(q16.astype(np.float32) * 1.37)):
        for splits in (0, 5, 128):   # 128: more CTAs per session than fit on the device with some shapes, so the merge is a launch of its own
            out, gated = (torch.full((len(lengths), Hq, d), float("nan"), device="cuda") for _ in range(2))
            kv.launch_decode_attention_batched([s.view() for s in sts], table, lens, max(lengths), q, query_heads=Hq, scale=d ** -0.5,
                                               output=out, gate=to_dev(gate), gated_output=gated, workspace=ws, num_splits=splits | kv.FORCE_GENERIC)
            for i, h in enumerate(hosts):
                ref, ref_g = h.decode_ref(q[i].float().cpu().numpy(), d ** -0.5, lengths[i], gate[i])
                _close(out[i].cpu().numpy(), ref, (lengths[i], splits))
                _close(gated[i].cpu().numpy(), ref_g, (lengths[i], splits, "gated"))


@pytest.mark.parametrize("d,H,Hq,qb,mode,dtype", [(256, 4, 24, 256, 0, np.float16), (256, 4, 24, 32, 3, np.float32), (256, 4, 24, 256, 3, np.float32),
                                                  (128, 8, 32, 32, 1, np.float16), (128, 8, 32, 128, 2, np.float32), (128, 8, 32, 32, 3, np.float16)])
def test_fused_append_in_every_mode(cuda, d, H, Hq, qb, mode, dtype):
    rng = np.random.default_rng(7 * d + qb + mode)
    w = (1.0 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    for L0 in (0, 15, 127, 1150):        # the new row first in a tile, last in one, behind many tiles; alone in the cache
        host = _filled(rng, max(L0, 1), H, d, qb, mode, 1211)
        st, ws = upload(host), kv.decode_workspace(Hq, d)
        for step in range(3):
            kn, vn = (rng.standard_normal((1, H * d)).astype(dtype) for _ in range(2))
            q = rng.standard_normal((Hq, d)).astype(dtype)
            pos = L0 + step
            host.append(kn.astype(np.float32), vn.astype(np.float32), w, pos, rope_mode=1 + step % 2)
            out = torch.full((Hq, d), float("nan"), device="cuda")
            kv.launch_decode_step(st.view(), to_dev(kn), to_dev(vn), to_dev(q), query_heads=Hq, scale=d ** -0.5, k_norm_weight=to_dev(w),
                                  rope_mode=kv.RopeMode(1 + step % 2), output=out, workspace=ws, num_splits=kv.FORCE_GENERIC,
                                  **({"position": pos} if step != 1 else {"decode_state": kv.make_decode_state(pos)}))
            ref, _ = host.decode_ref(q.astype(np.float32), d ** -0.5, pos + 1)
            _close(out.cpu().numpy(), ref, (L0, step))
        assert_planes_equal(st, host, f"mode {mode} at {L0}")
    # a device-side position beyond the capacity appends nothing
    before = [t.clone() for t in st.planes()]
    kv.launch_decode_step(st.view(), to_dev(kn), to_dev(vn), to_dev(q), query_heads=Hq, scale=d ** -0.5, rope_mode=kv.RopeMode.NONE, output=out,
                          workspace=ws, decode_state=kv.make_decode_state(1211))
    assert all(torch.equal(a, b) for a, b in zip(before, st.planes())) and torch.isfinite(out).all()


def test_value_scales_that_grow_by_orders_of_magnitude(cuda):
    """The multiplier of the weights is re-chosen, and the sums rescaled, when a later tile's value scales outgrow it."""
    rng = np.random.default_rng(3)
    for d, qb in ((256, 32), (256, 256), (128, 32)):
        L, H, Hq = 700, 2, 8
        host = ko.HostCache(L, H, d, qb, 3)
        v = ko.normal_f16(rng, (L, H * d)).astype(np.float32) * np.logspace(-4, 3, L, dtype=np.float32)[:, None]
        host.append(ko.normal_f16(rng, (L, H * d)).astype(np.float32), v.astype(np.float16).astype(np.float32), None, 0, rope_mode=0)
        st, q16, out = upload(host), ko.normal_f16(rng, (Hq, d)), torch.empty(Hq, d, device="cuda")
        ref, _ = host.decode_ref(q16.astype(np.float32), d ** -0.5, L)
        for splits in (1, 3):
            kv.launch_decode_attention_quant(st.view(), to_dev(q16), query_heads=Hq, scale=d ** -0.5, cache_length=L, output=out,
                                             workspace=kv.decode_workspace(Hq, d), num_splits=splits | kv.FORCE_GENERIC)
            _close(out.cpu().numpy(), ref, (d, qb, splits))


# Against float64 over the cache's own fp16 values; the relative 2-norm error has to stay that of fp32 arithmetic.  Per score a sum of d
# products (rounding about 2^-24 per level of the sum), an exponential of 2^-22 and weights kept to 2^-22: measured 1.5e-7 to 2.4e-7 here,
# and 4.4e-7 where one warp adds up 64 tiles or more (the last two cases); the bounds leave room for another draw of the inputs.  A chain
# of MMAs per score, truncated by the tensor core at every link, came to 3.8e-7 .. 6.2e-7, and one per output over all tiles to 1.4e-6 and 3.3e-6.
@pytest.mark.parametrize("d,H,Hq,L,splits,bound", [(256, 4, 24, 128, 0, 3.2e-7), (256, 4, 24, 1000, 0, 3.2e-7), (256, 4, 24, 6001, 0, 3.2e-7),
                                                   (128, 8, 32, 1000, 0, 2.9e-7), (128, 1, 4, 65536, 8, 6.0e-7), (256, 1, 6, 20011, 1, 6.0e-7)])
@pytest.mark.parametrize("act", [torch.float16, torch.float32])
def test_error_of_fp16_caches_is_that_of_fp32_sums(cuda, d, H, Hq, L, splits, bound, act):
    g = torch.Generator(device="cuda")
    g.manual_seed(L + d)
    st = kv.AttentionLayerKvCacheStorage(L, kv.KvCacheQuantMode.kFp16Fp16, kv_heads=H, head_dim=d, qblock=d)
    st.key_cache.copy_(torch.randn(H, L, d, generator=g, device="cuda"))
    st.value_cache.copy_(torch.randn(H, L, d, generator=g, device="cuda"))
    q = torch.randn(Hq, d, generator=g, device="cuda").to(act)
    out = torch.empty(Hq, d, device="cuda")
    kv.launch_decode_attention_quant(st.view(), q, query_heads=Hq, scale=d ** -0.5, cache_length=L, output=out,
                                     workspace=kv.decode_workspace(Hq, d), num_splits=splits)
    s = torch.einsum("hgd,hld->hgl", q.double().view(H, Hq // H, d), st.key_cache.double().view(H, L, d)) * d ** -0.5
    ref = torch.einsum("hgl,hld->hgd", s.softmax(-1), st.value_cache.double().view(H, L, d)).reshape(Hq, d)
    rel = ((out.double() - ref).norm() / ref.norm()).item()
    assert rel <= bound, rel


# Either side of lengths at which the longest split goes into another round of tiles, a ragged last tile, an explicit number of splits, the append in the
# last split; fp16 caches, so fp32 sums
@pytest.mark.parametrize("d,H,Hq,L,splits", [(128, 8, 32, 4656, 0), (128, 8, 32, 4657, 0), (128, 8, 32, 4700, 0), (256, 4, 24, 9104, 0), (256, 4, 24, 9105, 0),
                                             (128, 8, 32, 2064, 9), (128, 8, 32, 2065, 9), (128, 8, 32, 2065, 8), (128, 1, 1, 40000, 0)])
def test_shorter_last_splits(cuda, d, H, Hq, L, splits):
    g = torch.Generator(device="cuda")
    g.manual_seed(L)
    st = kv.AttentionLayerKvCacheStorage(L + 3, kv.KvCacheQuantMode.kFp16Fp16, kv_heads=H, head_dim=d, qblock=d)
    k, v = (torch.randn(L, H * d, generator=g, device="cuda").half() for _ in range(2))
    q, ws = torch.randn(Hq, d, generator=g, device="cuda").half(), kv.decode_workspace(Hq, d)
    out, stepped = (torch.full((Hq, d), float("nan"), device="cuda") for _ in range(2))
    kv.launch_kv_store_quant(st.view(), k[:-1], v[:-1], None, L - 1, 0, rope_mode=kv.RopeMode.NONE)
    kv.launch_decode_step(st.view(), k[-1], v[-1], q, query_heads=Hq, scale=d ** -0.5, rope_mode=kv.RopeMode.NONE, output=stepped, workspace=ws,
                          position=L - 1, num_splits=splits)
    kv.launch_decode_attention_quant(st.view(), q, query_heads=Hq, scale=d ** -0.5, cache_length=L, output=out, workspace=ws, num_splits=splits)
    K, V = (x.double().view(L, H, 1, d).expand(L, H, Hq // H, d).reshape(L, Hq, d) for x in (k, v))
    ref = torch.einsum("hl,lhd->hd", (torch.einsum("hd,lhd->hl", q.double(), K) * d ** -0.5).softmax(-1), V)
    for o in (stepped, out):
        assert torch.isfinite(o).all() and ((o.double() - ref).norm() / ref.norm()).item() <= REL


# steps from just below to just above the length from which, under launch overlap, one session's last splits are a round of tiles shorter
# (csrc/split_bounds.h: three rounds of 8 x 16 positions per split, 18 and 37 splits)
@pytest.mark.parametrize("d,H,Hq,qb,mode,line", [(128, 8, 32, 128, 0, 4608), (128, 8, 32, 32, 3, 4608), (128, 8, 32, 128, 1, 4608), (256, 4, 24, 256, 3, 9472),
                                                 (256, 4, 24, 32, 2, 9472)])
def test_overlapped_steps_whose_last_splits_are_shorter(cuda, d, H, Hq, qb, mode, line):
    g = torch.Generator(device="cuda")
    g.manual_seed(d + mode)
    below, steps = 3, 8
    L0 = line - below
    k, v = (torch.randn(L0 + steps, H * d, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(steps, Hq, d, generator=g, device="cuda").half()
    states = [kv.make_decode_state(L0 + i) for i in range(steps)]
    results = []
    try:
        for overlap in (0, 1):
            kv.set_launch_overlap(overlap)
            st = kv.AttentionLayerKvCacheStorage(line + 500, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=qb)
            ws, out = kv.decode_workspace(Hq, d), torch.full((steps, Hq, d), float("nan"), device="cuda")
            m, l, acc = (torch.empty(*shape, device="cuda") for shape in ((Hq,), (Hq,), (Hq, d)))
            kv.launch_kv_store_quant(st.view(), k[:L0], v[:L0], None, L0, 0, rope_mode=kv.RopeMode.NONE)
            torch.cuda.synchronize()
            for i in range(steps):   # back to back: copies of step i + 1 start while step i merges
                kv.launch_decode_step(st.view(), k[L0 + i:L0 + i + 1], v[L0 + i:L0 + i + 1], q[i], query_heads=Hq, scale=d ** -0.5, rope_mode=kv.RopeMode.NONE,
                                      output=out[i], workspace=ws, num_splits=kv.FORCE_GENERIC, decode_state=states[i])
            kv.launch_decode_partials(st.view(), q[0], query_heads=Hq, scale=d ** -0.5, range_begin=2, range_end=line + 4, part_m=m, part_l=l, part_acc=acc,
                                      workspace=ws, num_splits=kv.FORCE_GENERIC)
            torch.cuda.synchronize()
            results.append((out.double(), (acc / l[:, None]).double(), st.planes()))
    finally:
        kv.set_launch_overlap(0)
    (out0, part0, planes0), (out1, part1, planes1) = results
    assert all(torch.equal(a, b) for a, b in zip(planes0, planes1))
    assert torch.equal(out0[:below], out1[:below]) and not torch.equal(out0[below:], out1[below:])   # even splits on both sides, then not
    for a, b in ((out0, out1), (part0, part1)):
        assert torch.isfinite(b).all() and ((a - b).norm() / a.norm()).item() <= REL
    # a step above the line, with overlap, against float64 over the rows as the cache holds them
    K, V = (_plane(st, side, line + 1) for side in ("key", "value"))
    s = torch.einsum("hgd,hld->hgl", q[below].double().view(H, Hq // H, d), K) * d ** -0.5
    ref = torch.einsum("hgl,hld->hgd", s.softmax(-1), V).reshape(Hq, d)
    assert ((out1[below] - ref).norm() / ref.norm()).item() <= REL


def _plane(st, side, length):
    """A side's first rows as the cache holds them, in float64: [kv heads][length][head_dim]."""
    q8 = getattr(st, f"{side}_cache_q8")
    if q8 is None:
        return getattr(st, f"{side}_cache")[:, :length].double()
    scales = getattr(st, f"{side}_scales")[:, :length].double()
    return (q8[:, :length].double().unflatten(-1, (scales.shape[-1], -1)) * scales.unsqueeze(-1)).flatten(-2)


@pytest.mark.parametrize("poison", [float("nan"), 3.0])
def test_separate_merge_reads_only_what_its_launch_wrote(cuda, poison):
    """More splits than fit on the device with their merge: the merge kernel follows, and reads all splits of all sessions.  What an
    earlier launch with longer sessions, or anybody else, left in the workspace's plain third must not count."""
    rng = np.random.default_rng(5)
    d, H, Hq = 128, 4, 8
    ws = kv.decode_workspace(Hq, d, 3)
    ws[ws.numel() // 3 * 2 // 256 * 256:].view(torch.float32).fill_(poison)
    for lengths, splits in (([900, 300, 7], 128), ([40, 17, 600], 100), ([1, 500, 16], 128)):
        hosts = [_filled(rng, n, H, d, d, 0, n) for n in lengths]
        sts, q = [upload(h) for h in hosts], ko.normal_f16(rng, (3, Hq, d))
        out = torch.full((3, Hq, d), float("nan"), device="cuda")
        kv.launch_decode_attention_batched([s.view() for s in sts], kv.view_table(3), torch.tensor(lengths, dtype=torch.int32, device="cuda"), max(lengths),
                                           to_dev(q), query_heads=Hq, scale=d ** -0.5, output=out, workspace=ws, num_splits=splits)
        for i, h in enumerate(hosts):
            _close(out[i].cpu().numpy(), h.decode_ref(q[i].astype(np.float32), d ** -0.5, lengths[i])[0], (lengths, splits, i))


# the kernels that a 16-byte aligned call of these shapes takes: the streaming one, the two of int8 at head_dim 256 and 128, and a batch
@pytest.mark.parametrize("d,H,Hq,qb,mode,splits", [(256, 4, 24, 256, 0, 0), (128, 2, 6, 32, 1, 0), (256, 4, 24, 32, 3, 9), (128, 8, 32, 32, 3, 9), (128, 8, 32, 32, 3, 1)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_tensors_that_start_at_any_element(cuda, d, H, Hq, qb, mode, splits, dtype):
    rng = np.random.default_rng(d + mode)
    L, scale = 1000, d ** -0.5
    host = _filled(rng, L, H, d, qb, mode, L)
    st, ws = upload(host), kv.decode_workspace(Hq, d, 2)
    q16, gate = ko.normal_f16(rng, (2, Hq, d)), rng.standard_normal((2, Hq, d)).astype(np.float32)
    at = lambda t, off, n: torch.cat([torch.zeros(off, device="cuda", dtype=t.dtype), t.flatten()[:n]])[off:].view(-1, Hq, d)
    table, lengths = kv.view_table(2), torch.tensor([L, 333], dtype=torch.int32, device="cuda")
    refs = [host.decode_ref(q16[i].astype(np.float32), scale, n, gate[i]) for i, n in enumerate((L, 333))]
    for qoff, goff, ooff in ((1, 0, 0), (3, 1, 1), (0, 1, 0), (0, 0, 1), (4, 2, 2)):
        n = Hq * d
        q, g = to_dev(q16).to(dtype), to_dev(gate)
        out, gated = (torch.full((2 * n + 4,), float("nan"), device="cuda") for _ in range(2))
        one = lambda t: t[ooff:ooff + n].view(Hq, d)
        kv.launch_decode_attention_quant(st.view(), at(q, qoff, n)[0], query_heads=Hq, scale=scale, cache_length=L, output=one(out), gate=at(g, goff, n)[0],
                                         gated_output=one(gated), workspace=ws, num_splits=splits)
        tol = 1e-5 if mode != 3 or qoff * q.element_size() % 16 else 3e-4   # an unaligned query goes to the streaming kernel, others are taken as 15-bit
        for got, ref in ((one(out), refs[0][0]), (one(gated), refs[0][1])):
            err = np.linalg.norm(got.cpu().numpy().astype(np.float64) - ref) / np.linalg.norm(ref)
            assert err <= tol, (qoff, goff, ooff, err)
        two = lambda t: t[ooff:ooff + 2 * n].view(2, Hq, d)
        kv.launch_decode_attention_batched([st.view(), st.view()], table, lengths, L, at(q, qoff, 2 * n), query_heads=Hq, scale=scale, output=two(out),
                                           gate=at(g, goff, 2 * n), gated_output=two(gated), workspace=ws, num_splits=splits)
        for i in range(2):
            for got, ref in ((two(out)[i], refs[i][0]), (two(gated)[i], refs[i][1])):
                err = np.linalg.norm(got.cpu().numpy().astype(np.float64) - ref) / np.linalg.norm(ref)
                assert err <= 3e-4, (qoff, goff, ooff, i, err)
        m, l = (torch.empty(Hq, device="cuda") for _ in range(2))
        kv.launch_decode_partials(st.view(), at(q, qoff, n)[0], query_heads=Hq, scale=scale, range_begin=0, range_end=L, part_m=m, part_l=l,
                                  part_acc=one(out), workspace=ws, num_splits=splits)
        got = (one(out) / l[:, None]).cpu().numpy()
        assert np.linalg.norm(got.astype(np.float64) - refs[0][0]) / np.linalg.norm(refs[0][0]) <= 3e-4, (qoff, ooff, "partials")


@pytest.mark.parametrize("d,H,Hq,qb,mode", [(256, 4, 24, 256, 0), (128, 8, 32, 32, 3), (256, 4, 24, 32, 3), (128, 2, 4, 128, 1)])
@pytest.mark.parametrize("fused", [True, False])
def test_steps_on_one_cache_back_to_back_with_launch_overlap(cuda, d, H, Hq, qb, mode, fused):
    """Few CTAs per launch, so that several launches are resident at once: a step may read rows early only if they are older than the row
    of the appending launch before it, which is the only one that may be unfinished.  Same bits as without overlap."""
    g = torch.Generator(device="cuda")
    g.manual_seed(d + mode)
    L0, steps = 30, 100
    k, v = (torch.randn(L0 + steps, H * d, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(steps, Hq, d, generator=g, device="cuda").half()
    results = []
    try:
        for overlap in (0, 1):
            kv.set_launch_overlap(overlap)
            st, ws, out = kv.AttentionLayerKvCacheStorage(L0 + steps, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=qb), kv.decode_workspace(Hq, d), torch.empty(steps, Hq, d, device="cuda")
            kv.launch_kv_store_quant(st.view(), k[:L0], v[:L0], None, L0, 0, rope_mode=kv.RopeMode.NONE)
            torch.cuda.synchronize()
            for i in range(steps):
                pos, common = L0 + i, dict(query_heads=Hq, scale=d ** -0.5, output=out[i], workspace=ws)
                if fused:
                    kv.launch_decode_step(st.view(), k[pos:pos + 1], v[pos:pos + 1], q[i], position=pos, rope_mode=kv.RopeMode.NONE, **common)
                else:
                    kv.launch_kv_store_quant(st.view(), k[pos:pos + 1], v[pos:pos + 1], None, 1, pos, rope_mode=kv.RopeMode.NONE)
                    kv.launch_decode_attention_quant(st.view(), q[i], cache_length=pos + 1, **common)
            torch.cuda.synchronize()
            results.append([out, *st.planes()])
    finally:
        kv.set_launch_overlap(0)
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("d,qb,mode", [(256, 32, 0), (128, 32, 0), (256, 32, 2), (256, 256, 2), (128, 32, 2)])
@pytest.mark.parametrize("splits", [0, 1])
def test_infinities_stay_where_they_are(cuda, d, qb, mode, splits):
    """fp16 K, V in fp16 or int8: an infinite value (or value scale) makes its own dims infinite for the heads that see it and nothing else; a
    score of minus infinity takes its position out; one of plus infinity, or a NaN key, makes the head NaN.  As plain arithmetic does."""
    rng = np.random.default_rng(d + qb)
    L, H, Hq = 70, 2, 8
    k, v, q = rng.standard_normal((H, L, d)), rng.standard_normal((H, L, d)), rng.standard_normal((Hq, d))
    k[0, 5, 3] = -np.inf                                     # kv head 0: query heads 0 and 1 ignore position 5, 2 and 3 become NaN
    q[:2, 3], q[2:4, 3] = np.abs(q[:2, 3]), -np.abs(q[2:4, 3])
    st = kv.AttentionLayerKvCacheStorage(L, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=qb if mode else d)
    st.key_cache.copy_(torch.from_numpy(k))
    if mode == 0:
        st.value_cache.copy_(torch.from_numpy(v))
        st.value_cache[0, 40, 7], st.value_cache[1, 66, d - 1] = float("inf"), -float("inf")
        vd = st.value_cache.double()
    else:
        st.value_cache_q8.copy_(torch.from_numpy(np.clip(np.rint(v * 40), -127, 127)))
        st.value_cache_q8[st.value_cache_q8 == 0] = 1
        st.value_scales.fill_(1 / 40)
        st.value_scales[0, 40, 0], st.value_scales[1, 66, -1] = float("inf"), float("inf")
        vd = (st.value_cache_q8.double().view(H, L, d // st.qblock, -1) * st.value_scales.double().unsqueeze(-1)).view(H, L, d)
    q16 = torch.from_numpy(q).half().cuda()
    out = torch.empty(Hq, d, device="cuda")
    kv.launch_decode_attention_quant(st.view(), q16, query_heads=Hq, scale=d ** -0.5, cache_length=L, output=out,
                                     workspace=kv.decode_workspace(Hq, d), num_splits=splits | kv.FORCE_GENERIC)
    kd = st.key_cache.double()
    ref = torch.cat([((q16.double().view(H, Hq // H, d)[h, :, None, :] * kd[h]).sum(-1) * d ** -0.5).softmax(-1)[..., None].mul(vd[h]).sum(1) for h in range(H)])
    got = out.double()
    assert torch.equal(got.isnan(), ref.isnan()) and bool(ref.isnan().any())
    assert torch.equal(got.isinf(), ref.isinf()) and torch.equal(got[got.isinf()], ref[ref.isinf()]) and bool(ref.isinf().any())
    ok = ref.isfinite()
    assert bool((got[ok] - ref[ok]).norm() <= REL * ref[ok].norm())   # none are finite where every dim shares one infinite scale


@pytest.mark.parametrize("d,H,Hq,qb,mode", [(256, 4, 24, 256, 0), (256, 4, 24, 32, 3), (128, 8, 32, 128, 0)])
def test_workspaces_that_hold_the_plain_partials_are_enough(cuda, d, H, Hq, qb, mode):
    """head_dim + 2 floats per split and head in the last third; the in-launch merge needs a little more in front of it at head_dim 256, and a
    launch that is short of it runs its merge behind.  A launch that chooses its splits fits them to what is there."""
    rng = np.random.default_rng(d + mode)
    host = _filled(rng, 1500, H, d, qb, mode, 1501)          # odd: no kernel with a workspace rule of its own
    st, q = upload(host), ko.normal_f16(rng, (Hq, d))
    ref, _ = host.decode_ref(q.astype(np.float32), d ** -0.5, 1500)
    room = lambda n: n - n // 3 * 2 // 256 * 256
    for splits, fits in ((5, 5), (0, 1), (0, 3)):
        need = fits * Hq * (d + 2) * 4
        size = next(n for n in range(need, 4 * need) if room(n) >= need)
        out = torch.empty(Hq, d, device="cuda")
        go = lambda ws: kv.launch_decode_attention_quant(st.view(), to_dev(q), query_heads=Hq, scale=d ** -0.5, cache_length=1500, output=out,
                                                         workspace=ws, num_splits=splits)
        go(torch.zeros(size, dtype=torch.uint8, device="cuda"))
        _close(out.cpu().numpy(), ref, (splits, fits))
        short = next(n for n in range(size, 0, -1) if room(n) < Hq * (d + 2) * 4 * max(splits, 1))
        with pytest.raises(kv.B200KvError):
            go(torch.zeros(short, dtype=torch.uint8, device="cuda"))


@pytest.mark.parametrize("d,H,Hq,qb,mode", [(256, 4, 24, 32, 3), (128, 8, 32, 32, 3), (128, 2, 8, 128, 0)])
def test_the_separate_merge_can_be_asked_for(cuda, d, H, Hq, qb, mode):
    """Stage 1 and the merge kernel: two launches, and no word of the workspace's tagged part is touched (it may even hold garbage)."""
    rng = np.random.default_rng(d)
    L, lengths = 1500, [1500, 40]
    host = _filled(rng, L, H, d, qb, mode, 1504)
    st, ws = upload(host), kv.decode_workspace(Hq, d, 2)
    tagged = ws[:ws.numel() // 3 * 2 // 256 * 256]
    tagged.fill_(171)
    q, out = ko.normal_f16(rng, (2, Hq, d)), torch.empty(2, Hq, d, device="cuda")
    table, lens = kv.view_table(2), torch.tensor(lengths, dtype=torch.int32, device="cuda")
    for splits in (0, 3, 65535):
        for i, n in enumerate(lengths):
            kv.launch_decode_attention_quant(st.view(), to_dev(q[i]), query_heads=Hq, scale=d ** -0.5, cache_length=n, output=out[i], workspace=ws,
                                             num_splits=splits | kv.SEPARATE_MERGE)
        one = out.clone()
        kv.launch_decode_attention_batched([st.view(), st.view()], table, lens, L, to_dev(q), query_heads=Hq, scale=d ** -0.5, output=out, workspace=ws,
                                           num_splits=splits | kv.SEPARATE_MERGE)
        for got in (one, out):
            for i, n in enumerate(lengths):
                ref, _ = host.decode_ref(q[i].astype(np.float32), d ** -0.5, n)
                err = np.linalg.norm(got[i].cpu().numpy().astype(np.float64) - ref) / np.linalg.norm(ref)
                assert err <= 2e-4, (splits, n, err)
    assert bool((tagged == 171).all())


@pytest.mark.parametrize("d,H,Hq,mode,splits,path", [(128, 8, 32, 0, 3, 0), (256, 4, 24, 0, 3, 0), (256, 4, 24, 3, 3, 0), (128, 8, 32, 3, 3, 0), (128, 8, 32, 3, 3, 1)])
def test_a_launch_that_writes_nothing_gated_is_given_no_gate(cuda, d, H, Hq, mode, splits, path):
    """What a launch does not get it cannot read: the gate's address is in the parameters of launches with a gated output and of no others (only captured)."""
    L = 1504
    st = kv.AttentionLayerKvCacheStorage(L, kv.KvCacheQuantMode(mode), kv_heads=H, head_dim=d, qblock=32 if mode else d)
    q, k = torch.zeros(2, Hq, d, device="cuda", dtype=torch.float16), torch.zeros(1, H * d, device="cuda", dtype=torch.float16)
    gate, out, ws = torch.zeros(2, Hq, d, device="cuda"), torch.zeros(2, Hq, d, device="cuda"), kv.decode_workspace(Hq, d, 2)
    table, lengths, views = kv.view_table(2), torch.tensor([L, 300], dtype=torch.int32, device="cuda"), [st.view(), st.view()]
    common = dict(query_heads=Hq, scale=d ** -0.5, gate=gate, workspace=ws, num_splits=splits)
    kv.set_decode_kernel(path)
    try:
        kv.launch_decode_attention_batched(views, table, lengths, L, q, output=out, **common)   # fills the table
        torch.cuda.synchronize()
        calls = [lambda **o: kv.launch_decode_attention_quant(st.view(), q[0], cache_length=L, **common, **o),
                 lambda **o: kv.launch_decode_step(st.view(), k, k, q[0], position=L - 1, **common, **o),
                 lambda **o: kv.launch_decode_attention_batched(None, table, lengths, L, q, **common, **o)]
        for call in calls:
            for outputs, wanted in ((dict(output=out), False), (dict(gated_output=out), True)):
                blocks = captured_parameter_blocks(lambda stream: call(**outputs))
                assert len(blocks) == 1   # the merge is inside
                assert (gate.data_ptr().to_bytes(8, "little") in blocks[0]) == wanted
    finally:
        kv.set_decode_kernel(0)
