"""Helpers shared by the GPU parity tests: move a host (oracle) cache to a device
storage object and back."""
import numpy as np
import torch

import kvoracle as ko
from miinfer_b200 import kv

PLANES = [("key_f16", "key_cache"), ("value_f16", "value_cache"), ("key_q8", "key_cache_q8"),
          ("key_scales", "key_scales"), ("value_q8", "value_cache_q8"), ("value_scales", "value_scales")]


def device_storage_like(host: ko.HostCache) -> kv.AttentionLayerKvCacheStorage:
    return kv.AttentionLayerKvCacheStorage(host.capacity, kv.KvCacheQuantMode(host.quant_mode), kv_heads=host.kv_heads,
                                           head_dim=host.head_dim, qblock=host.qblock)


def upload(host: ko.HostCache) -> kv.AttentionLayerKvCacheStorage:
    st = device_storage_like(host)
    for hname, dname in PLANES:
        h = getattr(host, hname)
        if h is None:
            continue
        t = getattr(st, dname)
        src = torch.from_numpy(h.view(np.int16) if h.dtype == np.uint16 else h)
        t.copy_(src.view(t.dtype) if t.dtype != src.dtype else src)
    return st


def plane_bits(st: kv.AttentionLayerKvCacheStorage, dname: str) -> np.ndarray:
    t = getattr(st, dname)
    if t.dtype == torch.float16:
        return t.view(torch.int16).cpu().numpy().view(np.uint16)
    return t.cpu().numpy()


def assert_planes_equal(st: kv.AttentionLayerKvCacheStorage, host: ko.HostCache, what: str = "") -> None:
    for hname, dname in PLANES:
        h = getattr(host, hname)
        if h is None:
            assert getattr(st, dname) is None
            continue
        got = plane_bits(st, dname)
        if not np.array_equal(got, h):
            bad = np.argwhere(got != h)
            raise AssertionError(f"{what} plane {hname}: {len(bad)} of {h.size} elements differ, first at {bad[0]}: "
                                 f"gpu {got[tuple(bad[0])]} oracle {h[tuple(bad[0])]}")


def to_dev(a: np.ndarray, dtype=None) -> torch.Tensor:
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


def attention_error(got: np.ndarray, ref: np.ndarray):
    """(max-abs, relative L2) of an attention output against the oracle's."""
    diff = got.astype(np.float64) - ref.astype(np.float64)
    return float(np.max(np.abs(diff))), float(np.linalg.norm(diff) / max(np.linalg.norm(ref.astype(np.float64)), 1e-30))


def assert_attention_close(got: np.ndarray, ref: np.ndarray, what: str, tol_abs: float = 2.0e-3, tol_rel: float = 1.0e-3):
    """Two gates: the absolute one the path's specification states (max-abs 2e-3 against the fp32-accumulated
    reference) and a relative one (relative L2), because at long contexts the outputs themselves are of the order
    of 1e-2 and the absolute gate alone would pass a visibly wrong result.  The measured errors are printed."""
    assert np.isfinite(got).all(), f"{what}: non-finite output"
    max_abs, rel_l2 = attention_error(got, ref)
    print(f"[parity] {what}: max_abs {max_abs:.3e} rel_l2 {rel_l2:.3e} (output std {float(np.std(ref)):.3e})")
    assert max_abs <= tol_abs, f"{what}: max-abs error {max_abs:.3e} > {tol_abs}"
    assert rel_l2 <= tol_rel, f"{what}: relative L2 error {rel_l2:.3e} > {tol_rel}"
    return max_abs, rel_l2


def _captured_nodes(call):
    """The CUDA driver and the handles of the nodes that `call(stream)` captures; nothing runs."""
    import ctypes as C

    cu = C.CDLL("libcuda.so.1")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        call(torch.cuda.current_stream().cuda_stream)
    raw, n = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t()
    assert cu.cuGraphGetNodes(raw, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(raw, nodes, C.byref(n)) == 0
    return graph, cu, [C.c_void_p(node) for node in nodes]


def captured_node_types(call):
    """Types of the nodes that `call(stream)` captures (0 = kernel, 1 = memcpy); nothing runs."""
    import ctypes as C

    graph, cu, nodes = _captured_nodes(call)
    kind = C.c_int()
    return [kind.value for node in nodes if cu.cuGraphNodeGetType(node, C.byref(kind)) == 0]


def _captured_kernel_nodes(call):
    import ctypes as C

    class KernelNode(C.Structure):   # CUDA_KERNEL_NODE_PARAMS_v2
        _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.POINTER(C.c_void_p)), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]

    graph, cu, nodes = _captured_nodes(call)
    kernels = []
    for node in nodes:
        k = KernelNode()
        assert cu.cuGraphKernelNodeGetParams_v2(node, C.byref(k)) == 0
        kernels.append(k)
    return graph, cu, kernels


def captured_kernels(call):
    """Mangled names of the kernels that `call(stream)` captures; nothing runs."""
    import ctypes as C

    graph, cu, kernels = _captured_kernel_nodes(call)
    names = []
    for k in kernels:
        name = C.c_char_p()
        rc = cu.cuFuncGetName(C.byref(name), C.c_void_p(k.func)) if k.func else cu.cuKernelGetName(C.byref(name), C.c_void_p(k.kern))
        assert rc == 0
        names.append(name.value.decode())
    return names


def captured_grids(call):
    """Grid sizes of the kernels that `call(stream)` captures; nothing runs."""
    return [tuple(k.dims[:3]) for k in _captured_kernel_nodes(call)[2]]


def captured_parameter_blocks(call):
    """The first parameter, as bytes, of every kernel that `call(stream)` captures; nothing runs."""
    import ctypes as C

    graph, cu, kernels = _captured_kernel_nodes(call)
    blocks = []
    for k in kernels:
        offset, size = C.c_size_t(), C.c_size_t()
        info, handle = (cu.cuFuncGetParamInfo, k.func) if k.func else (cu.cuKernelGetParamInfo, k.kern)
        assert info(C.c_void_p(handle), C.c_size_t(0), C.byref(offset), C.byref(size)) == 0
        blocks.append(C.string_at(k.params[0], size.value))
    return blocks
