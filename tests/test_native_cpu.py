"""The CPython module under the launchers (csrc/python/native.cpp) takes and refuses what the launchers always did; no GPU needed: every
call here ends at an argument."""
import ctypes as C

import pytest
import torch

from miinfer_b200 import kv
from miinfer_b200._lib import View, native

V = View(capacity=8, kv_heads=1, head_dim=128, qblock=32, quant_mode=3)


class LongEnough(C.Structure):
    _fields_ = [("bytes", C.c_uint8 * 256)]


@pytest.mark.parametrize("not_a_view", [None, 7, b"x" * 256, bytearray(256), LongEnough(), (View * 2)(), torch.zeros(256, dtype=torch.uint8), C.byref(V)])
def test_only_a_view_is_a_view(not_a_view):
    t = torch.zeros(1, 128)
    for call in (lambda: kv.launch_kv_store_quant(not_a_view, t, t, None, 1, 0), lambda: kv.launch_decode_attention_quant(not_a_view, t, query_heads=1, scale=1.0, workspace=t),
                 lambda: kv.launch_decode_step(not_a_view, t, t, t, query_heads=1, scale=1.0, workspace=t),
                 lambda: kv.launch_suffix_attention_quant(not_a_view, t, None, t, None, 1, 0, query_heads=1, scale=1.0)):
        with pytest.raises((TypeError, C.ArgumentError)):
            call()
    with pytest.raises(TypeError):
        kv.launch_decode_attention_batched([not_a_view], t, t, 1, t, query_heads=1, scale=1.0, workspace=t)


def test_tensors_have_to_be_contiguous_cuda_tensors():
    t = torch.zeros(1, 128)
    with pytest.raises(ValueError, match="contiguous CUDA tensor"):
        kv.launch_kv_store_quant(V, t, t, None, 1, 0)
    with pytest.raises((TypeError, ValueError)):
        kv.launch_kv_store_quant(V, None, t, None, 1, 0)
    with pytest.raises(TypeError):
        kv.launch_kv_store_quant(V, "key", t, None, 1, 0)
    with pytest.raises(TypeError):
        native.append(V, t)


class NullStream:
    cuda_stream = 0


class Wrapped:
    """A storage that only knows its view."""

    def __init__(self, view):
        self._view = view

    def view(self):
        return self._view


def test_pool_arguments():
    pool = kv.SnapshotPool(granularity=1)
    for tokens, storages in ((iter([1, 2]), []), ([1, 2], None), ([1, 2], iter([])), ([1, "2"], []), ([1, 2], [object()]), ([1, 2], [Wrapped(3)])):
        with pytest.raises((TypeError, AttributeError)):
            pool.capture(tokens, storages, stream=NullStream())
        with pytest.raises((TypeError, AttributeError)):
            pool.restore(tokens, storages, stream=NullStream())
    planes = [torch.zeros(8, 128, dtype=torch.int8), torch.zeros(8, 4, dtype=torch.float16)]
    good = View(key_q8=planes[0].data_ptr(), key_scales=planes[1].data_ptr(), value_q8=planes[0].data_ptr(), value_scales=planes[1].data_ptr(), capacity=8,
                kv_heads=1, head_dim=128, qblock=32, quant_mode=3)
    if not torch.cuda.is_available():   # through every argument, as far as the library
        with pytest.raises(kv.B200KvError, match="no sm_100 device"):
            pool.capture([1, 2], [Wrapped(good)], stream=NullStream())


def test_another_python_or_torch_rebuilds_the_module(monkeypatch, tmp_path):
    from miinfer_b200 import build

    stamp = tmp_path / "_native.stamp"
    monkeypatch.setattr(build, "NATIVE_STAMP", stamp)
    assert build.needs_build()
    stamp.write_text(build.native_stamp())
    assert not build.needs_build()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.needs_build()
