"""What a node keeps between calls, without a device: a stand-in for the library answers size queries."""
import ctypes
import sys
import types

import pytest
import torch

from nnfusion_b200 import _lib as L
from nnfusion_b200.linear import DequantDot, DeviceWeight


class _FakeLib:
    """Workspace queries of the C ABI: a size per kernel and split, nothing is launched."""

    def nnf_b200_linear_workspace_bytes(self, handle, d):
        d = d._obj
        return 4096 + 256 * d.split_k + (8192 if d.kernel == L.KERNEL_GEMM else 0)

    def nnf_b200_workspace_reset(self, handle, stream, address, nbytes):
        return L.OK


@pytest.fixture
def node(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(cuda_stream=0))
    w = DeviceWeight(32, 256, 4, 128, torch.zeros((32, 128), dtype=torch.uint8), torch.ones((32, 2), dtype=torch.float16),
                     torch.zeros((32, 1), dtype=torch.uint8))
    ctx = types.SimpleNamespace(lib=_FakeLib(), handle=None, check=lambda rc: None)
    return DequantDot(w, ctx=ctx)


@pytest.mark.parametrize("name,value", [("kernel", L.KERNEL_GEMM), ("split_k", 2), ("y_dtype", torch.float32)])
def test_a_workspace_serves_one_descriptor(node, name, value):
    """Counters must start at zero and another descriptor's partial sums may lie where they are, so a changed attribute
    takes a buffer of its own (and finds the first one again when it is changed back)."""
    before = getattr(node, name)
    first = node.workspace(node.desc(8, torch.float16))
    assert node.workspace(node.desc(8, torch.float16)) is first
    setattr(node, name, value)
    other = node.workspace(node.desc(8, torch.float16))
    assert other is not first and other.data_ptr() != first.data_ptr()
    setattr(node, name, before)
    assert node.workspace(node.desc(8, torch.float16)) is first


def test_prepared_calls_refuse_descriptors_of_another_size():
    """Sizes are checked before anything is copied out of the buffers."""
    host = L.host_calls()
    with pytest.raises(ValueError):
        host.LinearCall(0, ctypes.c_void_p(), b"\0" * 8, None, 0, None, None, None, 16, 128)
    with pytest.raises(ValueError):
        host.AttnCall(0, 0, ctypes.c_void_p(), b"\0" * 8, None, None)
    with pytest.raises(ValueError):
        host.LinearCall(0, b"four", b"\0" * 24, None, 0, None, None, None, 16, 128)


def test_prepared_calls_keep_their_workspaces_alive():
    """Whatever becomes of the node's own reference, the address that a later call hands over stays that tensor's."""
    host = L.host_calls()
    t = torch.zeros(256, dtype=torch.uint8)
    held = sys.getrefcount(t)
    attention = host.AttnCall(0, 0, ctypes.c_void_p(), bytes(L.AttnDesc()), t, None)
    assert sys.getrefcount(t) == held + 1
    del attention
    assert sys.getrefcount(t) == held
    with pytest.raises(ValueError):
        host.AttnCall(0, 0, ctypes.c_void_p(), bytes(L.AttnDesc()), torch.zeros(8), None)  # not bytes


def test_a_missing_extension_costs_host_time_only(monkeypatch):
    """The C library alone suffices: no call fails, least of all after its launch has been issued."""
    monkeypatch.setattr(L, "_host_calls", None)
    monkeypatch.setitem(sys.modules, "nnfusion_b200._host_calls", None)     # the import raises
    monkeypatch.delattr("nnfusion_b200._host_calls", raising=False)
    with pytest.warns(RuntimeWarning, match="_host_calls.so"):
        assert L.host_calls() is None
    assert L.host_calls() is None
