"""Calls go through ``csrc/host_calls.cpp``: same bits and same errors as the Python path, and no stale descriptor after an
attribute of the node has changed."""
import numpy as np
import pytest

from nnfusion_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,dt,add", [(1, np.float16, False), (3, np.float16, True), (2, np.float32, False),
                                      (40, np.float16, False)])
def test_second_call_equals_first(M, dt, add):
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(11, M, 80, 512, x_dtype=dt)
    op = DequantDot(DeviceWeight.from_host(w), add=add)
    tx = torch.from_numpy(x).cuda()
    kw = dict(addend=torch.ones(M, 80, dtype=tx.dtype, device="cuda")) if add else {}
    first = op(tx, **kw)
    assert op._native is not None
    assert torch.equal(op(tx, **kw), first)
    out = torch.empty_like(first)
    assert op(tx, out=out, **kw) is out and torch.equal(out, first)
    with pytest.raises(ValueError):
        op(tx[:, :256], **kw)
    with pytest.raises(ValueError):
        op(tx, **({} if add else dict(addend=first)))
    op.y_dtype = torch.float32 if dt == np.float16 else torch.float16
    kw = dict(addend=kw["addend"].to(op.y_dtype)) if add else {}
    assert op(tx, **kw).dtype == op.y_dtype and op(tx, **kw).dtype == op.y_dtype


def test_module_keeps_leading_dimensions_and_follows_its_buffers():
    import torch
    from nnfusion_b200.jit import QuantLinear, jit
    x, w = synth.u4g128(12, 6, 48, 256)
    m = jit(QuantLinear.from_host(w).cuda())
    tx = torch.from_numpy(x).cuda().view(2, 3, 256)
    first = m(tx)
    assert first.shape == (2, 3, 48) and torch.equal(m(tx), first)
    assert torch.equal(m(tx.transpose(0, 1)), first.transpose(0, 1))    # not contiguous: the full path
    m.wq = torch.zeros_like(m.wq)
    assert not torch.equal(m(tx), first)


def test_a_node_whose_kernel_and_split_change():
    """Each descriptor has its own workspace: the large-M kernel's partial sums must not be taken for the small-M
    kernel's arrival counters, nor one split's for another's."""
    import torch
    from nnfusion_b200 import _lib as L
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    from oracle import oracle as orc
    from tests.util import TOL_F16, oracle_linear
    x, w = synth.u4g128(13, 8, 512, 10240)
    want = oracle_linear(x, w)
    op = DequantDot(DeviceWeight.from_host(w))
    tx = torch.from_numpy(x).cuda()
    for kernel, split_k in [(L.KERNEL_GEMM, 0), (L.KERNEL_GEMV, 3), (L.KERNEL_GEMV, 5), (L.KERNEL_GEMM, 0),
                            (L.KERNEL_AUTO, 0), (L.KERNEL_GEMV, 3)]:
        op.kernel, op.split_k = kernel, split_k
        for _ in range(2):
            y = torch.full((8, 512), float("nan"), dtype=torch.float16, device="cuda")  # rows nobody writes stay NaN
            op(tx, out=y)
            assert orc.max_rel_err(y.cpu().numpy(), want) <= min(TOL_F16, 2e-3), (kernel, split_k)


def test_an_allocation_that_fails_keeps_its_type():
    """A repeated call whose output does not fit raises torch's out-of-memory error, like the first one."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(14, 4096, 65536, 256)
    op = DequantDot(DeviceWeight.from_host(w))
    tx = torch.from_numpy(x).cuda()
    op(tx)  # 512 MB
    assert op._native is not None
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            op(tx)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert op(tx).shape == (4096, 65536)


def test_calls_after_the_context_was_closed_are_refused():
    """A prepared call must not use the context that its node's Context has given back."""
    import torch
    from nnfusion_b200.attention import DecodeAttention
    from nnfusion_b200.linear import Context, DequantDot, DeviceWeight, NNFB200Error
    ctx = Context(0)
    x, w = synth.u4g128(15, 2, 64, 512)
    op, at = DequantDot(DeviceWeight.from_host(w), ctx=ctx), DecodeAttention(2, 2, 128, 64, ctx=ctx)
    tx, q = torch.from_numpy(x).cuda(), torch.zeros(256, dtype=torch.float16, device="cuda")
    for _ in range(2):
        op(tx)
        at(q, q, q, 3)
    assert op._native is not None and at._native is not None
    torch.cuda.synchronize()
    ctx.close()
    for _ in range(2):
        with pytest.raises(NNFB200Error):
            op(tx)
        with pytest.raises(NNFB200Error):
            at(q, q, q, 3)


def test_a_workspace_that_the_node_lets_go_is_not_used_after():
    """The buffers of prepared calls belong to them: calls give the same result when the node's own table is emptied and
    the memory is asked for by somebody else."""
    import torch
    from nnfusion_b200.attention import DecodeAttention
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(16, 8, 512, 10240)
    op, at = DequantDot(DeviceWeight.from_host(w), split_k=4), DecodeAttention(8, 1, 128, 8192)
    at.k_cache.normal_()
    at.v_cache.normal_()
    tx, q = torch.from_numpy(x).cuda(), torch.ones(1024, dtype=torch.float16, device="cuda")
    first = op(tx), at(q, q[:128], q[:128], 8000)
    sizes = [t.numel() for t in (*op._ws.values(), *at._ws.values())]
    assert min(sizes) > 0
    op._ws.clear()
    at._ws.clear()
    others = [torch.full((n + 256,), 0xAB, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(3)]
    for _ in range(2):
        assert torch.equal(op(tx), first[0]) and torch.equal(at(q, q[:128], q[:128], 8000), first[1])
    assert all(bool((t == 0xAB).all()) for t in others)


def test_module_whose_weights_became_a_parameter():
    import torch
    from nnfusion_b200.jit import QuantLinear, jit
    x, w = synth.u4g128(17, 2, 48, 256)
    m = jit(QuantLinear.from_host(w).cuda())
    tx = torch.from_numpy(x).cuda()
    first = m(tx)
    m.wq = torch.nn.Parameter(m.wq.clone(), requires_grad=False)  # no longer among the buffers
    assert "wq" not in m._buffers
    assert torch.equal(m(tx), first) and torch.equal(m(tx), first)


def test_calls_without_the_extension(monkeypatch):
    import torch
    from nnfusion_b200 import _lib as L
    from nnfusion_b200.attention import DecodeAttention
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(18, 2, 64, 512)
    tx, q = torch.from_numpy(x).cuda(), torch.ones(256, dtype=torch.float16, device="cuda")
    want = DequantDot(DeviceWeight.from_host(w))(tx), DecodeAttention(2, 2, 128, 64)(q, q, q, 0)
    monkeypatch.setattr(L, "_host_calls", False)
    op, at = DequantDot(DeviceWeight.from_host(w)), DecodeAttention(2, 2, 128, 64)
    for _ in range(2):
        assert torch.equal(op(tx), want[0]) and torch.equal(at(q, q, q, 0), want[1])
    assert op._native is None and at._native is None


def test_new_row_counts_take_the_native_path(monkeypatch):
    """A row count or a position that has not been seen costs its plan, not the Python path; and a node's table of row
    counts is bounded."""
    import torch
    from nnfusion_b200.attention import DecodeAttention
    from nnfusion_b200.jit import QuantLinear, jit
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(19, 40, 48, 256)
    dw, tx = DeviceWeight.from_host(w), torch.from_numpy(x).cuda()
    rows = [1, 2, 16, 17, 40]
    with monkeypatch.context() as m:
        m.setattr(DequantDot, "_prepare", lambda self: None)
        want = [DequantDot(dw)(tx[:r]) for r in rows]
    module = jit(QuantLinear.from_host(w).cuda())
    op, at = DequantDot(dw), DecodeAttention(2, 1, 128, 2048)
    monkeypatch.setattr(DequantDot, "run_raw", None)            # the Python path's launch
    for r, y in zip(rows, want):
        assert torch.equal(op(tx[:r]), y) and torch.equal(op(tx[:r]), y) and torch.equal(module(tx[None, :r])[0], y)
    q = torch.ones(256, dtype=torch.float16, device="cuda")
    for position in (0, 40, 500, 2000, 3):                      # no workspace, then one of growing size
        y = at(q, q[:128], q[:128], position)
        assert torch.equal(at(q, q[:128], q[:128], position), y)
    tall = torch.zeros((5000, 256), dtype=torch.float16, device="cuda")
    for r in range(200, 5000):                                  # more lengths than are kept
        op(tall[:r])
    assert torch.equal(op(tx), want[-1])
