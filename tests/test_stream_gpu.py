"""The small-M form that streams the weights through shared memory (``nnfusion_b200/csrc/dq_stream.cu``: 9 to 16 rows of fp16,
uint4 weights, enough of them): both ends of its rows, ragged N, shares that begin and end inside a
tile, every prologue and epilogue, both output and scale types, and the rule that chooses it, against the oracle."""
import ctypes

import numpy as np
import pytest

from nnfusion_b200 import _lib as L
from nnfusion_b200 import synth
from oracle import oracle as orc
from tests.util import TOL_F16, oracle_linear

pytestmark = pytest.mark.gpu


def _plan_bits(op, M, dtype):
    d, out = op.desc(M, dtype), (ctypes.c_int32 * 8)()
    assert op.ctx.lib.nnf_b200_linear_plan(op.ctx.handle, ctypes.byref(d), ctypes.byref(out)) == L.OK
    return d, out


@pytest.mark.parametrize("M,N,K,group,scale,norm,epilogue,y32", [
    (9, 4100, 11008, 128, np.float16, False, "none", False),     # 33 tiles of 86 units on 296 CTAs, ragged N, odd groups a row
    (16, 4096, 11008, 128, np.float16, False, "add", True),
    (13, 3593, 8192, 128, np.float16, True, "silu", False),      # two weight sets, 57 tiles, odd N
    (16, 4032, 9216, 256, np.float32, True, "silu", True),
    (16, 9001, 9088, 128, np.float16, True, "bias", False),      # 71 tiles of 71 units
    (11, 40000, 4224, 128, np.float16, False, "none", False),    # 313 tiles of 33 units, 35 a CTA: whole tiles too
    (10, 9000, 8704, 0, np.float16, False, "bias", True),        # one group a row
    # halves of K that meet in a cluster's shared memory: not this form, no workspace touched
    (16, 4032, 5120, 256, np.float32, True, "silu", True),
    (16, 9001, 4608, 128, np.float16, True, "bias", False),
    (10, 9000, 6144, 0, np.float16, False, "bias", True),
])
def test_against_the_oracle(M, N, K, group, scale, norm, epilogue, y32):
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(M + N))
    x = synth.make_x(rng, M, K, np.float16)
    w = [synth.make_weights(rng, N, K, 4, group or K, scale) for _ in range(1 + (epilogue == "silu"))]
    gain = rng.uniform(0.9, 1.1, K).astype(np.float32) if norm else None
    bias = rng.standard_normal(N).astype(np.float32) if epilogue == "bias" else None
    op = DequantDot(*[DeviceWeight.from_host(v) for v in w], gain=torch.from_numpy(gain).cuda() if norm else None,
                    bias=torch.from_numpy(bias).cuda() if bias is not None else None, add=epilogue == "add",
                    y_dtype=torch.float32 if y32 else None)
    tx = torch.from_numpy(x).cuda()
    d, out = _plan_bits(op, M, tx.dtype)
    halves = bool(out[2] == 2 and out[7] & 1)
    assert halves == ((N, K) in ((4032, 5120), (9001, 4608), (9000, 6144)))
    assert bool(out[7] & 16) == (not halves)
    c = torch.randn(M, N, device="cuda").to(torch.float32 if y32 else torch.float16) if epilogue == "add" else None
    kw = dict(addend=c) if c is not None else {}
    y = torch.full((M, N), float("nan"), dtype=torch.float32 if y32 else torch.float16, device="cuda")
    op(tx, out=y, **kw)
    outs = [op(tx, **kw) for _ in range(20)]                     # back to back: the same bits, counters left zeroed
    op.ctx.device_status()
    assert all(torch.equal(o, y) for o in outs)
    want = oracle_linear(x, *w, gain=gain, bias=bias, out_dtype=np.float32)
    if c is not None:
        want = want + c.float().cpu().numpy()
    # exact integers, fp32 scales and sums: what is left is x's rounding behind the norm (2^-11 an element) and y's
    assert orc.max_rel_err(y.float().cpu().numpy(), want) <= min(TOL_F16, 1.5e-3 if norm or not y32 else 1e-4)


def test_a_smaller_workspace_takes_the_split_form():
    """A program whose workspace was sized before this form existed keeps running, and nothing is written behind its buffer."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    x, w = synth.u4g128(3, 16, 4096, 11008)
    op = DequantDot(DeviceWeight.from_host(w))
    tx, want = torch.from_numpy(x).cuda(), oracle_linear(x, w)
    d, _ = _plan_bits(op, 16, tx.dtype)
    need = int(op.ctx.lib.nnf_b200_linear_workspace_bytes(op.ctx.handle, ctypes.byref(d)))
    y = torch.empty((16, 4096), dtype=torch.float16, device="cuda")
    d2 = op.desc(16, tx.dtype)
    d2.split_k = 4                                               # what the split form asks for at the same cut
    split = int(op.ctx.lib.nnf_b200_linear_workspace_bytes(op.ctx.handle, ctypes.byref(d2)))
    assert split < need
    for size in (need, split):
        guarded = torch.zeros(size + 4096, dtype=torch.uint8, device="cuda")
        guarded[size:] = 0xAB
        for _ in range(2):
            y.fill_(float("nan"))
            op.run_raw(d, tx.data_ptr(), y.data_ptr(), guarded[:size])
            assert orc.max_rel_err(y.cpu().numpy(), want) <= 1.5e-3
        assert bool((guarded[size:] == 0xAB).all())


def test_activations_gain_and_addend_written_by_the_launch_ahead():
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(5))
    a = DequantDot(DeviceWeight.from_host(synth.make_weights(rng, 11008, 4096, 4, 128)), add=False)
    b = DequantDot(DeviceWeight.from_host(synth.make_weights(rng, 4096, 11008, 4, 128)), add=True)
    xs = [torch.from_numpy(synth.make_x(rng, 16, 4096, np.float16)).cuda() for _ in range(30)]
    h, want = torch.empty((16, 11008), dtype=torch.float16, device="cuda"), []
    for x in xs:
        a(x, out=h)
        torch.cuda.synchronize()
        want.append(b(h, addend=x).clone())
        torch.cuda.synchronize()
    got = []
    for x in xs:
        a(x, out=h)
        got.append(b(h, addend=x))
    torch.cuda.synchronize()
    assert not [i for i, (p, q) in enumerate(zip(got, want)) if not torch.equal(p, q)]


@pytest.mark.parametrize("M,N,K,pair", [(16, 8192, 8192, False), (12, 4032, 5120, True), (16, 4096, 4096, False)])
def test_one_node_on_two_streams(M, N, K, pair):
    """Where K is not cut, or cut in halves that meet in a cluster, a call touches no workspace: overlapping calls of one node
    give what calls one at a time give."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(N + K))
    op = DequantDot(*[DeviceWeight.from_host(synth.make_weights(rng, N, K, 4, 128)) for _ in range(1 + pair)])
    xs = [torch.from_numpy(synth.make_x(rng, M, K, np.float16)).cuda() for _ in range(2)]
    want = [op(x).clone() for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [[torch.empty_like(w) for _ in range(400)] for w in want]
    for i in range(400):
        for x, s, g in zip(xs, streams, got):
            with torch.cuda.stream(s):
                op(x, out=g[i])
    torch.cuda.synchronize()
    op.ctx.device_status()
    for w, g in zip(want, got):
        assert not [i for i, y in enumerate(g) if not torch.equal(y, w)]
    assert all(torch.equal(op(x), w) for x, w in zip(xs, want))


def _both_forms(op, x):
    """The call as the library serves it (the streaming form) and with K cut over CTAs by the small-M kernel, as its planner would."""
    import torch
    M, out = x.shape[0], []
    d, plan = _plan_bits(op, M, x.dtype)
    assert plan[7] & 16
    for split_k in (0, plan[2]):
        d = op.desc(M, x.dtype)
        d.split_k = split_k
        y = torch.full((M, op.w.N), float("nan"), dtype=op.y_dtype or x.dtype, device="cuda")
        op.run_raw(d, x.data_ptr(), y.data_ptr(), op.workspace(d))
        out.append(y)
    op.ctx.device_status()
    return out


@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("M,N,K", [(16, 4096, 11008), (9, 2048, 28672)])
def test_offsets_leave_as_they_came(M, N, K, mean):
    """Weights of q = zp = 0 give exactly 0, and the error against 64 bits is that of the small-M kernel's sums: both let the
    tensor core sum the unpacking's offsets as it sums the products.  (Measured at 16 x 4096 x 11008, of the norm: 1.7e-5, and
    1.5e-4 for activations of mean 1; the forms add up units in another order, hence the twentieth.)"""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(K))
    w = synth.make_weights(rng, N, K, 4, 128)
    w.q[:40], w.zp[:40] = 0, 0
    x = (rng.standard_normal((M, K)) + mean).astype(np.float16)
    stream, split = _both_forms(DequantDot(DeviceWeight.from_host(w), y_dtype=torch.float32), torch.from_numpy(x).cuda())
    assert int(stream[:, :40].count_nonzero()) == 0
    dense = (w.q.reshape(N, -1, 128) - w.zp[:, :, None].astype(np.float64)) * w.scale[:, :, None].astype(np.float64)
    want = x.astype(np.float64) @ dense.reshape(N, K).T
    err = [np.linalg.norm(y.double().cpu().numpy() - want) / np.linalg.norm(want) for y in (stream, split)]
    assert err[0] <= 1.05 * err[1]


@pytest.mark.parametrize("M,N,K,pair", [(16, 37888, 9216, False), (9, 4100, 11008, False), (16, 5000, 11008, True)])
def test_both_forms_on_one_buffer(M, N, K, pair):
    """Calls of one descriptor follow one another on a buffer whichever form they take (the sum over ranks and smaller buffers take
    the split form): each finds its arrival counters zeroed.  296 tiles, one a CTA, among them: none is shared."""
    import torch
    from nnfusion_b200.linear import DequantDot
    gen = torch.Generator(device="cuda").manual_seed(N)
    op = DequantDot(*[_device_weight(gen, N, K) for _ in range(1 + pair)])
    x = torch.randn(M, K, device="cuda", generator=gen).half()
    d, plan = _plan_bits(op, M, x.dtype)
    assert plan[7] & 16
    need = int(op.ctx.lib.nnf_b200_linear_workspace_bytes(op.ctx.handle, ctypes.byref(d)))
    d2 = op.desc(M, x.dtype)
    d2.split_k = plan[2]
    split = int(op.ctx.lib.nnf_b200_linear_workspace_bytes(op.ctx.handle, ctypes.byref(d2)))
    counters = (N + 15) // 16 * 4                                # the split form's, in front
    words = torch.zeros(16384, dtype=torch.int32, device="cuda")
    peer = torch.zeros(2 * M * N, dtype=torch.float32, device="cuda")
    peers = L.Peers(0, 1, (ctypes.c_void_p * 1)(peer.data_ptr()), (ctypes.c_void_p * 1)(words.data_ptr()), M * N * 4, 0)

    def run(ws, streaming):
        y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        if streaming or pair:
            op.run_raw(d, x.data_ptr(), y.data_ptr(), ws if streaming else ws[:split])
        else:
            op.ctx.check(op.ctx.lib.nnf_b200_linear_allreduce(
                op.ctx.handle, torch.cuda.current_stream().cuda_stream, ctypes.byref(d), x.data_ptr(), ctypes.byref(op._abi_w), None,
                y.data_ptr(), ws.data_ptr(), ws.numel(), ctypes.byref(peers)))
        return y

    fresh, ws = torch.zeros(need, dtype=torch.uint8, device="cuda"), torch.zeros(need, dtype=torch.uint8, device="cuda")
    want = {False: run(torch.zeros_like(fresh), False), True: run(fresh, True)}
    assert torch.linalg.vector_norm(want[True].double() - want[False].double()) <= 1e-3 * torch.linalg.vector_norm(want[False].double())
    for streaming in (True, False, True, True, False, False, True):
        assert torch.equal(run(ws, streaming), want[streaming])
        assert int(ws[:counters].count_nonzero()) == 0
    op.ctx.device_status()


def _device_weight(gen, N, K, odd=False):
    """Random weights on the device; odd: scales and zero-points that start 2 bytes and 1 byte past a 16-byte boundary."""
    import torch
    from nnfusion_b200.linear import DeviceWeight
    wq, zp = (torch.randint(0, 256, (N, n), dtype=torch.uint8, device="cuda", generator=gen) for n in (K // 2, (K // 128 + 1) // 2))
    scale = (torch.rand(N, K // 128, device="cuda", generator=gen) * 0.018 + 0.002).half()
    if odd:
        scale, zp = (torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape) for t in (scale, zp))
        assert scale.data_ptr() % 16 == 2 and zp.data_ptr() % 16 == 1
    return DeviceWeight(N, K, 4, 128, wq, scale, zp)


@pytest.mark.parametrize("norm", [False, True])
def test_not_finite_activations_stay_in_their_row(norm):
    """A row with an infinity or a NaN gives what the small-M kernel gives (the offsets' sums make NaN of it), the others what they
    give without it; the largest finite values stay finite where the result is."""
    import torch
    from nnfusion_b200.linear import DequantDot
    gen = torch.Generator(device="cuda").manual_seed(12)
    N, K = 4096, 11008
    op = DequantDot(_device_weight(gen, N, K), gain=torch.rand(K, device="cuda", generator=gen) + 0.5 if norm else None,
                    y_dtype=torch.float32)
    x = torch.randn(12, K, device="cuda", generator=gen).half()
    x[9] = 0
    x[9, 77] = 65504.0
    clean, _ = _both_forms(op, x)
    assert bool(torch.isfinite(clean).all())
    x[2, 4000], x[5, 1], x[8, 11007] = float("inf"), float("nan"), -float("inf")
    stream, split = _both_forms(op, x)
    rows = [2, 5, 8]
    assert torch.equal(torch.isnan(stream), torch.isnan(split)) and not bool(torch.isfinite(stream[rows]).any())
    keep = [m for m in range(12) if m not in rows]
    assert torch.equal(stream[keep], clean[keep])


def test_scales_and_zero_points_off_their_boundaries():
    import torch
    from nnfusion_b200.linear import DequantDot
    N, K = 4100, 11008
    ops = [DequantDot(_device_weight(torch.Generator(device="cuda").manual_seed(3), N, K, odd)) for odd in (False, True)]
    x = torch.randn(9, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).half()
    assert torch.equal(*[_both_forms(op, x)[0] for op in ops])


@pytest.mark.parametrize("M", [16, 48])
def test_two_host_threads_on_one_context(M):
    """Nodes made and called for the first time by two threads at once: the tensor maps of their weights go into the context's
    cache under its lock, and every call gets its own."""
    import threading
    import torch
    from nnfusion_b200.linear import DequantDot
    N, K, nodes = 4096, 11008, 12
    gen = torch.Generator(device="cuda").manual_seed(9)
    weights = [[_device_weight(gen, N, K) for _ in range(nodes)] for _ in range(2)]
    x = torch.randn(M, K, device="cuda", generator=gen).half()
    want = [[DequantDot(w)(x) for w in ws] for ws in weights]
    again = [[_device_weight(gen, 16, K) for _ in range(nodes)] for _ in range(2)]   # (new addresses: new entries)
    torch.cuda.synchronize()
    got, errors, start = [[], []], [], threading.Barrier(2)

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(timeout=30)
                for w, small in zip(weights[i], again[i]):
                    DequantDot(small)(x)
                    got[i].append(DequantDot(w)(x))
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # (shown by the assertion below)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
    assert not errors and not any(t.is_alive() for t in threads)
    assert all(torch.equal(a, b) for p, q in zip(want, got) for a, b in zip(p, q)) and [len(g) for g in got] == [nodes] * 2
