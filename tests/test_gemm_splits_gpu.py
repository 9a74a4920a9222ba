"""How the large-M kernel's tiles meet the pairs of CTAs (``gemm_layout`` in ``nnfusion_b200/csrc/dq_gemm_tcgen05.cu``):
K shared by the 2, 3 or 4 pairs of a cluster, seam shares through the workspace, several whole tiles a pair, at the edges
of batch tiles (16, 128, 256), of weight tiles (256) and of K chunks, against the oracle."""
import numpy as np
import pytest

from nnfusion_b200 import _lib as L
from nnfusion_b200 import synth
from oracle import oracle as orc
from tests.util import TOL_F16, gpu_linear, oracle_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,bits,dual", [
    (17, 256, 512, 4, False),       # 2 pairs share K, the second one's slice of 16 batch rows is empty
    (33, 257, 1088, 4, True),       # 3 pairs, gate and up, 17 k-blocks: the last chunk holds one
    (48, 513, 2112, 8, False),      # 4 pairs, 33 k-blocks of which two make a chunk
    (128, 130, 2048, 4, True),      # 4 pairs, gate and up
    (129, 1000, 11008, 4, False),   # a long K cut into 4 uneven ranges
    (300, 2500, 1088, 4, True),     # 2 or 3 pairs, up to 128 batch rows a tile, gate and up
    (1040, 2000, 640, 8, True),     # whole tiles
    (1040, 5000, 1024, 4, False),   # several whole tiles a pair, above 128 batch rows a tile
    (300, 9000, 1024, 4, True),     # one whole tile a pair, above 128 batch rows, gate and up
    (18, 19001, 3136, 4, False),    # 75 tiles on 74 pairs: seam shares, scalar stores
    (130, 19000, 3136, 4, False),   # the same above 128 batch rows a tile
])
def test_splits(M, N, K, bits, dual):
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(M + N))
    x = synth.make_x(rng, M, K, np.float16)
    w = [synth.make_weights(rng, N, K, bits, 64) for _ in range(1 + dual)]
    dev = [DeviceWeight.from_host(v) for v in w]
    tx = torch.from_numpy(x).cuda()
    r32 = oracle_linear(x, *w, out_dtype=np.float32)
    for y_dtype, add in [(torch.float16, False), (torch.float32, False)] + [(torch.float16, True), (torch.float32, True)] * (not dual):
        op = DequantDot(*dev, kernel=L.KERNEL_GEMM, y_dtype=y_dtype, add=add)
        c = torch.randn(M, N, device="cuda").to(y_dtype) if add else None
        kw = dict(addend=c) if add else {}
        y = op(tx, **kw)
        assert torch.equal(op(tx, **kw), y)          # bitwise repeatable, counters left zeroed
        op.ctx.device_status()
        want = r32 + c.float().cpu().numpy() if add else r32
        err = orc.max_rel_err(y.float().cpu().numpy(), want)
        # fp16 scale products and, with SiLU, one rounding of the gate to y's type: the kernel's other tests' bounds
        assert err <= min(TOL_F16, 3e-3 if dual else 2e-3), (y_dtype, add, err)


@pytest.mark.parametrize("M,N,K,dual", [(48, 4096, 11008, False), (100, 1000, 4096, True), (17, 2560, 2048, False)])
def test_pairs_that_share_k_repeat_back_to_back(M, N, K, dual):
    """Partial sums land where the peers' rings were: launch after launch without a pause must give the same bits."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(M))
    op = DequantDot(*[DeviceWeight.from_host(synth.make_weights(rng, N, K, 4, 128)) for _ in range(1 + dual)])
    x = torch.from_numpy(synth.make_x(rng, M, K, np.float16)).cuda()
    first = op(x).clone()
    outs = [op(x) for _ in range(300)]
    torch.cuda.synchronize()
    op.ctx.device_status()
    assert not [i for i, y in enumerate(outs) if not torch.equal(y, first)]


@pytest.mark.parametrize("M,N,K,dual,bias", [(17, 19, 5312, True, False), (18, 19001, 3136, False, True)])
def test_smaller_workspaces_are_used_as_far_as_they_go(M, N, K, dual, bias):
    """A program whose buffer was sized by another version of the library keeps running: the launch takes the best layout
    that the buffer holds, writes nothing behind it, and only a missing buffer is refused."""
    import ctypes
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight, NNFB200Error
    rng = np.random.Generator(np.random.PCG64(M + K))
    x = synth.make_x(rng, M, K, np.float16)
    w = [synth.make_weights(rng, N, K, 4, 64) for _ in range(1 + dual)]
    b = rng.standard_normal(N).astype(np.float32) if bias else None
    op = DequantDot(*[DeviceWeight.from_host(v) for v in w], bias=torch.from_numpy(b).cuda() if bias else None)
    tx, want = torch.from_numpy(x).cuda(), oracle_linear(x, *w, bias=b)
    d = op.desc(M, tx.dtype)
    need = int(op.ctx.lib.nnf_b200_linear_workspace_bytes(op.ctx.handle, ctypes.byref(d)))
    assert need > 1 << 20
    y = torch.empty((M, N), dtype=torch.float16, device="cuda")
    for size in (need, need - 256, need // 2, need // 4 // 256 * 256, 256):
        guarded = torch.zeros(size + 4096, dtype=torch.uint8, device="cuda")
        guarded[size:] = 0xAB
        for _ in range(2):
            y.fill_(float("nan"))
            op.run_raw(d, tx.data_ptr(), y.data_ptr(), guarded[:size])
            assert orc.max_rel_err(y.cpu().numpy(), want) <= min(TOL_F16, 3e-3 if dual else 2e-3), size
        assert bool((guarded[size:] == 0xAB).all())
    op.ctx.device_status()
    with pytest.raises(NNFB200Error) as e:
        op.run_raw(d, tx.data_ptr(), y.data_ptr(), None)
    assert e.value.status == L.EWORKSPACE


def _seam_bytes(M, N, K, bits, sets, bx):
    """Workspace of a launch whose tiles of bx batch rows are shared through it (148 SMs: 74 pairs)."""
    tiles = (M + bx - 1) // bx * ((N + 255) // 256)
    chunks = (K // 64 + (3 if bits == 4 else 1)) // (4 if bits == 4 else 2)
    return (2 * tiles * 4 + 255) // 256 * 256 + min(tiles * sets * chunks, 74) * 2 * 2 * sets * 128 * bx * 4


@pytest.mark.parametrize("M,N,K,bx,dual", [
    (23, 17, 5696, 16, True),       # 2 tiles on 74 pairs: one or two chunks a share, odd N
    (141, 312, 10816, 48, True),    # 7 of a weight set's 43 chunks a share: shares that hold the end of the gate's chunks
    (189, 306, 12864, 48, True),    # the same, N not a multiple of four
    (646, 6156, 2944, 224, True),   # 75 tiles, above 128 batch rows: whole tiles between the seams
    (686, 1281, 15040, 176, True),  # above 128 batch rows, odd N: several shares per weight set
    (129, 338, 15872, 48, False),   # with a bias
    (660, 6337, 3904, 224, False),  # with a bias, above 128 batch rows, odd N
])
def test_seam_shares_with_two_weight_sets_and_bias(M, N, K, bx, dual):
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(M * 7 + N))
    x = synth.make_x(rng, M, K, np.float16)
    w = [synth.make_weights(rng, N, K, 4, 64) for _ in range(1 + dual)]
    bias = None if dual else rng.standard_normal(N).astype(np.float32)
    rows = sorted({0, 1, 15, 16, bx - 1, min(bx, M - 1), M // 2, M - 2, M - 1} & set(range(M)))  # the oracle's rows are independent
    r32 = oracle_linear(x[rows], *w, bias=bias, out_dtype=np.float32)
    dev, tx = [DeviceWeight.from_host(v) for v in w], torch.from_numpy(x).cuda()
    for y_dtype in (torch.float16, torch.float32):
        op = DequantDot(*dev, bias=None if dual else torch.from_numpy(bias).cuda(), y_dtype=y_dtype)
        y = torch.full((M, N), float("nan"), dtype=y_dtype, device="cuda")
        op(tx, out=y)
        (ws,) = op._ws.values()
        assert ws.numel() == _seam_bytes(M, N, K, 4, 1 + dual, bx)      # this is the layout that the launch took
        assert bool(torch.isfinite(y).all()) and torch.equal(op(tx), y)
        op.ctx.device_status()
        err = orc.max_rel_err(y[rows].float().cpu().numpy(), r32)
        # fp16 scale products and, with SiLU, one rounding of the gate to y's type: the kernel's other tests' bounds
        assert err <= min(TOL_F16, 3e-3 if dual else 2e-3), (y_dtype, err)


@pytest.mark.parametrize("M", range(16, 257, 16))
def test_every_tile_width(M):
    """One batch tile of every width that the tensor core is given, with all its rows, and with one less."""
    rng = np.random.Generator(np.random.PCG64(M))
    w = synth.make_weights(rng, 300, 576, 4, 64)
    x = synth.make_x(rng, M, 576, np.float16)
    want = oracle_linear(x, w)
    for rows in (M, M - 1):
        y = gpu_linear(x[:rows], w, kernel=L.KERNEL_GEMM)
        assert orc.max_rel_err(y, want[:rows]) <= min(TOL_F16, 2e-3)  # fp16 scale products: the kernel's other tests' bound
