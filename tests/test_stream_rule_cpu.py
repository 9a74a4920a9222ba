"""Which calls of 9 to 16 rows take the form that streams its weights through shared memory (``stream_serves`` in
``nnfusion_b200/csrc/dq_stream.cu``), asked of the library's planner without a device (148 SMs assumed)."""
import ctypes

import pytest

from nnfusion_b200 import _lib as L
from nnfusion_b200 import build


@pytest.fixture(scope="module")
def lib():
    build.build_library()
    return L.load()


def _plan(lib, M, N, K, pair=False, norm=False, split_k=0):
    d = L.LinearDesc(M=M, N=N, K=K, w_bits=4, group_size=128, x_dtype=L.F16, y_dtype=L.F16, scale_dtype=L.F16, split_k=split_k,
                     epilogue=L.EPILOGUE_SILU_MUL if pair else L.EPILOGUE_NONE,
                     prologue=L.PROLOGUE_RMSNORM if norm else L.PROLOGUE_NONE)
    out = (ctypes.c_int32 * 8)()
    assert lib.nnf_b200_linear_plan(None, ctypes.byref(d), ctypes.byref(out)) == L.OK
    return list(out), int(lib.nnf_b200_linear_workspace_bytes(None, ctypes.byref(d)))


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("M", [9, 16])
def test_halves_that_meet_in_a_cluster_stay_there(lib, M, pair):
    """That form touches no workspace, so that calls of one node on two streams may overlap: such calls neither take the
    streaming form nor ask for its workspace.  (74 clusters of 2 CTAs are resident on 148 SMs.)"""
    found = 0
    for K in range(4224, 8193, 128):
        for N in (2048, 4096, 8192, 9001, 11008, 14336, 28672):
            out, need = _plan(lib, M, N, K, pair)
            if out[2] == 2 and out[7] & 1 and out[4] // 2 <= 74:
                found += 1
                assert not out[7] & 16, (N, K)
                assert need == _plan(lib, M, N, K, pair, split_k=2)[1], (N, K)
    assert found >= 100


@pytest.mark.parametrize("M,norm", [(9, False), (16, True)])
@pytest.mark.parametrize("N,K,pair,streams", [
    (4096, 11008, False, True), (8192, 28672, False, True), (28672, 8192, True, True),   # the projections of 7B and 70B shapes
    (3936, 12288, False, True), (1680, 11520, True, True),                               # (7 and 2 x 3 tiles to walk, 12 warps)
    (3344, 12288, False, False), (4608, 9728, False, False), (672, 28672, True, False),  # measured slower there:
    (3104, 17920, False, False), (2064, 28672, False, False),                            # few tiles to walk, many CTAs to a tile
    (4096, 4096, False, False), (11008, 4096, True, False),                              # K is not cut
])
def test_sides_of_the_line(lib, N, K, pair, streams, M, norm):
    assert bool(_plan(lib, M, N, K, pair, norm)[0][7] & 16) == streams
    assert not _plan(lib, 8, N, K, pair, norm)[0][7] & 16
