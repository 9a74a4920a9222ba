"""The small-M kernel's sums of a split K through the workspace, four values a thread (one row: every
other value): odd and even row counts at the edges
of the accumulator's columns (2, 8, 16), ragged N, split counts around the four read back at a time, with every epilogue."""
import numpy as np
import pytest

from nnfusion_b200 import _lib as L
from nnfusion_b200 import synth
from oracle import oracle as orc
from tests.util import TOL_F16, gpu_linear, oracle_linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M,N,splits", [(1, 2063, 3), (1, 4096, 5), (2, 4096, 3), (3, 2063, 4), (7, 2049, 5), (8, 4095, 4), (9, 2063, 3), (15, 2048, 5), (16, 2049, 4)])
def test_four_values_a_thread(M, N, splits, bits):
    rng = np.random.Generator(np.random.PCG64(M * N))
    K = 10240
    x = synth.make_x(rng, M, K, np.float16)
    w = synth.make_weights(rng, N, K, bits, 128)
    gain, bias = rng.uniform(0.9, 1.1, K).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    for kw in ({}, dict(bias=bias), dict(gain=gain), dict(out_dtype=np.float32)):
        y = gpu_linear(x, w, kernel=L.KERNEL_GEMV, split_k=splits if bits == 4 else splits + 3, repeat=2, **kw)
        assert np.array_equal(y[0], y[1])            # fixed order of the splits, counters left zeroed
        err = orc.max_rel_err(y[0], oracle_linear(x, w, **kw))
        assert err <= min(TOL_F16, 2e-3), (kw.keys(), err)  # fp32 sums, one rounding to fp16: the kernel's other tests' bound
