"""Operands that the launch directly ahead on the stream writes: every kernel starts while that launch is still running
and may read them only behind its wait for it."""
import numpy as np
import pytest

from nnfusion_b200 import synth

pytestmark = pytest.mark.gpu


def _chain(make_consumer, n, rounds=40):
    """A [1, n] fp32 tensor is rewritten by one linear and read by the next, back to back; the consumer's results must be
    those it gives when the device is idle in between.  ``make_consumer(tensor)`` returns the consumer's call."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(n))
    producer = DequantDot(DeviceWeight.from_host(synth.make_weights(rng, n, 1024, 4, 128)), y_dtype=torch.float32)
    between = torch.zeros((1, n), dtype=torch.float32, device="cuda")
    consume = make_consumer(between)
    xs = [torch.from_numpy(synth.make_x(rng, 1, 1024, np.float16)).cuda() for _ in range(rounds)]
    want = []
    for x in xs:
        producer(x, out=between)
        torch.cuda.synchronize()
        want.append(consume().clone())
        torch.cuda.synchronize()
    got = []
    for x in xs:
        producer(x, out=between)
        got.append(consume())
    torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    differ = [i for i, (a, b) in enumerate(zip(got, want)) if not torch.equal(a, b)]
    assert not differ, f"rounds {differ} read the operand of an earlier one"


@pytest.mark.parametrize("M,K,dual", [(1, 4096, False), (1, 4096, True), (5, 8192, False), (16, 4096, False), (40, 4096, False)])
def test_gain_written_by_the_launch_ahead(M, K, dual):
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(7))
    ws = [DeviceWeight.from_host(synth.make_weights(rng, 2048, K, 4, 128)) for _ in range(1 + dual)]
    x = torch.from_numpy(synth.make_x(rng, M, K, np.float16)).cuda()

    def make(gain):
        node = DequantDot(*ws, gain=gain.view(-1))
        return lambda: node(x)
    _chain(make, K)


@pytest.mark.parametrize("M,kernel,norm", [(1, 1, False), (1, 1, True), (8, 1, False), (16, 1, True), (2, 2, False), (2, 2, True)])
def test_activations_and_bias_written_by_the_launch_ahead(M, kernel, norm):
    """fp32 activations (all rows of one buffer) and a bias, for the small-M kernel and for the large-M kernel's pre-pass."""
    import torch
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(8))
    K, N = 2048, 1536
    w = DeviceWeight.from_host(synth.make_weights(rng, N, K, 4, 128))
    gain = torch.from_numpy(rng.uniform(0.9, 1.1, K).astype(np.float32)).cuda() if norm else None

    def activations(t):
        node = DequantDot(w, gain=gain, kernel=kernel)
        return lambda: node(t.view(M, K))
    _chain(activations, M * K)

    x = torch.from_numpy(synth.make_x(rng, M, K, np.float16)).cuda()

    def bias(t):
        node = DequantDot(w, gain=gain, bias=t.view(-1), kernel=kernel)
        return lambda: node(x)
    _chain(bias, N)


@pytest.mark.parametrize("norm", [False, True])
def test_exact_zero_point_kernel_behind_the_launch_ahead(norm):
    import torch
    from nnfusion_b200 import _lib as L
    from nnfusion_b200.linear import DequantDot, DeviceWeight
    rng = np.random.Generator(np.random.PCG64(9))
    K, N = 2048, 1536
    w = DeviceWeight.from_host(synth.make_weights(rng, N, K, 4, 128))
    gain = torch.from_numpy(rng.uniform(0.9, 1.1, K).astype(np.float32)).cuda() if norm else None

    def activations(t):
        node = DequantDot(w, gain=gain, flags=L.FLAG_EXACT_ZP)
        return lambda: node(t.view(2, K))
    _chain(activations, 2 * K)
