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
