"""Decode attention where its launch shape changes: sequences around the lengths at which warps, ranges and clusters of
ranges start, groups of more query heads than a CTA takes, and enough ranges for the workspace form."""
import numpy as np
import pytest

from tests.test_attention_gpu import _check, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos", [63, 64, 111, 112, 126, 127, 128, 129, 191, 192, 447, 448])
@pytest.mark.parametrize("H,Hkv", [(2, 2), (9, 1)])
def test_lengths_around_the_cuts(H, Hkv, pos):
    outs, ref, caches, caches_ref = _run(H, Hkv, 512, pos, seed=200 + pos, calls=2)
    _check(outs[0], ref)
    np.testing.assert_array_equal(outs[0], outs[1])
    np.testing.assert_array_equal(caches[1], caches_ref[1])


@pytest.mark.parametrize("H,Hkv,pos", [(8, 1, 4862), (8, 1, 4864), (24, 1, 8200), (4, 4, 9000), (20, 20, 700)])
def test_long_sequences_on_few_heads(H, Hkv, pos):
    """4864 rows: the last length that one cluster of 8 ranges takes; 20 heads: clusters of 5, the most that fit at once."""
    outs, ref, _, _ = _run(H, Hkv, pos + 1, pos, seed=300 + H, calls=2)
    _check(outs[0], ref)
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("rotary", [True, False])
@pytest.mark.parametrize("H,Hkv", [(1, 1), (9, 3), (32, 32), (64, 8)])
@pytest.mark.parametrize("pos", [0, 1, 7, 8, 15, 16, 30, 31, 32])
def test_short_sequences(H, Hkv, pos, rotary):
    """Up to 32 rows one CTA takes a query head (33: the first that does not), whatever shares its key/value head."""
    outs, ref, caches, caches_ref = _run(H, Hkv, 40, pos, seed=400 + pos, rotary=rotary, calls=2)
    _check(outs[0], ref)
    np.testing.assert_array_equal(outs[0], outs[1])
    np.testing.assert_array_equal(caches[1], caches_ref[1])
    np.testing.assert_allclose(caches[0].astype(np.float32), caches_ref[0].astype(np.float32), rtol=2e-3, atol=2e-3)
