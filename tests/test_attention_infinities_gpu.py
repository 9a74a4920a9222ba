"""Decode attention with infinities in the caches (keys or values that left the fp16 range, rows masked by an infinite key)
gives what the softmax gives for them: a row of score -inf has no weight, whichever warp or range it falls to."""
import numpy as np
import pytest

from oracle import attention as att
from oracle import oracle as orc
from tests.util import TOL_F16

pytestmark = pytest.mark.gpu


def _run(H, Hkv, pos, seed, change, splits=0):
    """One step without rotary embedding (so that the caller knows the queries); ``change(q, k_cache, v_cache)`` edits the
    operands in place."""
    import torch
    from nnfusion_b200.attention import DecodeAttention
    rng = np.random.Generator(np.random.PCG64(seed))
    cap = pos + 1
    q, kn, vn = (rng.standard_normal((h, 128)).astype(np.float16) for h in (H, Hkv, Hkv))
    kc, vc = (rng.standard_normal((Hkv, cap, 128)).astype(np.float16) for _ in range(2))
    kc[:, pos:], vc[:, pos:] = 0, 0
    q[:, 5] = np.abs(q[:, 5]) + np.float16(0.1)  # an infinity in dimension 5 of a key decides the score's sign
    change(q, kc, vc)
    op = DecodeAttention(H, Hkv, 128, cap, "cuda:0", rotary=False, splits=splits)
    op.k_cache.copy_(torch.from_numpy(kc))
    op.v_cache.copy_(torch.from_numpy(vc))
    y = op(*(torch.from_numpy(a).cuda() for a in (q, kn, vn)), pos).cpu().numpy().reshape(H, 128)
    op.ctx.device_status()
    with np.errstate(invalid="ignore", over="ignore"):
        ref, _ = att.decode_attention(q, kn, vn, kc.copy(), vc.copy(), pos, rotary=False)
    return y.astype(np.float32), np.asarray(ref, np.float32).reshape(H, 128)


_SHAPES = [(4, 4, 20), (4, 4, 100), (8, 1, 300), (9, 1, 130), (4, 4, 1200), (8, 1, 6000)]


@pytest.mark.parametrize("H,Hkv,pos", _SHAPES)
@pytest.mark.parametrize("masked", ["one", "block", "first rows", "all but two"])
def test_rows_masked_by_an_infinite_key(H, Hkv, pos, masked):
    """``block``: every row of a warp's first block; ``all but two``: whole ranges without a finite score."""
    rows = {"one": slice(3, 4), "block": slice(16, 32), "first rows": slice(0, min(pos - 2, 70)),
            "all but two": slice(0, pos - 2)}[masked]

    def change(q, kc, vc):
        kc[:, rows, 5] = -np.inf
    y, ref = _run(H, Hkv, pos, 60 + pos, change)
    assert np.isfinite(ref).all()
    assert np.isfinite(y).all() and orc.max_rel_err(y, ref) <= TOL_F16


@pytest.mark.parametrize("H,Hkv,pos", _SHAPES)
def test_an_infinite_score_leaves_nothing_finite(H, Hkv, pos):
    def change(q, kc, vc):
        kc[:, 3, 5] = np.inf
    y, ref = _run(H, Hkv, pos, 70 + pos, change)
    assert np.isnan(ref).all() and np.isnan(y).all()  # inf - inf


@pytest.mark.parametrize("H,Hkv,pos", _SHAPES)
@pytest.mark.parametrize("sign", [1, -1])
def test_infinite_values_stay_infinities(H, Hkv, pos, sign):
    """A value beyond the fp16 range is infinite in its own dimension for every query that looks at its row, and nowhere
    else; opposite infinities and a masked row's infinity have no value."""
    def change(q, kc, vc):
        vc[:, 3, 7], vc[:, pos // 2, 64] = sign * np.inf, -sign * np.inf
        vc[:, pos - 1, 100], vc[:, pos - 2, 100] = np.inf, -np.inf
        kc[:, 9, 5], vc[:, 9, 30] = -np.inf, np.inf
        q *= np.float16(0.25)  # weights of one order of magnitude: none underflows
    y, ref = _run(H, Hkv, pos, 80 + pos, change)
    assert np.isinf(ref[:, 7]).all() and np.isinf(ref[:, 64]).all() and np.isnan(ref[:, [30, 100]]).all()
    np.testing.assert_array_equal(np.isnan(y), np.isnan(ref))
    np.testing.assert_array_equal(y[np.isinf(ref)], ref[np.isinf(ref)])
    ok = np.isfinite(ref)
    assert ok.sum() == H * 124 and np.abs(y[ok] - ref[ok]).max() <= TOL_F16 * np.abs(ref[ok]).max()
