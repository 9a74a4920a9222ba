"""The arithmetic by which the CTAs of ``nnfusion_b200/csrc/dq_stream.cu`` share their units (``share_begin``, ``owner``,
``slot``), restated in Python: shares partition the units, ``owner`` names the share of a unit, and the parts of a shared tile go
to slots of their own inside the workspace."""
import pytest


@pytest.mark.parametrize("G", [296, 264, 148, 2, 1])
@pytest.mark.parametrize("tiles,KU", [(33, 86), (32, 86), (57, 64), (172, 32), (235, 16), (71, 48), (1185, 3), (3555, 1), (64, 224), (1, 200), (7, 5)])
def test_shares(tiles, KU, G):
    U = tiles * KU
    G = min(G, U)
    lo, rem = divmod(U, G)

    def begin(c):
        return c * lo + min(c, rem)

    def owner(u):
        more = rem * (lo + 1)
        return u // (lo + 1) if u < more else rem + (u - more) // lo

    assert begin(0) == 0 and begin(G) == U
    for c in range(G):
        assert begin(c + 1) - begin(c) == lo + (c < rem) > 0
        assert owner(begin(c)) == owner(begin(c + 1) - 1) == c
    slots = {}
    for t in range(tiles):
        first, last = owner(t * KU), owner(t * KU + KU - 1)
        for c in range(first, last + 1):
            assert begin(c) < (t + 1) * KU and begin(c + 1) > t * KU       # every one of them has a part of the tile
            if first != last:
                s = 2 * c + (0 if begin(c) >= t * KU else 1)
                assert s < 2 * G and slots.setdefault(s, t) == t
