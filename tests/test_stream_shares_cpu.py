"""How the CTAs of ``nnfusion_b200/csrc/dq_stream.cu`` share their units (``csrc/stream_shares.h``, compiled here as host code): shares
partition the units, ``owner`` names the share of a unit, and the parts of a shared tile go to slots of their own inside the workspace."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_SHIM = r"""
#include "stream_shares.h"
static nnf::StreamShares s;
extern "C" int set(int tiles, int KU, int most) { s.set(tiles, KU, most); return s.ctas; }
extern "C" int begin(int c) { return s.begin(c); }
extern "C" int units(int c) { return s.units(c); }
extern "C" int owner(int u) { return s.owner(u); }
extern "C" int slot(int c, int t) { return s.slot(c, t); }
extern "C" int slots() { return s.slots(); }
"""


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("shares")
    (d / "shim.cpp").write_text(_SHIM)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "nnfusion_b200", "csrc"), str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


@pytest.mark.parametrize("most", [296, 264, 148, 2, 1])
@pytest.mark.parametrize("tiles,KU", [(33, 86), (32, 86), (57, 72), (64, 224), (11, 224), (448, 64), (296, 72), (295, 72), (297, 72), (592, 65),
                                      (313, 33), (1185, 33), (1, 200), (7, 5), (3555, 1)])
def test_shares(shares, tiles, KU, most):
    U = tiles * KU
    G = shares.set(tiles, KU, most)
    assert G == min(most, U)
    begin, owner = shares.begin, shares.owner
    assert begin(0) == 0 and begin(G) == U
    for c in range(G):
        assert begin(c + 1) - begin(c) == shares.units(c) > 0
        assert owner(begin(c)) == owner(begin(c + 1) - 1) == c
    parts, n = {}, shares.slots()
    assert n <= 2 * G
    for t in range(tiles):
        first, last = owner(t * KU), owner(t * KU + KU - 1)
        for c in range(first, last + 1):
            assert begin(c) < (t + 1) * KU and begin(c + 1) > t * KU       # every one of them has a part of the tile
            if first != last:
                s = shares.slot(c, t)
                assert 0 <= s < n and parts.setdefault(s, (c, t)) == (c, t)
    assert n or not parts
