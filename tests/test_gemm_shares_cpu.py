"""The arithmetic by which the large-M kernel's pairs of CTAs share a launch (``nnfusion_b200/csrc/dq_gemm_tcgen05.cu``:
``WorkList``, ``pair_of_unit``, ``slot_of``, the contributors of a shared tile, the slices of a cluster), restated in Python and
checked for the properties the kernel relies on: shares partition the units; a share's segments lie inside one tile and one
weight set; a share has at most two tiles that it does not compute alone, whose sums of either weight set and CTA go to slots
of their own inside the workspace; and the pairs that the formulas name as contributors of a tile and weight set are those
that have a segment of it, in the order of their K ranges."""
import pytest


def shares(tiles, sets, cpt, G):
    U = tiles * sets * cpt
    return [(c * U // G, (c + 1) * U // G) for c in range(G)]


def segments(u_begin, u_end, sets, cpt):
    """(tile, weight set, first chunk, last chunk, computed whole by this pair, the pair's last segment of the tile)"""
    out, u, per_tile = [], u_begin, sets * cpt
    while u < u_end:
        tile, inside = divmod(u, per_tile)
        base = tile * per_tile
        which = 1 if inside >= cpt else 0
        c0 = inside - which * cpt
        c1 = min(cpt, c0 + (u_end - u))
        u += c1 - c0
        out.append((tile, which, c0, c1, u_begin <= base and base + per_tile <= u_end, u in (u_end, base + per_tile)))
    return out


def pair_of_unit(u, U, G):
    return ((u + 1) * G + U - 1) // U - 1


def slot_of(c, rank, t, which, sets, cpt, U, G):
    first_tile = (c * U // G) // (sets * cpt)
    return ((2 * c + rank) * 2 + (0 if t == first_tile else 1)) * sets + which


SHAPES = [(75, 13, 74), (43, 16, 74), (86, 16, 74), (344, 16, 74), (1376, 16, 74), (34, 68, 74), (4, 16, 64), (32, 8, 74),
          (3584, 32, 74), (1, 1, 1), (1, 5, 5), (3, 2, 6), (7, 3, 4), (75, 1, 74), (74, 43, 74), (5, 172, 74), (1000, 7, 66)]


@pytest.mark.parametrize("sets", [1, 2])
@pytest.mark.parametrize("tiles,cpt,G", SHAPES)
def test_seam_shares(tiles, cpt, G, sets):
    U = tiles * sets * cpt
    assert G <= U                                               # the host never launches more pairs than units
    sh = shares(tiles, sets, cpt, G)
    assert sh[0][0] == 0 and sh[-1][1] == U
    assert all(a[1] == b[0] and a[1] > a[0] for a, b in zip(sh, sh[1:]))   # a partition, in order; nobody is idle
    slots = set()
    parts = {}                                                  # (tile, weight set) -> [(pair, c0, c1)]
    arrivals = {}                                               # tile -> pairs that take a ticket
    for c, (b, e) in enumerate(sh):
        segs = segments(b, e, sets, cpt)
        assert sum(c1 - c0 for _, _, c0, c1, _, _ in segs) == e - b
        assert all(c1 > c0 for _, _, c0, c1, _, _ in segs)
        order = []                                              # this pair's tiles
        for t, *_ in segs:
            if t not in order:
                order.append(t)
        for t, which, c0, c1, whole, last in segs:
            same = [s for s in segs if s[0] == t]
            assert last == (same[-1][1] == which)               # one ticket per pair and tile
            if whole:
                assert c0 == 0 and c1 == cpt and len(same) == sets
                continue
            assert t in (order[0], order[-1])                   # only the first and the last tile can be shared
            for rank in range(2):
                s = slot_of(c, rank, t, which, sets, cpt, U, G)
                assert s not in slots and 0 <= s < G * 2 * 2 * sets
                slots.add(s)
            parts.setdefault((t, which), []).append((c, c0, c1))
            if last:
                arrivals.setdefault(t, []).append(c)
        for u in (b, e - 1, (b + e) // 2):
            assert pair_of_unit(u, U, G) == c
    per_tile = sets * cpt
    for t, pairs in arrivals.items():
        c_first, c_last = pair_of_unit(t * per_tile, U, G), pair_of_unit((t + 1) * per_tile - 1, U, G)
        assert pairs == list(range(c_first, c_last + 1)) and len(pairs) >= 2   # the last ticket is c_last - c_first
        first = [c_first, c_first if sets == 1 else pair_of_unit(t * per_tile + cpt, U, G)]
        last = [c_last if sets == 1 else pair_of_unit(t * per_tile + cpt - 1, U, G), c_last]
        for which in range(sets):
            mine = parts[t, which]
            assert [c for c, _, _ in mine] == list(range(first[which], last[which] + 1))
            assert mine[0][1] == 0 and mine[-1][2] == cpt
            assert all(a[2] == b[1] for a, b in zip(mine, mine[1:]))           # K ranges in the order of the pairs


@pytest.mark.parametrize("sets", [1, 2])
def test_whole_tiles_are_cut_at_tile_boundaries(sets):
    for tiles in (1, 5, 43, 64, 74, 129):
        for cpt in (1, 4, 16):
            for G in (1, 43, 74):
                if G > tiles:
                    continue
                cuts = [c * tiles // G * sets * cpt for c in range(G + 1)]
                assert cuts[0] == 0 and cuts[-1] == tiles * sets * cpt
                for b, e in zip(cuts, cuts[1:]):
                    assert e > b and all(s[4] and s[2] == 0 and s[3] == cpt for s in segments(b, e, sets, cpt))


@pytest.mark.parametrize("ksplit", [2, 3, 4])
def test_clusters_that_share_k(ksplit):
    """The parts of K of a cluster's pairs are a partition without empty ones; the slices of batch rows that they finish cover
    the tile in pieces of 16; and the parts that a CTA receives fit where its rings were."""
    for cpt in (ksplit, ksplit + 1, 5, 16, 43, 172):
        cuts = [part * cpt // ksplit for part in range(ksplit + 1)]
        assert cuts[0] == 0 and cuts[-1] == cpt and (cpt < ksplit or all(b > a for a, b in zip(cuts, cuts[1:])))
    for bx in range(16, 257, 16):
        rows = (bx // 16 + ksplit - 1) // ksplit * 16
        owner = [col // rows for col in range(0, bx, 16)]
        assert max(owner) < ksplit and rows * ksplit >= bx
        for sets in (1, 2) if bx <= 128 else (1,):
            rings = (96 + 8 * 16) * 1024 if bx <= 128 else (128 + 6 * 16) * 1024
            assert sets * ksplit * rows * 128 * 4 <= rings
