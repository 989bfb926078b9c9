"""The closed-form tile lists (csrc/necg_tiles.h) against lists built entry by entry."""
import numpy as np
import pytest

from emu import emu


@pytest.mark.parametrize("K", [1, 2, 31, 32, 33, 63, 64, 65, 200, 257, 353, 545, 2048])
@pytest.mark.parametrize("lc,w,nst,sms", [(1, 8, 24, 148), (2, 8, 24, 148), (3, 12, 4, 148), (16, 16, 2, 148), (5, 8, 1, 7),
                                          (1, 12, 24, 3), (64, 8, 3, 20)])
def test_lists(K, lc, w, nst, sms):
    got = emu.sym_lists(K, lc, w, nst, sms)
    nkb, pad = (K + 31) // 32, (-K) % 32
    ntk = [(32 * kb + 31 - pad) // lc + 1 for kb in range(nkb)]
    tiles = [(kb, c) for kb in range(nkb) for c in range(ntk[kb])]
    start = np.concatenate([[0], np.cumsum(ntk)])
    assert got["ntiles"] == len(tiles) and np.array_equal(got["tiles"], tiles) and np.array_equal(got["start"], start)
    # every pair (k >= l) is in exactly one tile
    assert sum(min(lc, 32 * kb + 31 - pad - c * lc + 1) for kb, c in tiles) == sum(32 * kb + 32 - pad for kb in range(nkb))
    whole = [(kb, c) for kb in range(nkb - 1, -1, -1) for c in range(0, ntk[kb], w)]
    G, T = len(whole), len(whole) % sms
    parts = min(sms // T if T else 1, 8, nst)
    if T and G - T + T * parts > len(tiles):
        parts = 1 + (len(tiles) - G) // T
    if parts < 2:
        T, parts = 0, 1
    units = [(kb, c, 0, 1) for kb, c in whole[:G - T]] + [(kb, c, p, parts) for kb, c in whole[G - T:] for p in range(parts)]
    assert (got["tail0"], got["ntail"], got["parts"], got["units"]) == (G - T, T, parts, len(units))
    assert len(units) <= len(tiles)  # bra partials per unit fit the slots of the tiles
    g = got["groups"]
    unpacked = np.stack([g[:, 0], g[:, 1] & 0xffffff, (g[:, 1] >> 24) & 15, ((g[:, 1] >> 28) & 7) + 1], 1)
    assert np.array_equal(unpacked, units)
    for kb in range(nkb):
        mine = [u for u, x in enumerate(units) if x[0] == kb]
        assert got["urange"][kb].tolist() == [mine[0], mine[-1] + 1] and mine == list(range(mine[0], mine[-1] + 1))
    slot = {}
    for j, (kb, c) in enumerate(whole[G - T:]):
        for i in range(w):
            slot[(kb, c + i)] = (j * w + i) * (parts - 1)
    assert got["tslot"].tolist() == [slot.get(t, -1) if T else -1 for t in tiles]
    eights = [(kb, c) for kb in range(nkb - 1, -1, -1) for c in range(0, ntk[kb], 8)]
    assert np.array_equal(got["bgroups"], eights)
    for kb in range(nkb):
        mine = [u for u, x in enumerate(eights) if x[0] == kb]
        assert got["burange"][kb].tolist() == [mine[0], mine[-1] + 1]
