"""Shared memory of the decode kernel: no team and no codebook copy is lost to the layout's padding."""
import ctypes as C
import itertools

import pytest

from util import load_pkg

pkg = load_pkg()
LIMIT, TEAMS = 227 * 1024, 3


def unpadded(tiers, dh, units):
    """Teams and copies where the query operand (dh / 16 x 512 bytes), the barriers, votes and statistics of three teams (1792)
    and the teams' own areas (V tiles 128 x dh x 2, weights 4096, key stages 9216, metadata 1024) lie back to back."""
    prefix = 4 * (units + 1) if units <= 2048 else 0
    sizes = [dh * (1 << bits) * 4 + 128 for _, bits in tiers]
    for teams in range(TEAMS, 0, -1):
        left = LIMIT - dh // 16 * 512 - 1792 - teams * (256 * dh + 14336) - prefix - sum(sizes)
        if left >= 0:
            break
    else:
        return 0, [1] * len(tiers)
    copies = []
    for (g, _), size in zip(tiers, sizes):
        copies.append(2 if g == 16 and size <= left else 1)
        left -= size * (copies[-1] - 1)
    return teams, copies


def planned(tiers, dh, units):
    t = pkg.TierSet(dh, [pkg.TierSpec(i + 1, g, bits) for i, (g, bits) in enumerate(tiers)]).to_c()
    teams, copies = C.c_int32(-1), (C.c_int32 * 4)()
    size = pkg._lib.load().sphkv_decode_smem(C.byref(t), dh, units, C.byref(teams), copies)
    assert teams.value == 0 or 0 < size <= LIMIT
    return teams.value, list(copies)[:len(tiers)]


# four and three 64-centroid tiers, and mixes, at batch x KV heads where a few hundred bytes decide
@pytest.mark.parametrize("dh,tiers,units", [
    (128, [(16, 6)] * 4, 128), (128, [(16, 6)] * 4, 191), (128, [(16, 6)] * 3, 160), (128, [(16, 6), (16, 4)], 640),
    (128, [(16, 6), (16, 4)], 703), (128, [(16, 6), (16, 6), (16, 5), (16, 2)], 150), (64, [(16, 6)] * 4, 512),
    (64, [(16, 6)] * 4, 1087)])
def test_a_few_hundred_bytes_cost_no_team_and_no_copy(dh, tiers, units):
    assert planned(tiers, dh, units) == unpadded(tiers, dh, units)


@pytest.mark.parametrize("dh", [64, 128])
def test_every_tier_set_has_the_teams_and_copies_that_fit(dh):
    kinds = [(g, bits) for g in (16, 32) for bits in range(1, 7)]
    sets = [list(s) for n in (1, 2, 3, 4) for s in itertools.combinations_with_replacement(kinds, n)]
    for tiers in sets + [s[::-1] for s in sets]:
        for units in (1, 8, 63, 64, 128, 191, 192, 320, 511, 512, 640, 703, 704, 1087, 1088, 2048, 2049):
            (teams, copies), (want, want_copies) = planned(tiers, dh, units), unpadded(tiers, dh, units)
            assert teams > want or (teams == want and sum(copies) >= sum(want_copies)), (tiers, units)
