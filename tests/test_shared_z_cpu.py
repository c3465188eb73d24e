"""CPU model of k_fz_shared's schedule with done members (csrc/fft_fast.cuh): a
CTA's items are tile 0 of member 0, issued before the flags are known, then the
active members of each tile; no copy lands in a buffer that an unfinished item
reads, every active member of every tile is transformed once with its tile's
Green table, and no done member is."""
import itertools

import pytest


def _replay(flags, tiles):
    active = [m for m, on in enumerate(flags) if on]
    na = len(active)
    lead = 0 if na and active[0] == 0 else 1
    nitems = tiles * na + lead if tiles else 0
    stage, green, finished, transformed = {}, {}, set(), []

    def issue(i, j, m, with_green):
        prev = stage.get(i & 1)
        assert prev is None or prev[0] in finished, "stage overwritten"
        stage[i & 1] = (i, j, m)
        if with_green:
            # nobody reads the buffer's former tile any more
            assert all(k in finished for k, (t, _) in items.items() if t == green.get(j & 1)), "Green overwritten"
            green[j & 1] = j

    items = {}  # item -> (turn, member), of the items whose copies were issued
    if tiles:
        items[0] = (0, 0)
        issue(0, 0, 0, True)
    for i in range(nitems):
        q = i - lead
        if i + 1 < nitems:
            j, m = (q + 1) // na, active[(q + 1) % na]
            items[i + 1] = (j, m)
            issue(i + 1, j, m, (q + 1) % na == 0 and q + 1 > 0)
        assert stage[i & 1][0] == i
        if q >= 0:
            j, m = q // na, active[q % na]
            assert stage[i & 1][1:] == (j, m) and green[j & 1] == j
            transformed.append((j, m))
        finished.add(i)
    if tiles and not nitems:
        raise AssertionError("a copy without a wait")
    return transformed


@pytest.mark.parametrize("members", [2, 3, 5])
@pytest.mark.parametrize("tiles", [0, 1, 2, 3, 6])
def test_every_active_member_once(members, tiles):
    for flags in itertools.product([False, True], repeat=members):
        got = _replay(flags, tiles)
        assert got == [(j, m) for j in range(tiles) for m in range(members) if flags[m]]


@pytest.mark.parametrize("members", [1, 31, 32, 33, 64])
def test_active_list(members):
    """The list the first warp builds with a ballot per 32 members, in order."""
    for flags in ([True] * members, [m % 3 != 0 for m in range(members)], [False] * members,
                  [m == members - 1 for m in range(members)]):
        out, n = {}, 0
        for m0 in range(0, members, 32):
            on = [m0 + lane < members and flags[m0 + lane] for lane in range(32)]
            mask = sum(1 << lane for lane in range(32) if on[lane])
            for lane in range(32):
                if on[lane]:
                    out[n + bin(mask & ((1 << lane) - 1)).count("1")] = m0 + lane
            n += bin(mask).count("1")
        assert [out[k] for k in range(n)] == [m for m in range(members) if flags[m]]
