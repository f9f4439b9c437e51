"""The versions of the exact-order sweep's exchange words (sweep_rows_kernel, k_linesolve.cu),
replayed on the CPU under a memory that keeps no order but a word's own.

A row of visits (ks, k, s) is one warp walking along j; visit v = 2 ks + s of line (k, j)
leaves version v + 1 in the line's word, which rows on other CTAs poll for.  The stores
of two versions of a word come from different warps and are relaxed, so nothing orders
them but coherence: a store comes after every store of the word that its own thread has
seen or made before, and anywhere else is possible.  Restated here: which words a visit
polls, for which version, and the store; every store enters its word's order at any place
coherence allows, and a poll may return any store not older than the last one seen.
The sweep must end for every choice: with the word of a row's first line seen before it
is stored to, it does.  Without that (but for planes of one line), a version can come to
rest under an older one and its reader polls for ever, which the replay must notice.
"""
import random

import pytest


class Stuck(Exception):
    pass


def replay(M, J, guard, rng):
    """M planes of J lines; guard "first": the first line's word is seen at version v before
    version v + 1 is stored; "single": only where a plane has one line."""
    order = {(k, j): [0] for k in range(1, M + 1) for j in range(J)}  # versions in coherence order
    seen = {}  # (row, line) -> place of the last store this row's warp has seen or made

    def poll(row, line, want):
        at = rng.randint(seen.get((row, line), 0), len(order[line]) - 1)
        seen[row, line] = at
        return order[line][at] == want

    # (ks, k, s), in the order rows are handed out
    at = {(m // M, M - m % M, s): (0, {}) for m in range(2 * M) for s in range(2)}
    visits, quiet = [], 0
    while at:
        moved = False
        for row in rng.sample(sorted(at), len(at)):
            ks, k, s = row
            j, got = at[row]
            v = 2 * ks + s
            need = {}
            if k < M:
                need[k + 1, j] = 2 * ks + 2
            if k > 1 and ks:
                need[k - 1, j] = 2 * ks
            if j + 1 < J and v:
                need[k, j + 1] = v
            if v and j == 0 and (guard == "first" or J == 1):
                need[k, j] = v
            for line, want in need.items():
                if line not in got and poll(row, line, want):
                    got[line] = True
            if len(got) < len(need):
                continue
            if v < 3 or k > 1:
                place = rng.randint(seen.get((row, (k, j)), 0) + 1, len(order[k, j]))
                order[k, j].insert(place, v + 1)
                for key in seen:
                    if key[1] == (k, j) and seen[key] >= place:
                        seen[key] += 1
                seen[row, (k, j)] = place
            visits.append((v, k, j))
            at[row] = (j + 1, {})
            if j + 1 == J:
                del at[row]
            moved = True
        quiet = 0 if moved else quiet + 1
        if quiet > 200:
            raise Stuck
    assert sorted(visits) == sorted((v, k, j) for v in range(4) for k in range(1, M + 1) for j in range(J))
    for line, versions in order.items():
        assert versions == sorted(versions), (line, versions)


@pytest.mark.parametrize("M,J", [(1, 1), (1, 4), (2, 1), (5, 1), (2, 2), (3, 2), (4, 5), (6, 3)])
def test_versions_land_in_turn(M, J):
    for seed in range(15):
        replay(M, J, "first", random.Random(seed))


@pytest.mark.parametrize("M,J", [(2, 2), (3, 2), (4, 5)])
def test_replay_notices_versions_out_of_turn(M, J):
    broken = 0
    for seed in range(15):
        try:
            replay(M, J, "single", random.Random(seed))
        except (Stuck, AssertionError):
            broken += 1
    assert broken > 0
