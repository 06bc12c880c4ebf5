"""The layer prologue's two rings (csrc/kda_chain.cu, layer_prologue_role) as a model: four warps cook rows in turn, a row's raw copy
lands in any order, and a barrier tells a waiter the parity of its phase only.  No order of events may let a warp read a raw
slot before its row has landed.  The order of the two waits is the source's.  No GPU."""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "glm53f-afd_b200", "csrc", "kda_chain.cu")


def waits():
    """For every place where the role waits for a row: the barriers in the order it waits for them."""
    with open(SOURCE) as f:
        role = f.read().split("void layer_prologue_role(", 1)[1].split("\n// ---- the recurrence", 1)[0]
    lines = [re.findall(r"mbar_wait\(&(\w+)\[", line) for line in role.splitlines()]
    return [tuple(x) for x in lines if x]


def depths():
    """The rings' depths with f32 and with bf16 states, in layer calls."""
    with open(SOURCE) as f:
        text = f.read()
    rings = [re.search(r"%s = MODE == kLayer \? \(sizeof\(S\) == 4 \? (\d+) : (\d+)\)" % ring, text).groups() for ring in ("kRawSlots", "kRowSlots")]
    assert rings[0] == rings[1]
    return tuple(int(x) for x in rings[0])


def stale_read(slots, order, seed, rows=40, single=0.0, teams=1):
    """One random run; whether a row was cooked before its copy had landed.  `single`: the share of rows cooked by a team of four warps,
    the teams in turn."""
    r = random.Random(seed)
    cooks, turn, team, warps = [], 0, 0, 4 * teams
    for _ in range(rows):
        if r.random() < single:
            cooks.append(tuple(range(4 * (team % teams), 4 * (team % teams) + 4)))
            team += 1
        else:
            cooks.append((turn % warps,))
            turn += 1
    phases = {"raw_full": [0] * slots, "row_empty": [0] * slots}  # phases completed
    raw_free, issued, released, landed, cooked, seen, at = [0] * slots, 0, 0, set(), set(), {}, [0] * warps
    while released < rows:
        moves = [("land", x) for x in range(issued) if x not in landed]
        if issued < rows and raw_free[issued % slots] >= issued // slots:
            moves.append(("issue", issued))
        if released in cooked:
            moves.append(("release", released))
        for w in range(warps):
            while at[w] < rows and w not in cooks[at[w]]:
                at[w] += 1
            if at[w] < rows:
                moves.append(("warp%d" % w, at[w]))
        what, x = r.choice(moves)
        s, lap = x % slots, x // slots
        if what == "issue":
            issued += 1
        elif what == "land":
            landed.add(x)
            phases["raw_full"][s] += 1
        elif what == "release":
            phases["row_empty"][s] += 1
            released += 1
        else:
            # a wait for phase parity P ends when the barrier's current phase has the other parity
            done = {"raw_full": phases["raw_full"][s] & 1 != lap & 1, "row_empty": phases["row_empty"][s] & 1 == lap & 1}
            k = seen.get((what, x), 0)
            seen[what, x] = k + (k < 2 and done[order[k]])
            if all(seen.get(("warp%d" % v, x), 0) == 2 for v in cooks[x]):
                if x not in landed:
                    return True
                cooked.add(x)
                raw_free[s] += 1
                for v in cooks[x]:
                    at[v] = x + 1
    return False


def test_the_model_finds_the_order_that_fails():
    assert any(stale_read(5, ("raw_full", "row_empty"), seed) for seed in range(40))


@pytest.mark.parametrize("slots", [5, 8, *depths()])
@pytest.mark.parametrize("single", [0.0, 0.3])
def test_no_row_is_read_before_it_has_landed(slots, single):
    orders = waits()
    assert len(orders) == 2 and all(len(o) == 2 for o in orders)  # rows cooked together, rows by one warp
    for order in set(orders):
        assert not any(stale_read(slots, order, seed, single=single) for seed in range(300)), order


def test_the_model_finds_rings_too_short_for_two_teams():
    order = ("row_empty", "raw_full")
    assert any(stale_read(6, order, seed, single=0.5, teams=2) for seed in range(150))


@pytest.mark.parametrize("slots", [9, depths()[1]])  # more than the eight warps: the rows between two of a warp's own
@pytest.mark.parametrize("single", [0.1, 0.5, 0.9, 1.0])
def test_two_teams_read_no_row_before_it_has_landed(slots, single):
    for order in set(waits()):
        assert not any(stale_read(slots, order, seed, single=single, teams=2) for seed in range(150)), order
