"""CPU: how the CTAs of the uneven batch's kernel take their items.  Each CTA holds a few
items ahead of the one it works on and waits, at an item's turn, for every item that it
reads.  The model runs with any number of CTAs of the grid resident; a CTA that is not
starts only when a resident one has left.  Taken by ticket, in order, every list ends;
dealt by CTA number (item k of CTA b is entry b + k * grid), a list with dependencies
does not end unless the whole grid is resident."""
import random

import pytest

AHEAD = 3  # tickets that a CTA holds beyond its current item


def _work_list(rng):
    """[(segment, needs)]: producers before consumers, needs = index of the segment read or -1."""
    phases, segments = [], []
    for _ in range(rng.randint(1, 5)):
        chain, dep = rng.randint(1, 3), -1
        for phase in range(chain):
            segments.append((phase, dep, rng.randint(1, 40)))
            dep = len(segments) - 1
    for phase in range(3):
        for s, (ph, dep, tiles) in enumerate(segments):
            if ph == phase:
                phases += [(s, dep)] * tiles
    return phases, [tiles for _, _, tiles in segments]


def _runs_to_end(items, tiles, grid, resident, rng, by_ticket):
    done = [0] * len(tiles)
    state = {"next": 0}

    def take(cta):
        if by_ticket:
            w, state["next"] = state["next"], state["next"] + 1
        else:
            w = cta["id"] + cta["taken"] * grid
        cta["taken"] += 1
        return w if w < len(items) else None

    waiting = [{"id": i, "taken": 0, "held": []} for i in range(grid)]
    running, finished = [], 0
    while finished < len(items):
        while waiting and len(running) < resident:
            cta = waiting.pop(0)
            cta["held"] = [take(cta) for _ in range(rng.randint(1, AHEAD + 1))]
            running.append(cta)
        ready = [c for c in running if c["held"][0] is None or items[c["held"][0]][1] < 0
                 or done[items[c["held"][0]][1]] >= tiles[items[c["held"][0]][1]]]
        if not ready:
            return False  # every running CTA waits for items that no running CTA will do
        cta = rng.choice(ready)
        w = cta["held"].pop(0)
        if w is None:
            running.remove(cta)
            continue
        done[items[w][0]] += 1
        finished += 1
        while len(cta["held"]) < rng.randint(1, AHEAD + 1):
            cta["held"].append(take(cta))
    return True


@pytest.mark.parametrize("resident", [1, 2, 5, 11, 12])
def test_tickets_end_with_any_number_of_resident_ctas(resident):
    rng = random.Random(resident)
    for _ in range(300):
        items, tiles = _work_list(rng)
        assert _runs_to_end(items, tiles, 12, resident, rng, by_ticket=True)


def test_the_model_shows_that_a_fixed_deal_needs_the_whole_grid():
    rng = random.Random(1)
    items, tiles = [(0, -1)] * 12 + [(1, 0)] * 12, [12, 12]
    assert _runs_to_end(items, tiles, 12, 12, rng, by_ticket=False)
    assert not _runs_to_end(items, tiles, 12, 11, rng, by_ticket=False)
