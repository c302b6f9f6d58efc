"""Tile tickets of the persistent step kernels, checked on the CPU.

A block of line_kernel refills its two stages with the tiles whose numbers it
drew from one counter, works through the stages in turn and stops at the
first that has no tile.  So the numbers a block draws must grow in the order
of its stages.  The model runs that loop over many blocks in random order;
the sources are searched for draws by more than one lane of a warp, whose
values CUDA hands out in no stated order.
"""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlb_b200", "csrc")
STAGES = 2


def collided(grid, ntiles, rng, swap):
    """How often each tile is collided by `grid` blocks; swap: a block's first
    two numbers reach its stages in the other order."""
    count = [0] * ntiles
    counter = STAGES * grid
    held, refill, turn = [], [], [0] * grid
    for b in range(grid):
        held.append([b + n * grid for n in range(STAGES)])
    for b in rng.sample(range(grid), grid):
        first = [counter + n for n in range(STAGES)]
        counter += STAGES
        refill.append((b, first[::-1] if swap else first))
    refill = dict(refill)
    running = list(range(grid))
    while running:
        b = rng.choice(running)
        s = turn[b] % STAGES
        if held[b][s] >= ntiles:
            running.remove(b)
            continue
        count[held[b][s]] += 1
        held[b][s] = refill[b][s]
        if held[b][s] < ntiles:
            refill[b][s] = counter
            counter += 1
        turn[b] += 1
    return count


# fewer tiles than blocks, the end inside the first two tiles, inside the
# first refills, beyond them
@pytest.mark.parametrize("ntiles", [3, 11, 15, 16, 17, 23, 31, 32, 33, 100])
def test_every_tile_is_collided_once(ntiles):
    rng = random.Random(ntiles)
    for _ in range(50):
        assert collided(8, ntiles, rng, swap=False) == [1] * ntiles


def test_numbers_out_of_order_lose_a_tile():
    assert collided(8, 17, random.Random(1), swap=True) != [1] * 17


def test_one_lane_takes_a_blocks_tickets():
    uses = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"\btake_tiles?\(", text):
            # the nearest condition before the call
            conds = re.findall(r"\bif \(([^()]*(?:\([^()]*\)[^()]*)*)\)", text[:m.start()])
            uses.append((name, conds[-1] if conds else ""))
    assert len(uses) >= 3
    for name, cond in uses:
        assert cond == "lane == 0", f"{name}: tickets drawn under `{cond}`"
