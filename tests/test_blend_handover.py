"""How the cooperative blend's warps learn that all pixels have stopped
(rasterize_kernel, dg_render.cu): warp 0 writes round r's word, one barrier ends the
round, and every warp reads the word and leaves the loop or goes on. Every order of two
warps' steps is walked here, on the CPU: all must leave after the round that warp 0
stopped in, since a warp that leaves earlier meets the others at the wrong barrier."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "diorama_gb300" / "csrc" / "dg_render.cu"


def last_rounds(words: int, stop_round: int) -> set:
    """The (warp, round) pairs at which a warp may leave the loop, over all interleavings."""
    left = set()
    seen = set()
    # Each warp: (round, step), step 0 before the round's barrier, 1 waiting at it, 2 past it.
    todo = [(((0, 0), (0, 0)), (0,) * words)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        warps, flags = state
        if all(w is not None and w[1] == 1 for w in warps):  # both have arrived
            todo.append((tuple((r, 2) for r, _ in warps), flags))
            continue
        for k, warp in enumerate(warps):
            if warp is None or warp[1] == 1:
                continue
            r, step = warp
            now = flags
            if step == 0:
                if k == 0 and r > 0:
                    now = flags[: r % words] + (int(r >= stop_round),) + flags[r % words + 1:]
                after = (r, 1)
            elif flags[r % words]:
                left.add((k, r))
                after = None
            else:
                after = (r + 1, 0)
            todo.append((warps[:k] + (after,) + warps[k + 1:], now))
    return left


def test_one_word_lets_a_warp_leave_a_round_early():
    assert last_rounds(1, 3) != {(0, 3), (1, 3)}


@pytest.mark.parametrize("stop_round", [1, 2, 3, 6])
def test_all_warps_leave_after_the_same_round(stop_round):
    words = int(re.search(r"STOP_WORDS = (\d+);", SOURCE.read_text()).group(1))
    assert last_rounds(words, stop_round) == {(0, stop_round), (1, stop_round)}
