"""Waits of the GEMM epilogues that give up: each of the four warps of a part finds out by itself whether a tile's
accumulators arrived, and behind that wait lie barriers that all four have to reach. Checked on the model of their steps for
every outcome of the waits, and on the sources that the kernels take those steps."""
import itertools
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "shadowspill_b200" / "ops" / "csrc"
WARPS, TILES, BLOCKS = 4, 2, 2


def _leaves_together(outcomes, agree):
    """Four warps through their tiles; a barrier opens when all four are at it. True when every warp reaches the end."""
    def warp(w):
        for t in range(TILES):
            ok = outcomes[w][t]
            if agree:
                ok = yield ok                      # the reducing barrier: all of them have what they waited for
            if not ok:
                return
            for _ in range(2 * BLOCKS):            # two barriers for each block of columns that leaves
                yield None
    waiting = {}
    running = {w: warp(w) for w in range(WARPS)}
    for w, g in running.items():
        try:
            waiting[w] = next(g)
        except StopIteration:
            pass
    while len(waiting) == WARPS:
        every = all(v is not False for v in waiting.values())
        arrived, waiting = waiting, {}
        for w in arrived:
            try:
                waiting[w] = running[w].send(every if arrived[w] is not None else None)
            except StopIteration:
                pass
    return not waiting


@pytest.mark.parametrize("agree", [True, False])
def test_warps_that_agree_never_leave_one_at_a_barrier(agree):
    each = list(itertools.product([True, False], repeat=TILES))
    stuck = sum(not _leaves_together(o, agree) for o in itertools.product(each, repeat=WARPS))
    assert (stuck == 0) if agree else (stuck > 0)


@pytest.mark.parametrize("name", ["gemm_tcgen05.cu", "gemm_tcgen05_2cta.cu"])
def test_the_epilogues_agree_before_they_store_by_tma(name):
    source = (CSRC / name).read_text()
    wait, store = source.index("KS_TIMEOUT_TMEM_FULL"), source.index("epilogue_tma(")
    between = source[wait:store]
    assert source.count("epilogue_tma(") == 1 and wait < store
    assert re.search(r"p\.tma_out\) ok = epilogue_part_agree\(part, ok\);\s*if \(!ok\) break;", between)
    assert not re.search(r"if \(!mbar_wait\(&tfull", source)         # no warp leaves on its own
