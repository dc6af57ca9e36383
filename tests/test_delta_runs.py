"""The rule that cuts the delta rule's state walks into runs (``ops/csrc/deltanet_chunk.cu``), restated and checked
against what it stands on: a run may start where no state comes in."""
import random

import pytest

CHUNK = 64


def _sequence_ids(lengths):
    n = -(-sum(lengths) // CHUNK)
    ids = [i for i, length in enumerate(lengths) for _ in range(length)]
    return ids + [2**31 - 1] * (n * CHUNK - len(ids)), n


def _run_start(sid, n, c):
    """The kernels' search for a run's first chunk (32 lanes, monotone sequence ids), restated."""
    if c <= 0 or c >= n:
        return min(max(c, 0), n)
    before, lo, hi = sid[(c - 1) * CHUNK], c, n
    while lo < hi:
        step = (hi - lo + 31) >> 5
        past = [lo + lane * step >= hi or sid[(lo + lane * step) * CHUNK] != before for lane in range(32)]
        if not any(past):
            lo += 31 * step + 1
            continue
        first = past.index(True)
        hi = min(hi, lo + first * step)
        lo = lo + (first - 1) * step + 1 if first else hi
    return lo


def _warm(sid, n, s):
    return int(0 < s < n and sid[s * CHUNK - 1] == sid[s * CHUNK])


@pytest.mark.parametrize("seed", range(40))
def test_runs_take_every_chunk_once_and_start_without_a_state(seed):
    r = random.Random(seed)
    for _ in range(20):
        longest = r.choice([3, 64, 100, 700, 3000])
        sid, n = _sequence_ids([r.choice([r.randint(1, longest), 64, 128]) for _ in range(r.choice([1, 2, 5, 30]))])
        passes_on = [False] + [sid[c * CHUNK + 63] == sid[c * CHUNK - 1] for c in range(1, n)]     # Gc of a chunk != 0
        for c in range(n + 1):
            plain = 0 if c == 0 else next((s for s in range(c, n) if sid[s * CHUNK] != sid[(s - 1) * CHUNK]), n)
            assert _run_start(sid, n, c) == plain
        bucket = max(1, -(-n * r.choice([1, 12, 32, 48, 128]) // 592))
        forward, reverse = [0] * n, [0] * n
        for y in range(-(-n // bucket)):
            first, end = _run_start(sid, n, y * bucket), _run_start(sid, n, (y + 1) * bucket)
            if first >= end:
                continue
            for c in range(first, end):
                forward[c] += 1
            if first:                     # the chunk before passes nothing of its own past on, or is another sequence's
                assert not passes_on[first - 1] if _warm(sid, n, first) else sid[first * CHUNK - 1] != sid[first * CHUNK]
            low, high = first - _warm(sid, n, first), end - _warm(sid, n, end)
            for c in range(low, high):
                reverse[c] += 1
            if low < high < n:
                assert not passes_on[high] if _warm(sid, n, end) else sid[high * CHUNK - 1] != sid[high * CHUNK]
        assert forward == reverse == [1] * n
