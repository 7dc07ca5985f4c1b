"""Where a cut step's segments stand: the numbers that the recurrence's kernels give their blocks and the places of the
scratch (csrc/recurrence.cu, ``RecSegments``), over drawn steps."""
import random


def test_segments_have_blocks_and_places_of_their_own():
    """Blocks from first row / seg + sequence on, places from 2 * first row / seg on for sequences of more than seg rows: no two
    segments share one, all lie within the launch and the scratch, and the search finds each block's sequence."""
    rng = random.Random(4)
    for _ in range(4000):
        seg = rng.choice([1, 2, 3, 16, 128])
        rows = [rng.choice([0, 1, seg - 1, seg, seg + 1, 2 * seg, 2 * seg + 1, rng.randint(0, 9 * seg)]) for _ in range(rng.randint(1, 12))]
        first = [sum(rows[:i]) for i in range(len(rows) + 1)]
        blocks, places = {}, {}
        for s, r in enumerate(rows):
            for i in range(-(-r // seg)):
                assert blocks.setdefault(first[s] // seg + s + i, (s, i)) == (s, i)
                if r > seg:
                    assert places.setdefault(2 * first[s] // seg + i, (s, i)) == (s, i)
        launched = first[-1] // seg + len(rows)
        assert all(b < launched for b in blocks) and all(p < 2 * first[-1] // seg for p in places)
        for b in range(launched):
            lo, hi = 0, len(rows) - 1
            while lo < hi:
                mid = (lo + hi + 1) // 2
                lo, hi = (mid, hi) if first[mid] // seg + mid <= b else (lo, mid - 1)
            i = b - (first[lo] // seg + lo)
            assert i >= 0 and ((lo, i) == blocks[b] if b in blocks else i * seg >= rows[lo])
