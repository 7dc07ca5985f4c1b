"""Where a cut step's segments stand: the numbers that the recurrence's kernels give their blocks and the places of the
scratch (csrc/recurrence.cu, ``RecSegments``), over drawn steps."""
import random
from types import SimpleNamespace

import pytest
import torch


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


@pytest.mark.parametrize("heads,dim,vdim,counts,cut", [
    (16, 128, 128, [255], False), (16, 128, 128, [256], False), (16, 128, 128, [512], True), (16, 128, 128, [2048], True), (16, 128, 128, [300] * 4, False),
    (16, 128, 128, [512] * 4, False), (16, 128, 128, [1024] * 4, False), (28, 128, 128, [300] * 2, False), (28, 128, 128, [2048], True),
    (28, 128, 128, [512] * 2, False), (12, 128, 128, [900, 883, 531, 1080], True), (16, 128, 128, [4000] + [60] * 60, True), (8, 64, 64, [256] * 16, False),
    (2, 64, 64, [256], False), (2, 64, 64, [2048], True), (4, 200, 64, [256] * 16, False), (14, 64, 64, [300] * 4, False), (1, 16, 8, [700, 5, 256], True)])
def test_long_steps_are_cut_where_that_is_faster(heads, dim, vdim, counts, cut):
    """Steps measured both ways: the ones that were 4 % and more faster whole are left whole, the others cut."""
    from cima_b200.kernels import Kernels
    batch = SimpleNamespace(max_rows=max(counts), n_rows=sum(counts), n_seqs=len(counts))
    columns = heads * -(-vdim // 32)
    assert Kernels.recurrence_segments(Kernels, batch, columns, torch.bfloat16, dim) == (-(-max(counts) // 128) if cut else 1)
    assert Kernels.recurrence_segments(Kernels, batch, columns, torch.float32, dim) == 1
