"""What the pairs of CTAs of the products of many tokens work on (csrc/wide_plan.cuh), on the CPU."""
import pytest

from bee2bee_b200 import ops


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("may_split", [False, True])
@pytest.mark.parametrize("pairs", [2, 6, 66, 74])
def test_arrivals_have_a_waiter(pairs, may_split, overlap):
    """Every tile is worked on (by both pairs of a cluster where it is cut).  The readers of an accumulator arrive on another CTA's barrier where a later product
    waits for them (the next one where the accumulators overlap, else the one after it) and nowhere else: that CTA may have left."""
    for tok_tiles, feature_tiles in [(1, 1), (1, pairs), (1, pairs + 1), (3, pairs), (2, pairs - 1), (5, pairs + 3), (1, 3 * pairs + pairs // 2)]:
        items = ops.native().gemm_wide_plan(tok_tiles, feature_tiles, 64, pairs, may_split, overlap)
        tiles = tok_tiles * feature_tiles
        rest = tiles % pairs
        cut = set(range(tiles - rest, tiles)) if may_split and 0 < rest <= pairs // 2 else set()
        seen = [t for mine in items for t, _ in mine]
        assert sorted(seen) == sorted(list(range(tiles)) + sorted(cut))
        for mine in items:
            gap = 1 if overlap else 2
            assert [sent for _, sent in mine] == [i + gap < len(mine) for i in range(len(mine))]
