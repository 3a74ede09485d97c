"""Exclusive scans at the sizes where their launches change (GPU): one CTA up to 8,192 elements,
one cluster up to 32,768 / 65,536 / 131,072, tile sums beyond. The generator scans its row
lengths, a sort 256 counts per 4,096 pairs."""
import numpy as np
import pytest

from oracle import vite_oracle as vo

pytestmark = pytest.mark.gpu

LIMITS = [8192, 32768, 65536, 131072]


@pytest.mark.parametrize("n", [x + d for x in LIMITS for d in (-2, -1, 0)])
def test_offsets_of_as_many_rows(ctx, n):
    """the generator scans n + 1 row lengths in place"""
    ref = vo.rgg(n)
    g = ctx.generate_rgg(n)
    rowptr, tail, weight = g.download()
    np.testing.assert_array_equal(rowptr, ref.rowptr)
    np.testing.assert_array_equal(tail, ref.tail)
    np.testing.assert_array_equal(weight, ref.weight)
    g.free()


@pytest.mark.parametrize("tiles", [x // 256 + d for x in LIMITS for d in (0, 1)])
def test_sorts_of_as_many_tiles(ctx, tiles):
    n = tiles * 4096
    rng = np.random.default_rng(tiles)
    truth, found = rng.integers(0, n // 50, n), rng.integers(0, n // 20, n)
    got, ref = ctx.compare_communities(truth, found), vo.compare(truth, found)
    for key, want in ref.items():
        assert got[key] == want, key
