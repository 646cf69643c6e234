"""Kept votes whose counts pass 2^24: ordered by the count as a float.

Below 2^24 one sort of (largest count - count, code) orders the kept votes.
From there on a float no longer tells neighbouring counts apart, and the
reference's order (its sort takes the count as a float, ties by code) needs
the two sorts that this reaches.  Copies of a few points on one circle give
such counts in a few cells: every scene point votes for every model copy.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THRESHOLD = 0.005


def _circle(degrees, copies):
    """A point at the origin with normal +z and copies of points on a circle around it, with radial tilted normals."""
    phi = np.repeat(np.radians(np.asarray(degrees, np.float64)), copies)
    p = np.stack([0.05 * np.cos(phi), 0.05 * np.sin(phi), 0 * phi], 1)
    q = np.stack([0.6 * np.cos(phi), 0.6 * np.sin(phi), 0 * phi + 0.8], 1)
    return (np.concatenate([np.zeros((1, 3)), p]).astype(np.float32),
            np.concatenate([[[0.0, 0.0, 1.0]], q]).astype(np.float32))


# vote codes of 32 bits and of 33
@pytest.mark.parametrize("copies", [40000, 70000])
def test_order_of_counts_past_float_resolution(pkg, ctx, copies):
    d = 0.013
    # the single points vote once into the cell of the first group's pairs,
    # which makes its count one more than the second group's
    model = pkg.Model(_circle([0, 48, 96, 144, 204], [420, 420, 140, 20, 1]), d, THRESHOLD, context=ctx)
    scene_cloud = _circle([5, 29, 209], [copies, 500, 1])
    scene = pkg.Scene(scene_cloud, d, len(scene_cloud[0]) + 1, context=ctx)
    codes, counts = model.all_votes(scene)
    top = int(counts.max())
    assert int(counts.astype(np.uint64).sum()) == (copies + 501) * 1001 and top >= 1 << 24
    as_float = counts.astype(np.float32)
    large = counts[counts >= 1 << 24]
    assert len(np.unique(large)) > len(np.unique(large.astype(np.float32)))
    kept = as_float > np.float32(THRESHOLD) * np.float32(top)
    order = np.lexsort((codes[kept], -as_float[kept]))
    assert 4 < kept.sum() < len(codes)
    model.ppf_lookup(scene)
    got_codes, got_counts = model.get_votes()
    assert np.array_equal(got_codes, codes[kept][order]) and np.array_equal(got_counts, counts[kept][order])
