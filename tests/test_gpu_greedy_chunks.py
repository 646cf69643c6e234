"""Greedy pose clustering at the edges of its 1024-pose chunks.

Poses are rotations about one axis and translations along another on a coarse
grid, so no distance or angle lies near a threshold and the host restatement
takes the same decisions: results are compared exactly.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,places", [
    (1, 1), (2, 2), (31, 4), (32, 40), (33, 33), (1023, 7), (1024, 1024), (1025, 300), (2049, 2049), (5000, 1500)])
def test_chunks_equal_host(pkg, ctx, oracle, n, places):
    rng = np.random.default_rng(n + places)
    k = rng.permutation(np.arange(n) % places)
    T = np.zeros((n, 4, 4), np.float32)
    angle = 0.5 * (k % 7) + 0.03 * rng.integers(0, 2, n)
    T[:, 0, 0] = T[:, 1, 1] = np.cos(angle)
    T[:, 1, 0] = np.sin(angle)
    T[:, 0, 1] = -T[:, 1, 0]
    T[:, 2, 2] = T[:, 3, 3] = 1
    T[:, 0, 3] = 0.1 * (k // 7) + 0.004 * rng.integers(0, 2, n)
    votes = rng.integers(1, 9, n).astype(np.uint32)
    d, rot = 0.01, 2 * np.float32(np.pi) / 30
    gp, gv = pkg.cluster_poses(T, votes, d, rot, context=ctx)
    hp, hv = oracle.cluster_poses(T, votes, d, rot)
    assert len(gv) == min(3, places)
    assert np.array_equal(gv, hv)
    assert np.array_equal(gp, hp)
