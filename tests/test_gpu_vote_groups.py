"""The vote pass's event groups: votes add up over the scene's points.

The votes of a scene reference point are a sum over the other scene points, so
the vote cells of a scene equal the sums of the cells of its parts, count for
count.  Parts of five points are counted vote by vote; the whole goes through
the grouped paths (swept pieces, several pieces per group, several lists per
reference point, 16-bit counters that spill).  All model points lie on circles
around the first one's normal, so that whole circles share one key and the
groups and runs have the sizes asked for.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circles(rng, radii_heights, n, jitter):
    """p0 at the origin with normal +z, then n points on circles around z with normals turned alike."""
    k = np.arange(n) % len(radii_heights)
    r, h = np.array(radii_heights)[k].T
    phi = rng.uniform(0, 2 * np.pi, n)
    p = np.stack([r * np.cos(phi), r * np.sin(phi), h], 1) + rng.normal(scale=jitter, size=(n, 3))
    q = np.stack([0.6 * np.cos(phi), 0.6 * np.sin(phi), np.full(n, 0.8)], 1)
    p = np.concatenate([np.zeros((1, 3)), p]).astype(np.float32)
    q = np.concatenate([[[0.0, 0.0, 1.0]], q]).astype(np.float32)
    return p, q


def _cells(pkg, ctx, model, p, q, d):
    scene = pkg.Scene((p, q), d, len(p) + 1, context=ctx)  # point 0 is the only reference point
    codes, counts = model.all_votes(scene)
    return codes, counts.astype(np.uint64)


def _sum_of_parts(pkg, ctx, model, p, q, d, step):
    codes, counts = [], []
    for b in range(1, len(p), step):
        part = np.r_[0, b:min(b + step, len(p))]
        c, n = _cells(pkg, ctx, model, p[part], q[part], d)
        codes.append(c)
        counts.append(n)
    codes, counts = np.concatenate(codes), np.concatenate(counts)
    keys, where = np.unique(codes, return_inverse=True)
    total = np.zeros(len(keys), np.uint64)
    np.add.at(total, where, counts)
    return keys, total


@pytest.mark.parametrize("n_model,n_scene,circles", [
    (1, 6, 1), (1, 7, 1), (127, 8, 1), (128, 31, 1), (129, 33, 1), (300, 7, 1), (300, 254, 1), (300, 255, 1),
    (511, 256, 1), (513, 257, 2), (1700, 40, 1),  # two chunks
    (700, 1300, 9), (3400, 600, 5)])
def test_cells_add_up_over_scene_points(pkg, ctx, n_model, n_scene, circles):
    rng = np.random.default_rng(n_model * 1000 + n_scene)
    rh = [(0.05 + 0.006 * c, 0.01 * (c % 3)) for c in range(circles)]
    mp, mq = _circles(rng, rh, n_model, 1e-5)
    sp, sq = _circles(rng, rh, n_scene, 1e-5)
    d = 0.013
    model = pkg.Model((mp, mq), d, 0.3, context=ctx)
    codes, counts = _cells(pkg, ctx, model, sp, sq, d)
    keys, total = _sum_of_parts(pkg, ctx, model, sp, sq, d, 5)
    assert len(codes) > 0
    assert np.array_equal(codes, keys) and np.array_equal(counts, total)


@pytest.mark.parametrize("copies", [255, 256, 7168, 7169, 40000])
def test_copies_of_points_multiply_the_cells(pkg, ctx, copies):
    """More events than one list holds, and counts far past 16 bits."""
    rng = np.random.default_rng(copies)
    mp, mq = _circles(rng, [(0.05, 0.0)], 600, 1e-6)
    sp, sq = _circles(rng, [(0.05, 0.0)], 3, 1e-6)
    d = 0.02
    model = pkg.Model((mp, mq), d, 0.3, context=ctx)
    codes, counts = _cells(pkg, ctx, model, sp, sq, d)
    rep = np.r_[0, np.repeat([1, 2, 3], copies)]
    codes2, counts2 = _cells(pkg, ctx, model, sp[rep], sq[rep], d)
    assert len(codes) > 0
    assert np.array_equal(codes, codes2) and np.array_equal(counts * np.uint64(copies), counts2)


def test_scene_with_another_quantum_hashes_every_pair(pkg, ctx):
    """The model's feature table holds for its own quantum only; a scene with
    another one, or points further apart than the table's rows, is looked up
    by key.  Both give the counts of pair_vote_counts."""
    spec = pkg.synthetic.config_plain(seed=191, n_model=300, n_plane=500, n_box=200)
    m, s, d = spec.models[0], spec.scene, spec.d_dists[0]
    far = s.points.copy()
    far[::7] += np.float32(3.0)  # about 300 quanta away: past the table, and past the row flags at 40
    far[::11] += np.float32(40.0)
    for scene_d, pts in ((d, s.points), (d, far), (np.float32(1.37) * np.float32(d), s.points)):
        model = pkg.Model(m, d, 0.3, context=ctx)
        scene = pkg.Scene((pts, s.normals), float(scene_d), 5, context=ctx)
        model.ppf_lookup(scene, raise_on_no_votes=False)
        counts = model.pair_vote_counts(scene)
        assert model.stats["n_votes"] == int(counts.sum())
        assert model.stats["n_matched_pairs"] == int(np.count_nonzero(counts))
        codes, n = model.all_votes(scene)
        assert int(n.sum()) == int(counts.sum())
