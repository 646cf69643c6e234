"""Vote lists that close because they hold too many groups.

A list of the vote pass takes scene pairs of at most a few hundred runs (640
groups in a wide block, 320 in a narrow one); past that every warp leaves the
walk, the list's votes are counted and the walk goes on.  The warps read the
group count while others raise it.  Fine quanta give a reference point more
groups than that with far fewer pairs than a list holds.  Votes add up over
the scene's points, and parts of 200 points never close a list.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _copies(pkg, n_model, tau, copies):
    rng = np.random.default_rng(n_model)
    model = pkg.synthetic.superellipsoid(rng, n_model)
    scene = pkg.synthetic.Cloud.concat([pkg.synthetic.add_noise(rng, model, 2e-4, 3.0) for _ in range(copies)])
    return model, scene, float(pkg.synthetic.d_dist_for(model, tau))


def _cells(pkg, ctx, model, cloud, d, df):
    return model.all_votes(pkg.Scene(cloud, d, df, context=ctx))


@pytest.mark.parametrize("n_model,tau,copies", [(700, 0.005, 2), (831, 0.004, 2), (1700, 0.01, 2), (1700, 0.005, 3)])
def test_lists_closed_by_their_groups_count_every_vote(pkg, ctx, n_model, tau, copies):
    m, s, d = _copies(pkg, n_model, tau, copies)
    model = pkg.Model(m, d, 0.3, context=ctx)
    runs = model.hash_array()["keys"]
    keys = pkg.pair_keys(s, d, 1, context=ctx)
    n = len(s.points)
    row = keys[0][np.isin(keys[0], runs)]
    assert len(np.unique(row)) > 700 and len(row) < 7000
    # one reference point: a wide block
    codes, counts = _cells(pkg, ctx, model, s, d, n + 1)
    part_codes, part_counts = [], []
    for b in range(1, n, 200):
        at = np.r_[0, b:min(b + 200, n)]
        c, k = _cells(pkg, ctx, model, (s.points[at], s.normals[at]), d, n + 1)
        part_codes.append(c)
        part_counts.append(k.astype(np.uint64))
    keys_, where = np.unique(np.concatenate(part_codes), return_inverse=True)
    total = np.zeros(len(keys_), np.uint64)
    np.add.at(total, where, np.concatenate(part_counts))
    assert len(codes) > 0
    assert np.array_equal(codes, keys_) and np.array_equal(counts.astype(np.uint64), total)


@pytest.mark.parametrize("n_model,tau,copies", [(700, 0.005, 2), (831, 0.004, 2), (1700, 0.005, 1)])
def test_every_reference_point_closes_lists(pkg, ctx, n_model, tau, copies):
    """All points as reference points (narrow blocks up to 831 rows) against few of them (wide blocks), ten times."""
    m, s, d = _copies(pkg, n_model, tau, copies)
    model = pkg.Model(m, d, 0.3, context=ctx)
    n = len(s.points)
    df = -(-n // 100)
    want_codes, want_counts = _cells(pkg, ctx, model, s, d, df)
    codes, counts = _cells(pkg, ctx, model, s, d, 1)
    both = (codes >> np.uint64(32)) % np.uint64(df) == 0
    assert len(want_codes) > 0
    assert np.array_equal(codes[both], want_codes) and np.array_equal(counts[both], want_counts)
    for _ in range(9):
        again = _cells(pkg, ctx, model, s, d, 1)
        assert np.array_equal(again[0], codes) and np.array_equal(again[1], counts)
