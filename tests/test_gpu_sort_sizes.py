"""The radix sort at the edges of its paths, through the model's hash array.

A model of n points sorts n * n keys: up to 4096 in one block, up to 8192 in
one tile, more in several.  The sort is stable, so the hash array's map equals
numpy's stable argsort of the pair keys, element for element.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 6, 31, 33, 64, 65, 90, 91, 127, 128, 129, 257])
def test_hash_array_is_the_stable_sort_of_the_keys(pkg, ctx, n):
    rng = np.random.default_rng(n)
    p = rng.uniform(-0.05, 0.05, (n, 3)).astype(np.float32)
    q = rng.normal(size=(n, 3)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    # many runs, few runs, and pairs past the feature table (the runs then come from sorted keys)
    for d in (0.02, 0.5, 0.0006):
        keys = pkg.pair_keys((p, q), d, 1, context=ctx).ravel()
        order = np.argsort(keys, kind="stable").astype(np.uint32)
        uniq, first, count = np.unique(keys, return_index=True, return_counts=True)
        H = pkg.Model((p, q), d, 0.3, context=ctx).hash_array()
        assert np.array_equal(H["map"], order)
        assert np.array_equal(H["keys"], uniq) and np.array_equal(H["counts"], count)
        assert np.array_equal(keys[order][H["first"]], uniq)


@pytest.mark.parametrize("n_plane,df", [(40, 1), (300, 3), (900, 2)])
def test_votes_come_in_order(pkg, ctx, n_plane, df):
    """64-bit codes, from a few cells to several tiles of them."""
    spec = pkg.synthetic.config_plain(seed=200 + n_plane, n_model=60, n_plane=n_plane, n_box=30)
    model = pkg.Model(spec.models[0], spec.d_dists[0], 0.3, context=ctx)
    scene = pkg.Scene(spec.scene, spec.d_dists[0], df, context=ctx)
    codes, counts = model.all_votes(scene)
    assert np.all(np.diff(codes.astype(np.int64)) > 0)
    model.ppf_lookup(scene)
    kept, n = model.get_votes()
    keep = counts.astype(np.float32) > np.float32(0.3) * np.float32(counts.max())
    order = np.lexsort((codes[keep], -counts[keep].astype(np.int64)))
    assert np.array_equal(kept, codes[keep][order]) and np.array_equal(n, counts[keep][order])
