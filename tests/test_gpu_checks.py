"""The self-checking build (PPF_B200_CHECKS=1) finds nothing and counts the same.

A context made under the variable runs the bounds-checked instances of the
vote kernels and the check of the model tables; either one raises on the first
index or table entry that is out of place.  Cells, kept votes and poses have
to be those of an unchecked context.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def checked(pkg, ctx, monkeypatch):
    monkeypatch.setenv("PPF_B200_CHECKS", "1")
    c = pkg.Context(0)
    yield c
    c.close()


def _plain(pkg, n_model, tau=None):
    spec = pkg.synthetic.config_plain(seed=n_model, n_model=n_model, n_plane=700, n_box=300)
    d = spec.d_dists[0] if tau is None else pkg.synthetic.d_dist_for(spec.models[0], tau)
    return spec.models[0], spec.scene, float(d)


def _copies(pkg, n_model, tau, copies):
    """Noisy copies of the model: more runs per reference point than a list holds at a fine quantum."""
    rng = np.random.default_rng(n_model)
    model = pkg.synthetic.superellipsoid(rng, n_model)
    scene = pkg.synthetic.Cloud.concat([pkg.synthetic.add_noise(rng, model, 2e-4, 3.0) for _ in range(copies)])
    return model, scene, float(pkg.synthetic.d_dist_for(model, tau))


def _planes(pkg):
    """One long run of a flat model and more scene pairs than a list holds: counters past 16 bits, several lists."""
    rng = np.random.default_rng(4)
    model = pkg.synthetic.ground_plane(rng, 600, 0.0, 0.1)
    return model, pkg.synthetic.ground_plane(rng, 16000, 0.3, 0.1), 0.08


CASES = {
    "narrow": (lambda p: _plain(p, 300), 1),
    "narrow, two chunks of 831 rows": (lambda p: _plain(p, 1662), 3),
    "wide": (lambda p: _plain(p, 900), 9),
    "wide, two chunks": (lambda p: _plain(p, 1700), 9),
    "pairs past the feature table": (lambda p: _plain(p, 700, 0.005), 3),
    "lists closed by their groups, wide": (lambda p: _copies(p, 1700, 0.005, 2), 50),
    "lists closed by their groups, narrow": (lambda p: _copies(p, 700, 0.005, 2), 1),
    "several lists, spilled counters": (_planes, 4000),
}


def _all(pkg, context, m, s, d, df):
    model = pkg.Model(m, d, 0.3, context=context)
    scene = pkg.Scene(s, d, df, context=context)
    cells = model.all_votes(scene)
    pose = model.ppf_lookup(scene, raise_on_no_votes=False)
    return (*cells, pose, *model.get_votes()), model.stats["max_vote_count"]


@pytest.mark.parametrize("name", list(CASES))
def test_checked_lookups_equal_unchecked_ones(pkg, ctx, checked, name):
    make, df = CASES[name]
    m, s, d = make(pkg)
    want, top = _all(pkg, ctx, m, s, d, df)
    got, _ = _all(pkg, checked, m, s, d, df)
    assert len(want[0]) > 0
    if "spilled" in name:
        assert top > 65535
    for x, y in zip(want, got):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("sizes", [(300, 500, 831), (300, 1700)])  # all narrow; one wide model
def test_checked_batches_equal_single_lookups(pkg, ctx, checked, sizes):
    specs = [_plain(pkg, n) for n in sizes]
    want = [_all(pkg, ctx, m, s, d, 2)[0] for m, s, d in specs]
    models = [pkg.Model(m, d, 0.3, context=checked) for m, s, d in specs]
    scenes = [pkg.Scene(s, d, 2, context=checked) for m, s, d in specs]
    poses = pkg.lookup_batch(models, scenes, context=checked)
    for model, pose, w in zip(models, poses, want):
        assert np.array_equal(pose, w[2])
        for x, y in zip(model.get_votes(), w[3:]):
            assert np.array_equal(x, y)
