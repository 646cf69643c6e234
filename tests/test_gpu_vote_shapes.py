"""The vote pass's two block shapes count the same cells.

A lookup with more reference points than the GPU has SMs runs small models in
narrow blocks; one with fewer always runs in wide ones.  The reference points
of a scene at a multiple of a stride are among those at the stride, so their
cells have to be the same, code for code and count for count.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(rng, n, centres):
    """Points on a sphere with radial normals, in tight bunches around the centres if there are any."""
    q = rng.normal(size=(n, 3)) if centres is None else centres[np.arange(n) % len(centres)]
    q = q / np.linalg.norm(q, axis=1, keepdims=True)
    p = 0.05 * q + rng.normal(scale=1e-4, size=(n, 3))
    return p.astype(np.float32), q.astype(np.float32)


@pytest.mark.parametrize("n_model,n_scene,narrow,wide,centres", [
    (2, 150, 1, 2, 0), (33, 149, 1, 3, 0), (300, 151, 1, 2, 0), (511, 700, 1, 7, 0), (830, 1000, 1, 9, 0),
    (831, 1000, 1, 9, 0), (832, 1000, 1, 9, 0),  # the last size that fits a narrow block, and the next
    (400, 3700, 12, 36, 4), (400, 7300, 24, 72, 9),  # more events than a narrow block holds at a time
    (831, 4000, 16, 48, 2)])  # long groups
def test_cells_do_not_depend_on_the_block_shape(pkg, ctx, n_model, n_scene, narrow, wide, centres):
    rng = np.random.default_rng(n_model * 10000 + n_scene)
    c = rng.normal(size=(centres, 3)) if centres else None
    d = 0.02
    m, s = _cloud(rng, n_model, c), _cloud(rng, n_scene, c)
    model = pkg.Model(m, d, 0.3, context=ctx)
    assert -(-n_scene // wide) < 148 < -(-n_scene // narrow) and wide % narrow == 0
    want_codes, want_counts = model.all_votes(pkg.Scene(s, d, wide, context=ctx))
    codes, counts = model.all_votes(pkg.Scene(s, d, narrow, context=ctx))
    both = (codes >> np.uint64(32)) % np.uint64(wide) == 0
    assert np.array_equal(codes[both], want_codes) and np.array_equal(counts[both], want_counts)
    assert len(want_codes) > 0 or n_model == 2
