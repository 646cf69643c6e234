"""The request loop's admission against the device memory that requests take.

One worker is kept busy by a first request while others queue; it then admits
as many of those as its budget allows.  The high-water mark of the device's
pool has to stay within the budget, for a scene that keeps nearly every
candidate cell as for one that keeps few, and a batch has to use a good part
of it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Pool:
    """Bytes in use in the device's stream-ordered pool."""

    def __init__(self):
        from cuda.bindings import driver, runtime

        self.rt, self.u64 = runtime, driver.cuuint64_t
        err, self.pool = runtime.cudaDeviceGetDefaultMemPool(0)
        assert int(err) == 0

    def _get(self, name):
        err, value = self.rt.cudaMemPoolGetAttribute(self.pool, getattr(self.rt.cudaMemPoolAttr, name))
        assert int(err) == 0
        return int(value)

    def reset(self):
        attr = self.rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
        assert int(self.rt.cudaMemPoolSetAttribute(self.pool, attr, self.u64(0))[0]) == 0
        return self._get("cudaMemPoolAttrUsedMemCurrent")

    def high(self):
        return self._get("cudaMemPoolAttrUsedMemHigh")


def _sparse(pkg):
    """About 1.4 M candidate cells, of which 40 thousand are kept."""
    spec = pkg.synthetic.config_plain(seed=6, n_model=2000, n_plane=6000, n_box=2000)
    return spec.models[0], spec.scene, float(spec.d_dists[0]), 5


def _dense(pkg):
    """A flat model on a ground plane: nearly every candidate cell is kept."""
    rng = np.random.default_rng(3)
    s = pkg.synthetic
    model = s.spheres_on_slab(rng, 800)
    placed = s.transform(model, s.make_pose(s.uniform_rotation(rng), [0.0, 0.02, 0.05]))
    scene = s.Cloud.concat([placed, s.ground_plane(rng, 30000, -0.1, 0.15)])
    return model, scene, float(s.d_dist_for(model, 0.1)), 151


@pytest.mark.parametrize("make,budget_mb,queued", [(_sparse, 500, 24), (_dense, 1500, 8)])
def test_batches_stay_within_the_budget_and_use_it(pkg, ctx, make, budget_mb, queued):
    m, s, d, df = make(pkg)
    model = pkg.Model(m, d, 0.3, context=ctx)
    want = model.ppf_lookup(pkg.Scene(s, d, df, context=ctx))
    srv = pkg.Server([model], memory_budget=budget_mb << 20, workers=1, max_batch=64)
    srv.wait(srv.submit(s, [0], df))  # the context's own buffers are there from here on
    pool = _Pool()
    before = pool.reset()
    tickets = [srv.submit(s, [0], df) for _ in range(queued + 1)]
    poses = [srv.wait(t)[0] for t in tickets]
    srv.close()
    used = pool.high() - before
    assert all(np.array_equal(p[0], want) for p in poses)
    assert used < budget_mb << 20
    assert used > 0.5 * (budget_mb << 20)
