"""The end of the four-CTA recursion: its two final inverse transforms share a buffer, the second's words written only
after every thread has read the first's. Many clusters at the narrowest widths, where the end is most of a query, over
the rings whose last local pass takes one bit (256, 1024) and two (512, 2048): word for word the one-CTA kernel's."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [1, 4])
@pytest.mark.parametrize("n", [256, 512, 1024, 2048])
def test_final_transforms(n, gamma):
    pkg = load_package()
    rng = np.random.default_rng(n + gamma)
    ctx = pkg.Context.default()
    params = pkg.InspireParams(ring_dim=n)
    crs = pkg.ServerCrs(params, rng.bytes(32), gamma)
    cache = pkg.ServerInspiringCache.new(crs, ctx=ctx)
    db = pkg.EncodedDatabase.from_columns(cache, [rng.integers(0, 1 << 16, size=(gamma, n), dtype=np.uint64)])
    db.precompute_packing_all()
    store = pkg.ServerSessionStore.new(ctx)
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, size=(3, n), dtype=np.uint64), gamma)
    source = pkg.PackingKeySource.Registered(store.register_server_side(keys, cache))
    queries = [pkg.SeededBatchQuery(0, rng.bytes(32), rng.integers(0, pkg.DEFAULT_Q, size=n, dtype=np.uint64))
               for _ in range(64)]
    batch = pkg.SeededQueryBatch(source, queries)

    def respond(ctas):
        ctx.set_launch_shape(ctas)
        try:
            return pkg.respond_seeded_batch(crs, db, batch, cache, store)
        finally:
            ctx.set_launch_shape(0)

    want = respond(1)
    for _ in range(20):
        for r, w in zip(respond(4), want):
            assert np.array_equal(r.a, w.a) and np.array_equal(r.b, w.b)
