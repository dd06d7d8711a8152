"""The recursion kernels over every ring they take, at the narrowest widths and a wide one, both
gadgets, under one, two and four CTAs per query: each against the oracle's bytes. The transforms' pass
schedules differ by ring (their stage counts leave other remainders), and the queries' words sit at the
ends of their range, where the lazy sums are largest."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return load_package()


def edge_words(rng, shape, q):
    x = rng.integers(0, q, size=shape, dtype=np.uint64)
    pick = rng.integers(0, 4, size=shape)
    x[pick == 0] = q - 1
    x[pick == 1] = 0
    return x


@pytest.mark.parametrize("approx", [False, True])
@pytest.mark.parametrize("n,gamma", [(256, 1), (256, 2), (256, 128), (512, 4), (512, 64), (1024, 2), (1024, 32),
                                     (2048, 1), (2048, 2), (2048, 16)])
def test_rings(pkg, oracle, n, gamma, approx):
    rng = np.random.default_rng(n + 7 * gamma + approx)
    ctx = pkg.Context.default()
    params = pkg.InspireParams(ring_dim=n, approximate_packing_gadget=approx)
    P = oracle.Params(n=n, approx=approx)
    w_seed = rng.bytes(32)
    crs = pkg.ServerCrs(params, w_seed, gamma)
    cache = pkg.ServerInspiringCache.new(crs, ctx=ctx)
    cols = rng.integers(0, 1 << 16, size=(gamma, n), dtype=np.uint64)
    cols[0, ::3] = 0xFFFF
    db = pkg.EncodedDatabase.from_columns(cache, [cols])
    db.precompute_packing_all()
    y = edge_words(rng, (params.packing_key_rows(), n), pkg.DEFAULT_Q)
    keys = pkg.ClientPackingKeys(y, gamma)
    queries = [pkg.ClientQuery(0, edge_words(rng, n, pkg.DEFAULT_Q), edge_words(rng, n, pkg.DEFAULT_Q)) for _ in range(3)]
    ocache = oracle.Cache(P, gamma, w_seed)
    want = [ocache.respond_per_query(cols, q.a, q.b, y) for q in queries]
    batch = pkg.SeededQueryBatch(pkg.PackingKeySource.Inline(keys), queries)
    for ctas in (1, 2, 4):
        ctx.set_launch_shape(ctas)
        try:
            out = pkg.respond_seeded_batch(crs, db, batch, cache)
        finally:
            ctx.set_launch_shape(0)
        for r, (a, b) in zip(out, want):
            assert np.array_equal(r.a, a) and np.array_equal(r.b[:gamma], b[:gamma]), (n, gamma, approx, ctas)
