"""A batch larger than the GPU: whole waves of one CTA a query, the rest in the shape of a batch of its size. Every query's
words are those of one CTA a query throughout, whichever part it falls in."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gamma,approx", [(256, 4, False), (512, 16, True)])
def test_tails(n, gamma, approx):
    torch = pytest.importorskip("torch")
    pkg = load_package()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(n)
    params = pkg.InspireParams(ring_dim=n, approximate_packing_gadget=approx)
    crs = pkg.ServerCrs(params, rng.bytes(32), gamma)
    ctx = pkg.Context.default()
    cache = pkg.ServerInspiringCache.new(crs)
    db = pkg.EncodedDatabase.from_columns(cache, [rng.integers(0, 1 << 16, (gamma, n), dtype=np.uint64) for _ in range(3)])
    db.precompute_packing_all()
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, (2 if approx else 3, n), dtype=np.uint64), gamma)
    counts = [sms + 1, sms + sms // 4, sms + sms // 4 + 1, sms + sms // 2 + 1, 2 * sms + 5]
    qs = [pkg.SeededBatchQuery(int(rng.integers(0, 3)), rng.bytes(32), rng.integers(0, pkg.DEFAULT_Q, n, dtype=np.uint64))
          for _ in range(max(counts))]

    def answers(count):
        batch = pkg.SeededQueryBatch(pkg.PackingKeySource.Inline(keys), qs[:count])
        return pkg.respond_seeded_batch(crs, db, batch, cache)

    ctx.set_launch_shape(1)
    try:
        want = answers(max(counts))
    finally:
        ctx.set_launch_shape(0)
    for count in counts:
        got = answers(count)
        assert all(np.array_equal(g.a, w.a) and np.array_equal(g.b, w.b) for g, w in zip(got, want)), count
