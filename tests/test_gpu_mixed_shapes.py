"""The shapes that a mixed launch of several widths plans, seen in its number of launches (a scan and one a shape): a
tuned row's times that are not above 0 are shapes that were not measured, not free ones; a row of a larger batch says
nothing of one query; a pair threshold of 0 keeps one CTA a query. Responses are the same under every plan."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, WIDTHS, EACH = 2048, (16, 64, 256), 6


@pytest.fixture
def served():
    pkg = load_package()
    rng = np.random.default_rng(24)
    ctx = pkg.Context(0)
    store = pkg.ServerSessionStore.new(ctx)
    queries = []
    for gamma in WIDTHS:
        cache = pkg.ServerInspiringCache.new(pkg.ServerCrs(pkg.InspireParams(), rng.bytes(32), gamma), ctx=ctx)
        db = pkg.EncodedDatabase.from_columns(cache, [rng.integers(0, 1 << 16, size=(gamma, N), dtype=np.uint64)])
        db.precompute_packing_all()
        keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, size=(3, N), dtype=np.uint64), gamma)
        handle = store.register_server_side(keys, cache)
        for _ in range(EACH):
            q = pkg.SeededBatchQuery(0, rng.bytes(32), rng.integers(0, pkg.DEFAULT_Q, size=N, dtype=np.uint64))
            queries.append(pkg.MixedQuery(db, store, handle, q))
    ctx.set_launch_shape(1)
    want = pkg.respond_mixed_batch(queries)
    ctx.set_launch_shape(0)

    def launches():
        before = ctx.launch_count
        out = pkg.respond_mixed_batch(queries)
        for r, w in zip(out, want):
            assert np.array_equal(r.a, w.a) and np.array_equal(r.b, w.b)
        return ctx.launch_count - before

    yield ctx, launches
    ctx.close()


def load_rows(ctx, tmp_path, rows):
    """Loads a table of `rows` ((gamma, batch, ms of 1, 2 and 4 CTAs)) for this device's SM count."""
    path = tmp_path / "shapes.txt"
    ctx.save_tuning(path)
    head = path.read_text().splitlines()[:2]
    path.write_text("\n".join(head + [" ".join(map(str, (N, g, b, *ms))) for g, b, ms in rows]) + "\n")
    ctx.load_tuning(path)


TIMES = {16: (0.12, 0.08, 0.05), 64: (0.45, 0.28, 0.18), 256: (1.8, 1.1, 0.7)}


@pytest.mark.parametrize("rows,launched", [
    # One query's times: the widest on clusters, the narrowest on one CTA.
    ([(g, 1, t) for g, t in TIMES.items()], "several"),
    # One CTA not measured: the narrowest on pairs, the widest on fours.
    ([(g, 1, (0, *t[1:])) for g, t in TIMES.items()], "several"),
    # Rows of 64 queries alone, where one CTA is the fastest: no times of one query.
    ([(g, 64, (t[0], 3 * t[0], 6 * t[0])) for g, t in TIMES.items()], "several"),
    # Clusters not measured at any width.
    ([(g, 1, (t[0], 0, 0)) for g, t in TIMES.items()], "one"),
])
def test_tuned_rows(served, tmp_path, rows, launched):
    ctx, launches = served
    load_rows(ctx, tmp_path, rows)
    assert (launches() > 2) == (launched == "several")


def test_pair_threshold(served):
    ctx, launches = served
    assert launches() > 2
    ctx.set_pair_threshold(0)
    assert launches() == 2
