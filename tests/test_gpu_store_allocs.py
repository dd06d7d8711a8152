"""Store builds under failing device allocations (made to fail on the host): whichever allocation of a build fails, in a
context that has built nothing yet, no shard is left with a store that was not built, and the next build succeeds."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, GAMMA, SHARDS = 256, 16, 4


@pytest.mark.parametrize("whole", [False, True])  # one shard's build, or the database's
def test_failed_builds_leave_no_store(whole):
    pkg = load_package()
    rng = np.random.default_rng(11 + whole)
    w_seed = rng.bytes(32)
    columns = [rng.integers(0, 1 << 16, size=(GAMMA, N), dtype=np.uint64) for _ in range(SHARDS)]
    want, refused = None, 0
    for k in range(3 * SHARDS + 3 if whole else 6):  # the k-th allocation fails; 0: none does
        ctx = pkg.Context(0)
        cache = pkg.ServerInspiringCache.new(pkg.ServerCrs(pkg.InspireParams(ring_dim=N), w_seed, GAMMA), ctx=ctx)
        db = pkg.EncodedDatabase.from_columns(cache, columns)
        base = ctx.device_bytes
        build = db.precompute_packing_all if whole else db.shards[1].precompute_packing
        ctx._lib.ig_debug_fail_alloc_at(ctx.h, k)
        failed = False
        try:
            build()
        except pkg.PirError as e:
            assert e.code == 8 and "injected" in str(e)
            failed = True
        ctx._lib.ig_debug_fail_alloc_at(ctx.h, 0)
        stored = [s for s in range(SHARDS) if db.shards[s].packing_store()]
        if k == 0:
            assert not failed
            want = {s: db.store_sums(s) for s in stored}
        if failed:
            refused += 1
            assert stored == list(range(len(stored))) if whole else not stored
        else:
            assert stored == (list(range(SHARDS)) if whole else [1])
        for s in stored:
            assert np.array_equal(db.store_sums(s), want[s]), (k, s)
        build()
        for s in want:
            assert np.array_equal(db.store_sums(s), want[s]), (k, s)
        for s in range(SHARDS):
            if db.shards[s].packing_store():
                db.shards[s].drop_packing_store()
        assert ctx.device_bytes - base < SHARDS * GAMMA * N * 8 * 2  # the build's scratch alone
        ctx.close()
    # One shard's scratch and three buffers a store; a group's scratch that fails gives way to one shard's.
    assert refused == (3 * SHARDS + 1 if whole else 4)
