"""Host-buffer batches at the size where their large arrays stop passing through the pinned image (256 KB an array:
16 queries of ring 2048): the words are those of single calls on both sides of it, and a refused batch writes no result."""
import ctypes

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, GAMMA, SHARDS = 2048, 16, 3


@pytest.fixture(scope="module")
def served():
    pkg = load_package()
    rng = np.random.default_rng(16)
    crs = pkg.ServerCrs(pkg.InspireParams.d2048(), rng.bytes(32), GAMMA)
    cache = pkg.ServerInspiringCache.new(crs)
    db = pkg.EncodedDatabase.from_columns(cache, [rng.integers(0, 1 << 16, (GAMMA, N), dtype=np.uint64) for _ in range(SHARDS)])
    db.precompute_packing_all()
    store = pkg.ServerSessionStore.new(pkg.Context.default())
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, (3, N), dtype=np.uint64), GAMMA)
    return pkg, rng, db, store, store.register_server_side(keys, cache)


def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


@pytest.mark.parametrize("seeded", [True, False])
def test_batches_around_the_direct_size(served, seeded):
    pkg, rng, db, store, handle = served
    ctx = pkg.Context.default()
    fn = ctx._lib.ig_respond_seeded_batch if seeded else ctx._lib.ig_respond_batch
    count = 33
    ids = rng.integers(0, SHARDS, count).astype(np.uint32)
    first = (rng.integers(0, 256, (count, 32), dtype=np.uint8) if seeded
             else rng.integers(0, pkg.DEFAULT_Q, (count, N), dtype=np.uint64))
    bs = rng.integers(0, pkg.DEFAULT_Q, (count, N), dtype=np.uint64)

    def call(lo, hi, shard_ids=ids):
        # Results at an odd offset of a larger buffer: the words around them stay.
        buf = np.full((2, (hi - lo) * N + 5), 7, np.uint64)
        a, b = buf[0, 3:], buf[1, 3:]
        rc = fn(ctx.h, db.h, store.h, handle, None, 0, 0, hi - lo, _ptr(shard_ids[lo:hi]), _ptr(first[lo:hi]), _ptr(bs[lo:hi]),
                0, _ptr(a), _ptr(b))
        return rc, buf

    single = [call(i, i + 1) for i in range(count)]
    assert all(rc == 0 for rc, _ in single)
    for c in (15, 16, 17, 33):
        rc, buf = call(0, c)
        assert rc == 0
        for half in range(2):
            want = np.concatenate([s[half, 3:3 + N] for _, s in single[:c]])
            assert np.array_equal(buf[half, 3:-2], want), c
            assert (buf[half, :3] == 7).all() and (buf[half, -2:] == 7).all()
    # A shard changed since its store was built: the batch is refused and leaves its results as they were.
    db.set_shard(1, rng.integers(0, 1 << 16, (GAMMA, N), dtype=np.uint64))
    for c in (2, 33):
        rc, buf = call(0, c, np.ones(count, np.uint32))
        assert rc != 0 and (buf == 7).all()
    db.precompute_packing_all()
