"""Encodes over a range of shards of which only some hold a store: the tag check covers the stored ones alone. A
stored shard whose columns changed is refused until it is rebuilt, one whose columns did not change is still served,
and a shard whose store was dropped or never built stays without one and answers from its new columns."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, GAMMA, SHARDS = 256, 16, 6
KEPT, DROPPED, CHANGED, NEVER = (0, 5), 1, 2, (3, 4)


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.mark.parametrize("first", [SHARDS, 3])  # shards of the first encode
def test_encode_over_partly_stored_shards(pkg, first):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(first)
    crs = pkg.ServerCrs(pkg.InspireParams(ring_dim=N), rng.bytes(32), GAMMA)
    cache = pkg.ServerInspiringCache.new(crs)
    entry = 2 * GAMMA
    raw = rng.integers(0, 256, size=SHARDS * N * entry, dtype=np.uint8)
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, size=(3, N), dtype=np.uint64), GAMMA)
    dev = torch.from_numpy(raw).cuda()
    torch.cuda.synchronize()
    db = pkg.EncodedDatabase(cache, SHARDS)

    def encode(shards):
        torch.cuda.synchronize()
        db.encode_records(None, entry, device_ptr=dev.data_ptr(), nbytes=shards * N * entry)

    def ask(d, s):
        q = pkg.SeededClientQuery(s, bytes([s]) * 32, np.arange(N, dtype=np.uint64), inspiring_packing_keys=keys)
        r = pkg.respond_seeded_inspiring(crs, d, q)
        return r.a, r.b

    encode(first)
    built = [s for s in (*KEPT, DROPPED, CHANGED) if s < first]
    for s in built:
        db.shards[s].precompute_packing()
    db.shards[DROPPED].drop_packing_store()
    before = {s: ask(db, s) for s in KEPT if s < first}
    # One byte of the changed shard and of one without a store.
    for s in (CHANGED, NEVER[0]):
        dev[s * N * entry + 7] ^= 1
        raw[s * N * entry + 7] ^= 1
    encode(SHARDS)
    stored = [s for s in built if s != DROPPED]
    assert [s for s in range(SHARDS) if db.shards[s].packing_store()] == sorted(stored)
    ref = pkg.EncodedDatabase.from_records(cache, raw.tobytes(), entry, SHARDS)
    for s in range(SHARDS):
        if s == CHANGED:
            with pytest.raises(pkg.PirError, match="store refused"):
                ask(db, s)
            continue
        got = ask(db, s)
        for x, y in zip(got, ask(ref, s)):
            assert np.array_equal(x, y), s
        if s in before:
            for x, y in zip(got, before[s]):
                assert np.array_equal(x, y), s
    db.precompute_packing_all()
    for s in range(SHARDS):
        for x, y in zip(ask(db, s), ask(ref, s)):
            assert np.array_equal(x, y), s
