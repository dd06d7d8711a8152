"""Store builds and encodes of several shards a launch: step-1 sums word for word the oracle's over widths with
odd and even log, compact and wide shards side by side; encodes at odd and even entry sizes, aligned and
not, with a partial last shard; a changed shard among unchanged ones is the one refused."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    return load_package()


@pytest.mark.parametrize("n,gamma", [(256, 1), (256, 2), (256, 128), (512, 4), (1024, 8), (2048, 1), (2048, 16),
                                     (2048, 32)])
def test_sums_of_mixed_shards(pkg, oracle, n, gamma):
    rng = np.random.default_rng(n + gamma)
    w_seed = rng.bytes(32)
    crs = pkg.ServerCrs(pkg.InspireParams(ring_dim=n), w_seed, gamma)
    cache = pkg.ServerInspiringCache.new(crs)
    shards = []
    for s in range(5):
        cols = rng.integers(0, 1 << 16, size=(gamma, n), dtype=np.uint64)
        if s % 2:  # wide words, some at and above q
            cols[0] = rng.integers(0, 1 << 64, size=n, dtype=np.uint64)
            cols[0, :4] = [pkg.DEFAULT_Q, pkg.DEFAULT_Q - 1, (1 << 64) - 1, 1 << 60]
        else:
            cols[-1] = 0xFFFF
        shards.append(cols)
    db = pkg.EncodedDatabase.from_columns(cache, shards)
    db.precompute_packing_all()
    ocache = oracle.Cache(oracle.Params(n=n), gamma, w_seed)
    for s, cols in enumerate(shards):
        assert np.array_equal(db.store_sums(s), oracle.Store(ocache, cols % np.uint64(pkg.DEFAULT_Q)).sums()), s


@pytest.mark.parametrize("entry,shift", [(1, 0), (31, 0), (32, 0), (32, 1), (64, 2)])
def test_encode_many_shards(pkg, entry, shift):
    torch = pytest.importorskip("torch")
    n, gamma = 256, (entry + 1) // 2
    rng = np.random.default_rng(entry + shift)
    crs = pkg.ServerCrs(pkg.InspireParams(ring_dim=n), rng.bytes(32), gamma)
    cache = pkg.ServerInspiringCache.new(crs)
    entries = 6 * n + 37  # the last shard holds 37
    raw = rng.integers(0, 256, size=entries * entry, dtype=np.uint8)
    db = pkg.EncodedDatabase(cache, 7)
    dev = torch.zeros(raw.size + shift, dtype=torch.uint8, device="cuda")
    dev[shift:] = torch.from_numpy(raw).cuda()
    torch.cuda.synchronize()
    db.encode_records(None, entry, device_ptr=dev.data_ptr() + shift, nbytes=raw.size)
    db.precompute_packing_all()
    host = np.zeros((7, n, 2 * gamma), dtype=np.uint8)
    host.reshape(-1, 2 * gamma)[:entries, :entry] = raw.reshape(entries, entry)
    words = host[..., 0::2].astype(np.uint64) | (host[..., 1::2].astype(np.uint64) << np.uint64(8))
    ref = pkg.EncodedDatabase.from_columns(cache, [w.T.copy() for w in words])
    ref.precompute_packing_all()
    for s in range(7):
        assert np.array_equal(db.store_sums(s), ref.store_sums(s)), s
    # One byte of shard 4 changes: that shard alone is refused until its store is rebuilt.
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, size=(3, n), dtype=np.uint64), gamma)

    def ask(s):
        q = pkg.SeededClientQuery(s, bytes(32), np.arange(n, dtype=np.uint64), inspiring_packing_keys=keys)
        return pkg.respond_seeded_inspiring(crs, db, q)

    before = [ask(s) for s in range(7)]
    dev[shift + 4 * n * entry] ^= 1
    torch.cuda.synchronize()
    db.encode_records(None, entry, device_ptr=dev.data_ptr() + shift, nbytes=raw.size)
    for s in range(7):
        if s == 4:
            with pytest.raises(pkg.PirError, match="store refused"):
                ask(s)
        else:
            r = ask(s)
            assert np.array_equal(r.a, before[s].a) and np.array_equal(r.b, before[s].b)
    db.shards[4].precompute_packing()
    ask(4)
