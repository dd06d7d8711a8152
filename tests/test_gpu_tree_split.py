"""The OnePacking tree over its splits: a batch's size decides how many subtrees a query is walked in, from one
to 32 (fewer at narrow widths, none at width one). Every split gives the oracle's words."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gamma,batches", [(256, 1, (1, 9)), (256, 2, (1, 9)), (256, 8, (1, 400)), (256, 128, (1, 40, 700)),
                                             (512, 64, (1, 50)), (2048, 16, (1, 20))])
def test_splits(oracle, n, gamma, batches):
    pkg = load_package()
    rng = np.random.default_rng(n + gamma)
    P = oracle.Params(n=n)
    logn = n.bit_length() - 1
    w_seed = rng.bytes(32)
    galois = rng.integers(0, pkg.DEFAULT_Q, size=(logn, 3, 2, n), dtype=np.uint64)
    crs = pkg.ServerCrs(pkg.InspireParams(ring_dim=n), w_seed, gamma, galois_keys=galois)
    cache = pkg.ServerInspiringCache.new(crs)
    shards = [rng.integers(0, 1 << 16, size=(gamma, n), dtype=np.uint64) for _ in range(2)]
    shards[1][0] = rng.integers(0, pkg.DEFAULT_Q, size=n, dtype=np.uint64)  # a wide shard
    db = pkg.EncodedDatabase.from_columns(cache, shards)
    ocache = oracle.Cache(P, gamma, w_seed)
    for count in batches:
        qs = []
        for i in range(count):
            a = rng.integers(0, pkg.DEFAULT_Q, size=n, dtype=np.uint64)
            b = rng.integers(0, pkg.DEFAULT_Q, size=n, dtype=np.uint64)
            a[:3] = [0, pkg.DEFAULT_Q - 1, pkg.DEFAULT_Q - 1]
            qs.append(pkg.ClientQuery(i % 2, a, b))
        out = pkg.respond_one_packing_batch(crs, db, qs)
        for i in {0, 1 % count, count // 2, count - 1}:
            ao, bo = ocache.respond_one_packing(shards[i % 2], qs[i].a, qs[i].b, galois)
            assert np.array_equal(out[i].a, ao) and np.array_equal(out[i].b, bo), (count, i)
