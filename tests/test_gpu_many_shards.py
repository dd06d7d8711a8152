"""Store builds and encodes of more shards than a grid's y and z take, at the narrowest ring and width: the first and last
shards of each launch against a database of those shards alone."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, ENTRY, SHARDS = 256, 2, 65536 + 3


def test_build_of_65539_shards():
    torch = pytest.importorskip("torch")
    pkg = load_package()
    rng = np.random.default_rng(65539)
    ctx = pkg.Context(0)
    cache = pkg.ServerInspiringCache.new(pkg.ServerCrs(pkg.InspireParams(ring_dim=N), rng.bytes(32), 1), ctx=ctx)
    raw = rng.integers(0, 256, size=(SHARDS, N * ENTRY), dtype=np.uint8)
    dev = torch.from_numpy(raw).cuda()
    torch.cuda.synchronize()
    db = pkg.EncodedDatabase(cache, SHARDS)
    db.encode_records(None, ENTRY, device_ptr=dev.data_ptr(), nbytes=raw.size)
    db.precompute_packing_all()
    pick = [0, 1, 16383, 16384, 32767, 32768, 49151, 49152, 65534, 65535, 65536, SHARDS - 1]
    few = pkg.EncodedDatabase.from_records(cache, raw[pick].tobytes(), ENTRY, len(pick))
    few.precompute_packing_all()
    for k, s in enumerate(pick):
        assert np.array_equal(db.store_sums(s), few.store_sums(k)), s
    ctx.close()
