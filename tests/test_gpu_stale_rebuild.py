"""A batch queued on a lane while a stale shard's store is rebuilt: it is refused, or it answers from the rebuilt store,
whenever it comes to run; it never answers from a store that is still being written."""
import ctypes

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

N, GAMMA, SHARDS, LONG = 2048, 32, 48, 608
STALE = SHARDS - 1  # built last


@pytest.mark.parametrize("ahead", [1, 2, 3])  # batches that keep the GPU busy while the probe is queued
def test_queued_batch_and_rebuild(ahead):
    torch = pytest.importorskip("torch")
    pkg = load_package()
    rng = np.random.default_rng(ahead)
    ctx = pkg.Context(0)
    crs = pkg.ServerCrs(pkg.InspireParams(), rng.bytes(32), GAMMA)
    cache = pkg.ServerInspiringCache.new(crs, ctx=ctx)
    entry = 2 * GAMMA
    records = torch.from_numpy(rng.integers(0, 256, size=SHARDS * N * entry, dtype=np.uint8)).cuda()
    db = pkg.EncodedDatabase(cache, SHARDS)
    store = pkg.ServerSessionStore.new(ctx)
    keys = pkg.ClientPackingKeys(rng.integers(0, pkg.DEFAULT_Q, size=(3, N), dtype=np.uint64), GAMMA)
    handle = store.register_server_side(keys, cache)
    seeds = torch.from_numpy(np.frombuffer(rng.bytes(32 * LONG), dtype=np.uint8).copy()).cuda()
    bs = torch.from_numpy(rng.integers(0, pkg.DEFAULT_Q, size=(LONG, N), dtype=np.uint64).view(np.int64)).cuda()

    class Out:
        def __init__(self, count):
            self.a, self.b = (torch.zeros((count, N), dtype=torch.int64, device="cuda") for _ in range(2))
            self.status = torch.full((count,), -1, dtype=torch.int32, device="cuda")

    def launch(ids, out):
        ids = np.asarray(ids, dtype=np.uint32)
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in (seeds, bs, out.a, out.b, out.status)]
        ctx.check(ctx._lib.ig_respond_seeded_batch_device(ctx.h, db.h, store.h, int(handle), len(ids),
                                                          ctypes.c_void_p(ids.ctypes.data), ptr[0], ptr[1], 0, *ptr[2:]))

    def encode():
        torch.cuda.synchronize()
        db.encode_records(None, entry, device_ptr=records.data_ptr(), nbytes=records.numel())

    encode()
    db.precompute_packing_all()
    ctx.set_lanes(2)
    ctx.set_launch_shape(1)
    busy, probe, want = [Out(LONG) for _ in range(ahead)], Out(1), Out(1)
    torch.cuda.synchronize()
    for _ in range(8):
        records[STALE * N * entry:] ^= 0x5A
        encode()  # the last shard is stale now
        for o in busy:
            launch(np.arange(LONG) % STALE, o)
        probe.status.fill_(-1)
        torch.cuda.synchronize()
        for o in busy:
            launch(np.arange(LONG) % STALE, o)
        launch([STALE], probe)
        db.precompute_packing_all()
        ctx.join()
        torch.cuda.synchronize()
        launch([STALE], want)
        ctx.join()
        torch.cuda.synchronize()
        assert int(want.status[0]) == 0
        status = int(probe.status[0])
        assert status in (0, 1)  # 1: refused
        if status == 0:
            assert torch.equal(probe.a, want.a) and torch.equal(probe.b, want.b)
    ctx.set_launch_shape(0)
    ctx.set_lanes(1)
    ctx.close()
