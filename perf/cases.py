"""The work a user of this framework has it do, as cases with sizes, inputs and one pass each.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  a program's state before the call: database, seats, queries, buffers
    run(state)           one pass through the public entry points, and its outputs
    work(case)           the bytes and operations one pass cannot do without
    exact(case, seed)    outputs in 64-bit arithmetic, where they are computed numbers

Every output is a whole number (residues mod q, response words, status words), exact by
construction: nothing is rounded on the way, so there is no 64-bit value to approach.

A batch goes through the C ABI (include/inspire_gb300.h), as a server holding its own request
buffers calls it; a lone query goes through the Python mirror. All states of a process share one
context, as a server's databases and sessions do.
"""
import ctypes
import importlib

import numpy as np
import torch

pkg = importlib.import_module("inspire-rs_gb300")

N = 2048  # ring of every shipped parameter set
Q = pkg.DEFAULT_Q
SWITCH = {0: 0, 36: pkg.MOD_SWITCH_TARGET_36BIT, 45: pkg.MOD_SWITCH_TARGET_45BIT}


def listed():
    return [
        # The smallest call a server gets: one query on 32-byte records, its key inline.
        {"name": "lone-32B", "kind": "respond", "gamma": 16, "approx": False, "batch": 1, "shards": 64, "switch": 0,
         "inline": True, "device": False, "lanes": 1},
        # An interactive request: one query on 512-byte records under a registered key, answered
        # over the 36-bit modulus.
        {"name": "lone-512B", "kind": "respond", "gamma": 256, "approx": False, "batch": 1, "shards": 128,
         "switch": 36, "inline": False, "device": False, "lanes": 1},
        # A served batch in host buffers, one caller.
        {"name": "batch-64", "kind": "respond", "gamma": 256, "approx": False, "batch": 64, "shards": 128,
         "switch": 36, "inline": False, "device": False, "lanes": 1},
        # The same batch device-resident, batch after batch over four lanes: a saturated server.
        {"name": "stream-64", "kind": "respond", "gamma": 256, "approx": False, "batch": 64, "shards": 256,
         "switch": 36, "inline": False, "device": True, "lanes": 4},
        # A large odd batch in one launch, approximate gadget: offline bulk retrieval.
        {"name": "bulk-509", "kind": "respond", "gamma": 256, "approx": True, "batch": 509, "shards": 256,
         "switch": 36, "inline": False, "device": True, "lanes": 1},
        # 2048-byte records, the widest served: a long recursion over a batch smaller than the GPU.
        {"name": "wide-33", "kind": "respond", "gamma": 1024, "approx": False, "batch": 33, "shards": 48,
         "switch": 45, "inline": False, "device": False, "lanes": 1},
        # Queries of three record widths and both gadgets in one launch.
        {"name": "mixed-128", "kind": "mixed", "batch": 128, "shards": 48},
        # Requests arriving one by one at a saturated serving loop.
        {"name": "serving-1024", "kind": "serving", "gamma": 256, "requests": 1024, "window": 512, "shards": 128},
        # The two-prime variant: 256-byte cells, a served batch over eight keys.
        {"name": "special-256", "kind": "special", "batch": 256, "tables": 128},
        # The automorphism-tree variant (OnePacking).
        {"name": "tree-64", "kind": "tree", "gamma": 256, "batch": 64, "shards": 64, "switch": 36},
        # The unpacked variant (NoPacking): one ciphertext per column, 8.4 MB a response.
        {"name": "unpacked-16", "kind": "unpacked", "gamma": 256, "batch": 16, "shards": 64},
        # A database update: records encoded into their shards, the packing stores rebuilt, and the
        # updated shards queried once each.
        {"name": "update-64", "kind": "update", "gamma": 256, "shards": 64},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["respond"] * 6 + ["mixed", "serving", "special", "special", "tree", "unpacked", "update"])
    gamma = rng.choice([16, 64, 128, 256, 512, 1024])
    if kind == "respond":
        batch = _log_int(rng, 1, min(509, 509 * 256 // gamma))
        return {"kind": kind, "gamma": gamma, "approx": rng.random() < 0.5, "batch": batch,
                "shards": rng.randint(8, max(8, 128 * 256 // max(gamma, 128))), "switch": rng.choice([0, 36, 45]),
                "inline": rng.random() < 0.3 and batch < 16, "device": batch > 1 and rng.random() < 0.5,
                "lanes": rng.choice([1, 1, 2, 4])}
    if kind == "mixed":
        return {"kind": kind, "batch": _log_int(rng, 2, 128), "shards": rng.randint(8, 48)}
    if kind == "serving":
        return {"kind": kind, "gamma": rng.choice([16, 64, 128, 256]), "requests": _log_int(rng, 64, 1024),
                "window": _log_int(rng, 8, 512), "shards": rng.randint(32, 128)}
    if kind == "special":
        return {"kind": kind, "batch": _log_int(rng, 1, 256), "tables": rng.randint(8, 128)}
    if kind == "tree":
        gamma = rng.choice([16, 64, 128, 256])
        return {"kind": kind, "gamma": gamma, "batch": _log_int(rng, 1, 64), "shards": rng.randint(8, 64),
                "switch": rng.choice([0, 36, 45])}
    if kind == "unpacked":
        gamma = rng.choice([16, 64, 128, 256])
        return {"kind": kind, "gamma": gamma, "batch": _log_int(rng, 1, 16 * 256 // gamma if gamma > 16 else 64),
                "shards": rng.randint(8, 64)}
    gamma = rng.choice([16, 64, 128, 256, 512])
    return {"kind": kind, "gamma": gamma, "shards": _log_int(rng, 1, min(64, 64 * 256 // gamma))}


# ------------------------------------------------------------------------------------------
def _ptr(a):
    if isinstance(a, torch.Tensor):
        return ctypes.c_void_p(a.data_ptr())
    return ctypes.c_void_p(a.ctypes.data)


def _words(rng, shape):
    return rng.integers(0, Q, size=shape, dtype=np.uint64)


def _signed(a):
    """The same words as int64 (every one is below 2^63)."""
    return a.view(np.int64)


class State:
    """What a program holds between calls; the device objects go with it."""

    def __init__(self, case):
        self.case, self.kind = case, case["kind"]
        self.ctx = pkg.Context.default(0)
        self.lib = self.ctx._lib
        self.owned = []  # (destroy call, handle), released last first
        self.loop = None

    def own(self, name, handle):
        self.owned.append((getattr(self.lib, name), handle))

    def __del__(self):
        if self.loop is not None:
            self.loop.close()
        for destroy, handle in reversed(self.owned):
            destroy(self.ctx.h, handle)


def _database(st, rng, gamma, shards, approx=False, galois=None, caches=None):
    """A database of 2*gamma-byte uniform records, encoded on the GPU with a store on every shard,
    and its cache (or one cache per gadget in `caches`)."""
    params = pkg.InspireParams(approximate_packing_gadget=approx)
    crs = pkg.ServerCrs(params, rng.bytes(32), gamma, galois_keys=galois)
    cache = pkg.ServerInspiringCache.new(crs, ctx=st.ctx)
    st.own("ig_crs_destroy", cache.h)
    db = pkg.EncodedDatabase(cache, shards)
    st.own("ig_db_destroy", db.h)
    records = _records(rng, gamma, shards)
    db.encode_records(None, 2 * gamma, device_ptr=records.data_ptr(), nbytes=records.numel())
    return crs, cache, db


def _records(rng, gamma, shards):
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    r = torch.randint(0, 256, (shards * N * 2 * gamma,), dtype=torch.uint8, device="cuda", generator=gen)
    torch.cuda.synchronize()  # the library encodes on its own stream
    return r


def _keys(rng, params, gamma):
    return pkg.ClientPackingKeys(_words(rng, (params.packing_key_rows(), N)), gamma)


def _queries(st, rng, batch, shards):
    st.ids = rng.integers(0, shards, size=batch, dtype=np.uint32)
    st.seeds = np.frombuffer(rng.bytes(32 * batch), dtype=np.uint8).copy()
    st.bs = _words(rng, (batch, N))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = State(case)
    st.ctx.set_lanes(case.get("lanes", 1))
    kind = st.kind
    if kind == "special":
        return _prepare_special(st, rng)
    if kind == "mixed":
        return _prepare_mixed(st, rng)
    gamma, shards = case["gamma"], case["shards"]
    if kind == "tree":
        st.crs, st.cache, st.db = _database(st, rng, gamma, shards, galois=_words(rng, (11, 3, 2, N)))
    else:
        st.crs, st.cache, st.db = _database(st, rng, gamma, shards, case.get("approx", False))
    batch = case.get("batch") or case.get("requests") or shards
    _queries(st, rng, batch, shards)
    if kind == "unpacked":
        st.out = torch.empty((batch, gamma + 1, 2, N), dtype=torch.int64, pin_memory=True)
        return st
    if kind == "tree":
        st.a, st.b = np.zeros((batch, N), np.uint64), np.zeros((batch, N), np.uint64)
        return st
    keys = _keys(rng, st.crs.params, gamma)
    st.store = pkg.ServerSessionStore(st.ctx)
    st.own("ig_session_store_destroy", st.store.h)
    st.handle = st.store.register_server_side(keys, st.cache)
    if kind == "update":
        st.ids = np.arange(shards, dtype=np.uint32)
        st.records = _records(rng, gamma, shards)
        st.entry = 2 * gamma
    st.db.precompute_packing_all()
    if kind == "serving":
        st.handles = np.full(batch, int(st.handle), dtype=np.uint64)
        st.seeds = st.seeds.reshape(batch, 32)
        st.loop = pkg.ServingLoop(st.ctx, slots=4, max_batch=64)
        return st
    if kind == "update" or case["device"]:
        st.d_seeds = torch.from_numpy(st.seeds).cuda()
        st.d_bs = torch.from_numpy(_signed(st.bs)).cuda()
        st.d_a = torch.zeros((batch, N), dtype=torch.int64, device="cuda")
        st.d_b = torch.zeros((batch, N), dtype=torch.int64, device="cuda")
        st.d_status = torch.zeros(batch, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()  # the library reads them on its own stream
    elif batch == 1:
        st.query = pkg.SeededClientQuery(int(st.ids[0]), st.seeds.tobytes(), st.bs[0],
                                         inspiring_packing_keys=keys if case["inline"] else None,
                                         session_handle=None if case["inline"] else st.handle)
    else:
        st.y = keys.y_body
        st.a, st.b = np.zeros((batch, N), np.uint64), np.zeros((batch, N), np.uint64)
    return st


def _prepare_mixed(st, rng):
    """Three record widths, each database serving an exact-gadget and an approximate-gadget seat."""
    batch, shards = st.case["batch"], st.case["shards"]
    sets = []
    st.store = pkg.ServerSessionStore(st.ctx)
    for gamma, count in ((16, 4 * shards), (256, 2 * shards), (1024, max(1, shards // 2))):
        crs, cache, db = _database(st, rng, gamma, count)
        db.precompute_packing_all()
        crs_a = pkg.ServerCrs(pkg.InspireParams.d2048_approximate_gadget(), rng.bytes(32), gamma)
        cache_a = pkg.ServerInspiringCache.new(crs_a, ctx=st.ctx)
        st.own("ig_crs_destroy", cache_a.h)
        handles = [int(st.store.register_server_side(_keys(rng, c.crs.params, gamma), c)) for c in (cache, cache_a)]
        sets.append((db, count, handles))
    st.own("ig_session_store_destroy", st.store.h)
    st.sets = sets
    which = rng.integers(0, 3, size=batch)
    gadget = rng.integers(0, 2, size=batch)
    _queries(st, rng, batch, 1)
    st.dbs = np.array([sets[w][0].h for w in which], dtype=np.uint64)
    st.stores = np.full(batch, st.store.h, dtype=np.uint64)
    st.handles = np.array([sets[w][2][g] for w, g in zip(which, gadget)], dtype=np.uint64)
    st.ids = np.array([rng.integers(0, sets[w][1]) for w in which], dtype=np.uint32)
    st.targets = np.full(batch, SWITCH[36], dtype=np.uint64)
    st.a, st.b = np.zeros((batch, N), np.uint64), np.zeros((batch, N), np.uint64)
    return st


def _prepare_special(st, rng):
    sm = pkg.special_modulus
    p = sm.Params.ring2048_cell256()
    st.server = sm.Server(p, st.ctx)
    st.own("ig_sm_server_destroy", st.server.h)
    batch = st.case["batch"]
    seats = []
    for _ in range(8):
        key = sm.PackingKey(rng.bytes(32), rng.integers(0, p.q, size=N, dtype=np.uint32),
                            rng.integers(0, p.special_prime, size=N, dtype=np.uint32))
        seats.append(st.server.seat(key))
        st.own("ig_sm_seat_destroy", seats[-1])
    tables = []
    for _ in range(st.case["tables"]):
        cells = rng.integers(0, 256, size=(N, p.cell_bytes), dtype=np.uint8)
        cells[:, p.record_bytes:] = 0
        tables.append(st.server.table(cells.tobytes()))
        st.own("ig_sm_table_destroy", tables[-1])
    st.tables = np.array(tables, dtype=np.uint64)[rng.integers(0, len(tables), size=batch)]
    st.seats = np.array(seats, dtype=np.uint64)[rng.integers(0, len(seats), size=batch)]
    st.seeds = np.frombuffer(rng.bytes(32 * batch), dtype=np.uint8).copy()
    st.bodies = rng.integers(0, p.q, size=(batch, N), dtype=np.uint32)
    st.mask = np.zeros((batch, N), np.uint32)
    st.body = np.zeros((batch, p.body_coefficients()), np.uint32)
    return st


def run(st):
    case, kind, ctx, lib = st.case, st.kind, st.ctx, st.lib
    if kind == "respond" and case["batch"] == 1 and not case["device"]:
        r = pkg.respond_seeded_inspiring(st.crs, st.db, st.query, None if case["inline"] else st.store,
                                         SWITCH[case["switch"]])
        return {"a": _signed(r.a), "b": _signed(r.b)}
    if kind == "respond" and not case["device"]:
        key = (0, 0, _ptr(st.y), st.y.shape[0], case["gamma"]) if case["inline"] else (st.store.h, int(st.handle),
                                                                                       None, 0, 0)
        ctx.check(lib.ig_respond_seeded_batch(ctx.h, st.db.h, *key, case["batch"], _ptr(st.ids), _ptr(st.seeds),
                                              _ptr(st.bs), SWITCH[case["switch"]], _ptr(st.a), _ptr(st.b)))
        return {"a": _signed(st.a), "b": _signed(st.b)}
    if kind in ("respond", "update"):
        if kind == "update":
            st.db.encode_records(None, st.entry, device_ptr=st.records.data_ptr(), nbytes=st.records.numel())
            st.db.precompute_packing_all()
        ctx.check(lib.ig_respond_seeded_batch_device(ctx.h, st.db.h, st.store.h, int(st.handle), len(st.ids),
                                                     _ptr(st.ids), _ptr(st.d_seeds), _ptr(st.d_bs),
                                                     SWITCH[case.get("switch", 36)], _ptr(st.d_a), _ptr(st.d_b),
                                                     _ptr(st.d_status)))
        return {"a": st.d_a, "b": st.d_b, "status": st.d_status}
    if kind == "mixed":
        ctx.check(lib.ig_respond_mixed_batch(ctx.h, case["batch"], _ptr(st.dbs), _ptr(st.stores), _ptr(st.handles),
                                             _ptr(st.ids), _ptr(st.seeds), _ptr(st.bs), _ptr(st.targets), _ptr(st.a),
                                             _ptr(st.b)))
        return {"a": _signed(st.a), "b": _signed(st.b)}
    if kind == "serving":
        a, b, _, _ = st.loop.replay(st.db, st.store, st.ids, st.handles, st.seeds, st.bs, SWITCH[36],
                                    window=case["window"])
        return {"a": _signed(a), "b": _signed(b)}
    if kind == "special":
        ctx.check(lib.ig_sm_respond_batch(ctx.h, st.server.h, case["batch"], _ptr(st.tables), _ptr(st.seats),
                                          _ptr(st.seeds), _ptr(st.bodies), _ptr(st.mask), _ptr(st.body)))
        return {"mask": st.mask.view(np.int32), "body": st.body.view(np.int32)}
    if kind == "tree":
        ctx.check(lib.ig_respond_one_packing_batch(ctx.h, st.db.h, case["batch"], _ptr(st.ids), _ptr(st.seeds), None,
                                                   _ptr(st.bs), SWITCH[case["switch"]], _ptr(st.a), _ptr(st.b)))
        return {"a": _signed(st.a), "b": _signed(st.b)}
    ctx.check(lib.ig_respond_nopacking_batch(ctx.h, st.db.h, case["batch"], _ptr(st.ids), _ptr(st.seeds), None,
                                             _ptr(st.bs), _ptr(st.out)))
    return {"ciphertexts": st.out}


# ------------------------------------------------------------------------------------------
# Operations are counted as one multiplication and one addition per modular product: a ring
# transform takes n/2 log2 n of them.
_TRANSFORM = N // 2 * 11


def _recursion(gamma):
    """Products of one query: per link one inverse and two forward transforms and the pointwise
    products with the key rows and the store."""
    return (gamma - 1) * (3 * _TRANSFORM + 7 * N)


def _served_bytes(gamma, batch, shards):
    """16-bit columns and the 64-bit store of each shard read once; seed, b, a and b per query."""
    return min(batch, shards) * gamma * N * 10 + batch * (3 * N * 8 + 32)


def work(case):
    kind = case["kind"]
    if kind == "respond":
        products = case["batch"] * _recursion(case["gamma"])
        size = _served_bytes(case["gamma"], case["batch"], case["shards"])
    elif kind == "serving":
        products = case["requests"] * _recursion(case["gamma"])
        size = _served_bytes(case["gamma"], case["requests"], case["shards"])
    elif kind == "mixed":
        third = case["batch"] / 3
        products = sum(third * _recursion(g) for g in (16, 256, 1024))
        size = sum(_served_bytes(g, third, s) for g, s in ((16, 4 * case["shards"]), (256, 2 * case["shards"]),
                                                           (1024, max(1, case["shards"] // 2))))
    elif kind == "special":  # 32-bit words, four transforms a link, 512 columns
        products = case["batch"] * 511 * (4 * _TRANSFORM + 6 * N)
        size = min(case["batch"], case["tables"]) * 512 * N * 5 + case["batch"] * (3 * N * 4 + 32)
    elif kind == "tree":  # per column a transform and four key switches (gamma of 2048 leaves)
        nodes = sum(min(case["gamma"], N >> k) for k in range(1, 12))
        products = case["batch"] * (case["gamma"] * _TRANSFORM + nodes * (3 * _TRANSFORM + 8 * N))
        size = min(case["batch"], case["shards"]) * case["gamma"] * N * 2 + case["batch"] * (3 * N * 8 + 32)
    elif kind == "unpacked":
        products = case["batch"] * case["gamma"] * (3 * _TRANSFORM + 2 * N)
        size = (min(case["batch"], case["shards"]) * case["gamma"] * N * 2
                + case["batch"] * ((case["gamma"] + 1) * 2 * N * 8 + N * 8 + 32))
    else:  # update: column transforms, the per-slot fold, then one query a shard
        lg = case["gamma"].bit_length() - 1
        fold = case["gamma"] * (_TRANSFORM + N * (lg / 2 + 2))
        products = case["shards"] * (fold + _recursion(case["gamma"]))
        size = (case["shards"] * case["gamma"] * N * (2 + 8 + 2 + 8)
                + _served_bytes(case["gamma"], case["shards"], case["shards"]))
    return {"bytes": size, "flops": 2 * products}


def exact(case, seed):
    """None: outputs are whole numbers, equal or not; 64-bit arithmetic is what computes them."""
    return None
