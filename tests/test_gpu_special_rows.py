"""The special_modulus body fold over tables that do not fill their ring: the rows go to chunks of a fourth, read eight
side by side, so the sizes around those edges are the ones that can go wrong. Exact against the oracle."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 5, 31, 33, 2041, 2047])
def test_partial_tables(oracle, rows):
    sm = load_package().special_modulus
    server, oserver = sm.Server(sm.Params()), oracle.SmServer()
    rng = np.random.default_rng(rows)
    cells = np.zeros((rows, 256), dtype=np.uint8)
    cells[:, :246] = rng.integers(0, 256, (rows, 246), dtype=np.uint8)
    cells[0, :246] = 0x88  # the lowest nibble value throughout
    table, otable = server.table(cells.tobytes()), oserver.table(cells.tobytes())
    client = oracle.SmClient(bytes([9] * 32))
    seat, oseat = server.seat(sm.PackingKey(*client.key())), oserver.seat(client.key())
    for row in {0, rows - 1}:
        seed, body = client.query(row)
        r = server.respond_batch([table], [seat], [sm.Query(seed, body)])[0]
        mask, obody = oserver.respond(otable, oseat, seed, body)
        assert (r.mask == mask).all() and (r.body == obody).all(), row
        assert client.decode(r.mask, r.body) == cells[row, :246].tobytes()
