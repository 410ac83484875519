"""Sectors whose rank tables fit take their keys from those tables
(k_tab_emit); LGT_BASIS_TABLES=0 forces the ordered compaction of all
candidates.  Both give the same basis bit for bit and the same ranks, for
wide and narrow lattices, link truncations and sectors (an empty one among
them); lattices without tables still build."""
import numpy as np
import pytest

import lgt_gb300 as lgt

pytestmark = pytest.mark.gpu


def _charges(nx, ny, kind):
    if kind == "stag":
        return lgt.staggered_charges(nx, ny)
    if kind == "string":
        return lgt.string_charges(nx, ny)
    q = np.zeros((nx, ny), np.int32)
    if kind == "far":  # charges too far apart for the truncated links
        q[0, 0], q[nx - 1, ny - 1] = 5, -5
    return q


@pytest.mark.parametrize("nx,ny,dg,kind", [
    (2, 2, 1, "stag"), (4, 2, 1, "stag"), (2, 4, 1, "zero"), (3, 3, 2, "stag"), (2, 6, 1, "stag"),
    (5, 2, 1, "stag"), (4, 3, 1, "stag"), (3, 4, 1, "string"), (3, 4, 1, "stag"),
    (2, 4, 3, "stag"), (6, 2, 1, "stag"), (3, 3, 1, "far"), (1, 5, 1, "stag"), (5, 1, 1, "stag"),
    (5, 3, 1, "stag"), (3, 2, 7, "stag"),
])
def test_tables_match_compaction(monkeypatch, nx, ny, dg, kind):
    monkeypatch.setenv("LGT_BASIS_FUSED", "0")
    q = _charges(nx, ny, kind)
    got = {}
    for tables in ("0", "1"):
        monkeypatch.setenv("LGT_BASIS_TABLES", tables)
        b, _ = lgt.build_basis(nx, ny, dg, q)
        keys = b.order_keys()
        assert np.all(keys[1:] > keys[:-1])
        absent = np.concatenate((keys[:200] + np.uint64(1), keys[:200] ^ np.uint64(1)))
        got[tables] = (b.dim, keys, b.rank(keys), b.rank(absent),
                       b.ref_keys() if dg == 1 else None)
        b.close()
    for a, r in zip(got["1"], got["0"]):
        np.testing.assert_array_equal(a, r)
    np.testing.assert_array_equal(got["1"][2], np.arange(got["1"][0]))
