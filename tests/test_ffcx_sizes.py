"""Which forms given as FFCx bodies take the 32-entity tile and constant tables:
those whose element tensor is large enough for them to pay."""
import pytest

from test_ffcx_tables import _source

TABLE = "static const double T[16] = {" + ", ".join("%d.5" % q for q in range(16)) + "};\nA[0] += T[3];\n"


@pytest.mark.parametrize("rank,k,tile,tables", [(2, (4, 4), False, False), (2, (10, 4), True, True), (2, (4, 10), True, True), (2, (10, 10), True, True),
                                                (2, (12, 12), True, True), (2, (20, 20), False, True), (2, (3, 13), False, False),
                                                (1, (10, 1), False, False), (1, (60, 1), False, False), (0, (1, 1), False, False)])
def test_by_size(rank, k, tile, tables):
    src = _source(TABLE, rank, k)
    assert ("#define WARP_TILE 1" in src) == tile and ("__constant__" in src) == tables
