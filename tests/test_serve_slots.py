"""What a service reserves for a slot: a row-walk plan only where the engine
builds one, so that no request waits or is refused for memory nobody takes."""
import pytest

from conftest import ensure_library


@pytest.mark.parametrize("kind,precision,n,plan", [
    ("p1", "fp32", 8, False), ("p1", "fp32", 25, False), ("p1", "fp32", 26, True), ("p1", "fp64", 26, True),
    ("p2", "fp64", 8, False), ("p2", "fp64", 22, False), ("p2", "fp64", 23, True), ("p2", "fp32", 40, False),
    ("vp2", "fp32", 31, False), ("vp2", "fp32", 32, True), ("vp2", "fp64", 40, False)])
def test_plan_bytes_where_there_is_a_plan(kind, precision, n, plan):
    ensure_library()
    from cudolfinx import serve

    s = serve.problem_sizes(kind, n)
    # values, slot map, b, x, BC data, six solver vectors, FP32 values (vector P2: their block columns), coefficients
    base = (8 * s["nnz"] + s["cells"] * s["k"] ** 2 + 16 * s["rows"] + 9 * s["rows"] + 48 * s["rows"] + 4 * s["nnz"]
            + (s["nnz"] // 9 * 4 + s["rows"] // 3 * 4 + 8 * s["cells"] if kind == "vp2" else 0) + 8 * s["cells"])
    more = serve.slot_bytes(kind, n, precision) - base
    assert more >= 60 * s["cells"] if plan else more == 0
    if precision == "fp32":
        assert serve.slot_bytes(kind, n) == base + more
