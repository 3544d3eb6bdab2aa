"""Constant tables of the generated element code stand only in the units that use
them: a table is in the constant bank of every kernel of a unit, and each launch
pays for the bank."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-dolfinx_b200", "csrc")


def _visible(text, defined):
    """Lines of the header that a unit with these macros compiles (it has only #ifdef / #endif)."""
    out, hidden = [], 0
    for line in text.splitlines():
        if line.startswith("#ifdef"):
            hidden += 1 if hidden or line.split()[1] not in defined else 0
            if not hidden:
                out.append("")
            continue
        if line.startswith("#endif") and hidden:
            hidden -= 1
            continue
        if not hidden:
            out.append(line)
    return out


def test_units_hold_the_tables_they_use():
    header = open(os.path.join(CSRC, "fe_element_code.cuh")).read()
    guards = set(re.findall(r"^#ifdef (\w+)", header, flags=re.M))
    assert {"FE_P3_ROW_TABLES", "FE_FACET_TABLES"} <= guards
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        unit = open(f).read()
        if '"fe_element_code.cuh"' not in unit:
            continue
        visible = "\n".join(_visible(header, set(re.findall(r"^#define (FE_\w+_TABLES)", unit, flags=re.M))))
        for table in re.findall(r"^(?:static )?__constant__ \w+ (kP3Row\w|kFacet\w+)\[", visible, flags=re.M):
            users = [m for m in re.findall(r"__device__ __forceinline__ void (\w+)\([^{]*\{(?:[^}]*\b%s\b)" % table, visible)]
            assert table in unit or any(re.search(r"\b%s\b" % u, unit) for u in users), (os.path.basename(f), table)
