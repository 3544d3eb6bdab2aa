"""Tables of FFCx bodies that move to constant memory: a body compiles, or is
refused, as it does with its tables where they stand."""
import ctypes

import pytest

from conftest import ensure_library
from test_ffcx_host import _nvrtc_compile

USE = "for (int i = 0; i < 2; ++i) A[i] += T[i];\n"
T = "static const double T[2] = {1.0, -2.5e-3};\n"


def _source(body, rank=2, k=(10, 10)):
    ensure_library()
    from cudolfinx import _lib

    n = ctypes.c_int64()
    args = (0, rank, k[0], 1, k[1], 1, 0, None, b"tabulate_x", body.encode())
    _lib.check(_lib.lib.fe_ffcx_source(*args, None, 0, ctypes.byref(n)))
    buf = ctypes.create_string_buffer(n.value + 1)
    _lib.check(_lib.lib.fe_ffcx_source(*args, buf, n.value + 1, ctypes.byref(n)))
    return buf.value.decode()


@pytest.mark.parametrize("body,moves", [
    (T + USE, True),
    ("alignas(32) " + T + USE, True),
    # a name that is also a function of the math library, or the kernel's own
    (T.replace("T[", "y0[") + USE.replace("T[", "y0["), True),
    (T.replace("T[", "FfcxArgs[") + USE.replace("T[", "FfcxArgs["), True),
    # the table of one of two branches
    ("#define FINE 1\n#if FINE\n" + T + "#else\nstatic const double T[2] = {3.0, 4.0};\n#endif\n" + USE, False),
    ("#if 0\n" + T + "#endif\nconst double T[2] = {0.0, 1.0};\n" + USE, False),
    # a comment before the table that ends like an alignment
    ("int k = 0; // alignas(8)\n" + T + "k += 1;\n" + USE, True),
    ("// a continued line \\\n" + T + "const double T[2] = {0.0, 1.0};\n" + USE, False),
    # the same name again in an inner scope
    (T + "{ const double T[2] = {5.0, 6.0}; A[0] += T[0]; }\n" + USE, True),
    # declarations that only end like a table's
    ("__device__ " + T + USE, False),
    ("if (c[0] > 0.0) " + T + "const double T[2] = {0.0, 1.0};\n" + USE, False),
])
def test_compiles_as_written(body, moves):
    src = _source(body)
    assert ("__constant__ double" in src) == moves
    as_it_stands = _nvrtc_compile("#define restrict __restrict__\ntypedef unsigned char uint8_t;\n__device__ void f(double* A, "
                                  "const double* w, const double* c, const double* coordinate_dofs, const int* "
                                  "entity_local_index, const uint8_t* quadrature_permutation)\n{\n" + body + "}\n")[0]
    rc, log = _nvrtc_compile(src)
    assert (rc == 0) == (as_it_stands == 0), log


@pytest.mark.parametrize("body", [
    T + T + USE,                                                     # the same name twice
    T.replace("T[", "A[") + USE.replace("T[", "A["),                 # a parameter's name
    T + "T[0] = 2.0;\n" + USE,                                       # written to
    "const double y = T[0];\n" + T + USE,                            # used before it is declared
    "{\n" + USE + "}\n" + T,                                         # the same, in a block
])
def test_refused_as_written(body):
    rc, _ = _nvrtc_compile(_source(body))
    assert rc != 0
