"""What the variant "row-walk" is refused for, and what it leaves behind."""
import numpy as np
import pytest

import ffcx_bodies as fb
from conftest import ensure_library

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["ffcx", "facet", "interior facet", "block", "mass"])
def test_refused_where_there_is_no_walk(what):
    """A form without a row walk says so, as for the other variants it does not
    have, instead of assembling with the scatter."""
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    mesh = fem.create_unit_cube(2)
    V, Q = fem.functionspace(mesh, ("P", 1)), fem.functionspace(mesh, ("DG", 0))
    asm = cx.CUDAAssembler()
    mat = None
    if what == "ffcx":
        B = fb.stiffness(1, "dg0")
        k = fem.Function(Q, np.ones(mesh.num_cells))
        a = cx.form(fem.FFCxForm([fem.FFCxIntegral(B["integral_type"], B["name"], B["body"])], [V, V], [k]))
    elif what == "facet":
        a = cx.form(fem.facet_mass(V, 1.0))
    elif what == "interior facet":
        a = cx.form(fem.jump_penalty(fem.functionspace(mesh, ("DG", 1)), 1.0))
    elif what == "block":
        block = cx.form([[fem.stiffness(V, 1.0)]])
        mat, a = asm.create_matrix_block(block), block.forms[0][0]
    else:
        a = cx.form(fem.mass(V, 1.0))
    with pytest.raises(RuntimeError, match="row walk|atomic scatter only"):
        asm.assemble_matrix(a, mat, variant="row-walk")


@pytest.mark.parametrize("kind", ["p1", "p2"])
def test_a_call_with_the_variant_leaves_the_default_as_it_was(kind):
    """Below the sizes where the walk is the default, "auto" stays the scatter
    after a call that asked for the walk.  The two evaluate the element entries
    by different formulas, so on a jittered mesh some entries differ in their
    last bits; the walk itself is bitwise reproducible."""
    ensure_library()
    import cudolfinx as cx
    from cudolfinx import fem

    V = fem.functionspace(fem.create_unit_cube(4, jitter=0.2, seed=3), ("P", int(kind[1])))
    a = cx.form(fem.stiffness(V, 0.7))
    asm = cx.CUDAAssembler()
    A = asm.create_matrix(a)
    values = []
    for variant in ("row-walk", "auto", "row-walk"):
        asm.assemble_matrix(a, A, variant=variant)
        values.append(A.values.cpu().numpy())
    assert np.array_equal(values[0], values[2]) and not np.array_equal(values[0], values[1])
