"""State uploads and downloads of the unstructured solver leave the rest of it alone: the checkpoint, which
holds both state buffers, has the same bytes after a download as before it, and an upload changes the present
state's buffer only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(name):
    from hyperflow_gb300 import meshgen
    from test_uns import load
    g = load("tri_hole_3k")
    if name == "one cell":      # no interior edge
        return g["case"], meshgen.hmsh_text(g["verts"][:1], np.full((1, 3), -2, np.int32))
    return g["case"], meshgen.hmsh_text(g["verts"], g["codes"])


@pytest.mark.parametrize("edge", [False, True])
@pytest.mark.parametrize("name", ["one cell", "tri_hole_3k"])
def test_transfers_leave_the_other_buffer(name, edge):
    from hyperflow_gb300 import UnsSolver
    case, text = _mesh(name)
    a, b = UnsSolver(case, mesh_text=text), UnsSolver(case, mesh_text=text)
    for s in (a, b):
        s.set_edge_mode(edge)
    for steps in (4, 3):
        a.run(steps)
        b.run(steps)
        before = b.checkpoint()
        U = b.state()
        assert b.checkpoint() == before == a.checkpoint()
        b.set_state(U)
        assert b.checkpoint() == before
        np.testing.assert_array_equal(b.state(), U)
    a.run(5)
    b.run(5)
    np.testing.assert_array_equal(a.state(), b.state())
    assert a.time() == b.time()
