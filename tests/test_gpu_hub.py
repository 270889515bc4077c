"""Bodies with one node of many neighbours: a box whose inner cells are replaced
by the cone of their boundary to a new node.  The assembled matrix's row of that
node is one long chain, so TL_SOLVER_AUTO takes such single bodies element by
element; the assembled forms still solve them."""
import numpy as np
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, relative_error

pytestmark = pytest.mark.gpu


def coned(cells, k):
    """A box of cells with its inner k^3 replaced by a cone: (mesh, neighbours of the cone's node and itself)."""
    m = tb.box_mesh(cells, voxel=0.1)
    tets = m.tet_nodes.astype(np.int64)
    lo = np.array([(c - k) // 2 for c in cells])
    centre = m.rest_positions[tets].mean(1) / 0.1
    inner = ((centre > lo) & (centre < lo + k)).all(1)
    faces = np.sort(tets[inner][:, [[1, 2, 3], [0, 3, 2], [0, 1, 3], [0, 2, 1]]].reshape(-1, 3), 1)
    faces, times = np.unique(faces, axis=0, return_counts=True)
    faces = faces[times == 1]
    used = np.unique(np.concatenate([tets[~inner].ravel(), faces.ravel()]))
    rank = np.zeros(m.nodes, np.int64)
    rank[used] = np.arange(used.size)
    rest = np.concatenate([m.rest_positions[used], [0.1 * (lo + 0.5 * k)]])
    cone = np.concatenate([np.full((len(faces), 1), used.size), rank[faces]], 1)
    tets = np.concatenate([rank[tets[~inner]], cone])
    edges = np.stack([rest[tets[:, c]] - rest[tets[:, 0]] for c in (1, 2, 3)], 2)
    flip = np.linalg.det(edges) < 0.0
    tets[flip, 1], tets[flip, 2] = tets[flip, 2].copy(), tets[flip, 1].copy()
    edges = np.stack([rest[tets[:, c]] - rest[tets[:, 0]] for c in (1, 2, 3)], 2)
    volume = np.linalg.det(edges) / 6.0
    mass = np.bincount(tets.ravel(), np.repeat(250.0 * volume, 4))
    mesh = tb.PreparedMesh(rest, mass, (rest[:, 1] < 1e-9).astype(np.uint8), tets.astype(np.uint32),
                           np.linalg.inv(edges), volume, np.zeros(len(tets), np.uint32))
    return mesh, np.unique(cone).size


def run(mesh, form, precision):
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    s = tb.System(mesh, [mat], precision)
    s.set_solver(form)
    s.set_state(tb.rest_state(mesh))
    reports = [s.step(tb.Settings(), GRAVITY, DT)[0] for _ in range(2)]
    x = s.get_state().position
    s.close()
    return x, reports[-1]


# cells, cone, its row, whether AUTO goes element by element: four workers share a slice of the small body, one of the
# next; past a cluster's size
@pytest.mark.parametrize("cells,k,row,elementwise", [((9, 9, 9), 4, 99, False), ((9, 9, 9), 5, 153, True),
                                                     ((12, 13, 14), 2, 27, False), ((12, 13, 14), 3, 57, True),
                                                     ((17, 17, 18), 2, 27, False), ((17, 17, 18), 3, 57, True)])
def test_auto_takes_a_hub_element_by_element(cells, k, row, elementwise):
    mesh, found = coned(cells, k)
    assert found == row
    (xa, ra), (xe, re) = run(mesh, "auto", tb.FP64), run(mesh, "elementwise", tb.FP64)
    if elementwise:
        assert np.array_equal(xa, xe) and ra.kernel_launches == re.kernel_launches
    else:
        assert not np.array_equal(xa, xe)
        assert relative_error(xa, xe, mesh.rest_positions) <= 1e-10
        assert ra.cg_iterations == re.cg_iterations


@pytest.mark.parametrize("cells,k", [((9, 9, 9), 7), ((12, 13, 14), 7), ((17, 17, 18), 7)])
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-10), (tb.FP32_MIXED, 1e-5)])
def test_assembled_form_of_a_hub(cells, k, precision, tol):
    """A row of 297 blocks: in a cluster most of them stay in L2."""
    mesh, _ = coned(cells, k)
    (xa, _), (xe, _) = run(mesh, "assembled", precision), run(mesh, "elementwise", precision)
    assert relative_error(xa, xe, mesh.rest_positions) <= tol
