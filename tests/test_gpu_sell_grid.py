"""The single-body assembled PCG past a cluster's size against the
element-by-element form: a grid of at most one block per SM with all or most
column slots in shared memory, the largest such body and the smallest past it,
in both row groups."""
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, relative_error

pytestmark = pytest.mark.gpu


# 5,202 nodes; 37,856, whose 1,183 slices fill 148 blocks of 8; 38,367, a part more
@pytest.mark.parametrize("cells", [(16, 16, 17), (51, 27, 25), (48, 28, 26)])
@pytest.mark.parametrize("row_group", [2, 4])
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-10), (tb.FP32_MIXED, 1e-5)])
def test_one_block_per_sm(cells, row_group, precision, tol):
    mesh = tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=3)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    out = {}
    for form in ("auto", "elementwise"):
        s = tb.System(mesh, [mat], precision)
        s.set_solver(form)
        s.tune_shape(row_group=row_group)
        s.set_state(tb.rest_state(mesh))
        its = [s.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations for _ in range(2)]
        out[form] = s.get_state().position, its
        s.close()
    assert relative_error(out["auto"][0], out["elementwise"][0], mesh.rest_positions) <= tol
    if precision == tb.FP64:
        assert out["auto"][1] == out["elementwise"][1]
