"""The batched assembled PCG whose bodies are iterated by groups of blocks
(kPcgSell over a queue of items) against the two-phase order: bodies over many
blocks each, more items than resident blocks, bodies of exactly one block's
rows and one past it, in both row groups.  The bars are those of the batch's
other orders: the same iterates in exact arithmetic."""
import numpy as np
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, relative_error

pytestmark = pytest.mark.gpu

# three bodies share the grid; one-block bodies of 256 and 288 rows; 700 bodies, more than a grid of two blocks per SM
BATCHES = {"spread": [(9, 7, 8), (12, 3, 5), (4, 4, 4)], "edge": [(7, 7, 3), (8, 7, 3), (1, 1, 1), (7, 3, 7)],
           "queue": [(2, 3, 2), (1, 1, 2), (3, 2, 4), (2, 2, 2)] * 175}


@pytest.mark.parametrize("name", sorted(BATCHES))
@pytest.mark.parametrize("row_group", [2, 4])
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-10), (tb.FP32_MIXED, 1e-5)])
def test_queue_order_matches_the_two_phase_order(name, row_group, precision, tol):
    meshes = [tb.box_mesh(c, voxel=0.1, jitter=0.01, seed=i % 7) for i, c in enumerate(BATCHES[name])]
    mats = [[tb.PhysicalMaterial(density=1000.0, youngs_modulus=10.0 ** (5 + i % 3), poissons_ratio=0.3)]
            for i in range(len(meshes))]
    out = {}
    for form in ("auto", "assembled-two-phase"):
        s = tb.System(meshes, mats, precision)
        s.set_solver(form)
        s.tune_shape(row_group=row_group)
        for i, m in enumerate(meshes):
            s.set_state(tb.rest_state(m), i)
        its = [[r.cg_iterations for r in s.step(tb.Settings(), GRAVITY, DT)] for _ in range(3)]
        out[form] = [s.get_state(i).position for i in range(len(meshes))], its
        s.close()
    for i, m in enumerate(meshes):
        assert relative_error(out["auto"][0][i], out["assembled-two-phase"][0][i], m.rest_positions) <= tol, i
    if precision == tb.FP64:
        assert out["auto"][1] == out["assembled-two-phase"][1]
