"""The two applications of a solver state's factor: its explicit inverse
(kPcgInverse, the default) and its triangular solves (kPcgFactor, the lean
form).  They apply the same factor, so their steps agree as two orderings of it
do: the bars of test_gpu_factor, the same iteration counts and counters.
Sizes: one leaf; a leaf of just under and over 64 free nodes; several levels;
rows past the length a whole block takes."""
import numpy as np
import pytest

import talus_b200 as tb
from talus_b200 import _capi as capi
from tests.helpers import DT, GRAVITY, plastic_block, relative_error

pytestmark = pytest.mark.gpu


def run(lean, precision, mesh, mat, state, steps):
    s = tb.System(mesh, [mat], precision)
    capi.check(capi.lib().tl_system_use_factor(s.handle, 2 if lean else 1, 32), s.context.handle)
    s.set_state(state)
    its = [s.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations for _ in range(steps)]
    x, stats = s.get_state().position, s.factor_stats()
    s.close()
    stats.pop("refactor_seconds")
    return x, its, stats


@pytest.mark.parametrize("cells", [(1, 1, 1), (3, 4, 3), (4, 3, 4), (6, 5, 7), (16, 8, 8)])
@pytest.mark.parametrize("precision,tol", [(tb.FP64, 1e-8), (tb.FP32_MIXED, 1e-5)])
def test_inverse_matches_the_triangular_solves(cells, precision, tol):
    mesh, mat = plastic_block(cells)
    state = tb.rest_state(mesh)
    inv, lean = (run(f, precision, mesh, mat, state, 3) for f in (False, True))
    assert relative_error(inv[0], lean[0], mesh.rest_positions) <= tol
    if precision == tb.FP64:
        assert inv[1] == lean[1] and inv[2] == lean[2]


def test_inverse_of_a_free_body():
    mesh = tb.box_mesh((5, 6, 7), voxel=0.1, jitter=0.01, seed=4, anchor_axis=3)
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)
    state = tb.rest_state(mesh)
    arm = mesh.rest_positions - mesh.rest_positions.mean(0)
    state.velocity[...] = np.array([0.3, 0.5, -0.2]) + np.cross([1.0, -2.0, 0.5], arm)
    inv, lean = (run(f, tb.FP64, mesh, mat, state, 3) for f in (False, True))
    assert relative_error(inv[0], lean[0], mesh.rest_positions) <= 1e-9
    assert inv[1] == lean[1] and inv[2] == lean[2]


def test_form_can_change_between_steps():
    mesh, mat = plastic_block((6, 5, 7))
    s = tb.System(mesh, [mat], tb.FP64)
    s.set_state(tb.rest_state(mesh))
    for enable in (1, 2, 1, 0, 2):
        capi.check(capi.lib().tl_system_use_factor(s.handle, enable, 32), s.context.handle)
        assert s.step(tb.Settings(), GRAVITY, DT)[0].non_finite == 0
    s.close()


@pytest.mark.parametrize("enable", [1, 2])
def test_a_dropped_state_gives_its_memory_back(enable):
    """16 x 8 x 8 cells: 17 MB of inverse, or 12 MB of factor blocks.  Allocations come in pieces of 2 MB."""
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    mesh, mat = plastic_block((16, 8, 8))
    s = tb.System(mesh, [mat], tb.FP64)
    s.set_state(tb.rest_state(mesh))
    use = lambda e: capi.check(capi.lib().tl_system_use_factor(s.handle, e, 32), s.context.handle)  # noqa: E731
    use(enable)  # the kernels' own memory, once
    s.step(tb.Settings(), GRAVITY, DT)
    use(0)
    s.step(tb.Settings(), GRAVITY, DT)
    before = free()
    use(enable)
    first = s.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations
    assert free() < before - (8 << 20)
    use(0)
    assert free() >= before - (2 << 20)
    assert s.step(tb.Settings(), GRAVITY, DT)[0].non_finite == 0
    use(enable)
    assert s.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations > 0 and first > 0
    s.close()


def test_the_form_that_runs_is_reported():
    mesh, mat = plastic_block((4, 3, 4))
    s = tb.System(mesh, [mat], tb.FP64)
    s.set_state(tb.rest_state(mesh))
    assert s.factor_form() is None
    for enable, form in ((1, "inverse"), (2, "lean"), (1, "inverse")):
        capi.check(capi.lib().tl_system_use_factor(s.handle, enable, 32), s.context.handle)
        s.step(tb.Settings(), GRAVITY, DT)
        assert s.factor_form() == form
    capi.check(capi.lib().tl_system_use_factor(s.handle, 0, 32), s.context.handle)
    assert s.factor_form() is None
    s.close()
