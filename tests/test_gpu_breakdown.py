"""Solves that end on the breakdown test (p.A p > 0 and r.u > 0): a squeezed
neo-Hookean body's tangent is indefinite.  Every order of the batched PCG stops
at the same iterate and reports that iterate's residual and the products it
made, and no solve is reported as converged that is not."""
import numpy as np
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY

pytestmark = pytest.mark.gpu

CELLS = [(4, 6, 5), (3, 4, 4)]


def report(form, squeeze, youngs, settings):
    meshes = [tb.box_mesh(c, voxel=0.1, jitter=0.01, seed=1 + i) for i, c in enumerate(CELLS)]
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=youngs, poissons_ratio=0.3)
    s = tb.System(meshes, [[mat], [mat]], tb.FP64)
    s.set_solver(form)
    for i, m in enumerate(meshes):
        state = tb.rest_state(m)
        state.position[:, 1] *= squeeze
        s.set_state(state, i)
    out = list(s.step(settings, GRAVITY, DT))
    s.close()
    return out


@pytest.mark.parametrize("squeeze,youngs", [(0.5, 1e6), (0.7, 1e8), (0.2, 1e8)])
def test_a_broken_down_solve_reports_its_residual(squeeze, youngs):
    settings = tb.Settings(law=tb.NEO_HOOKEAN, tolerance=1e-6, cg_iterations=2000)
    ref = report("elementwise", squeeze, youngs, settings)
    assert all(r.cg_worst_relative_residual > 0.1 and r.cg_capped_solves == 0 for r in ref)
    for form in ("assembled-two-phase", "assembled-pipelined", "auto"):
        for r, e in zip(report(form, squeeze, youngs, settings), ref):
            assert r.cg_iterations == e.cg_iterations, form
            # the iterates of two operators and orders in FP64, after at most 151 updates of an indefinite system
            assert abs(r.cg_worst_relative_residual / e.cg_worst_relative_residual - 1.0) <= 1e-4, form
            if form == "assembled-two-phase":
                assert r.operator_applications == e.operator_applications


@pytest.mark.parametrize("limit", [5, 2000])
def test_the_pipelined_orders_count_the_same_products(limit):
    settings = tb.Settings(tolerance=1e-3, cg_iterations=limit)
    lockstep, gang = (report(f, 1.0, 1e6, settings) for f in ("assembled-pipelined", "auto"))
    assert [r.operator_applications for r in lockstep] == [r.operator_applications for r in gang]
    assert all(r.operator_applications >= r.cg_iterations for r in gang)
