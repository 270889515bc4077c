"""Solves to tight tolerances in the pipelined orders of the assembled PCG, on
stiff and on layered bodies.  The step's own measure has to hold: no solve of a
body ends above the tolerance it was given, however small the steps' reported
iteration counts are.  The bar is the stopping rule itself, |r| <= tolerance
|right|, with the rounding of the ratio that is reported."""
import numpy as np
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, plastic_block

pytestmark = pytest.mark.gpu

ROUNDING = 1.0 + 1e-12


def material(youngs, poisson=0.35):
    return tb.PhysicalMaterial(density=1000.0, youngs_modulus=youngs, poissons_ratio=poisson)


def stepped(meshes, mats, precision, tolerance, form, law=tb.COROTATED, youngs=None):
    s = tb.System(meshes, mats, precision)
    s.set_solver(form)
    if youngs is not None:
        s.set_youngs(youngs)
    for i, m in enumerate(s.meshes):
        state = tb.rest_state(m)
        free = (m.anchored == 0)[:, None]
        state.velocity[...] = 0.2 * free * np.sin(3.0 * m.rest_positions + i)
        s.set_state(state, i)
    settings = tb.Settings(law=law, tolerance=tolerance, cg_iterations=4000)
    reports = [s.step(settings, GRAVITY, DT) for _ in range(2)]
    s.close()
    return reports


def check(reports, tolerance):
    for step in reports:
        for b, r in enumerate(step):
            assert r.cg_capped_solves == 0, b
            assert r.cg_worst_relative_residual <= tolerance * ROUNDING, (b, r.cg_worst_relative_residual)


TOLERANCES = [(tb.FP32_MIXED, 1e-5), (tb.FP32_MIXED, 1e-6), (tb.FP64, 1e-11), (tb.FP64, 1e-12)]


@pytest.mark.parametrize("precision,tolerance", TOLERANCES)
def test_batch_of_stiff_bodies(precision, tolerance):
    rng = np.random.default_rng(4)
    dims = [tuple(int(c) for c in d) for d in rng.integers(4, 20, (24, 3))]
    meshes = [tb.box_mesh(c, voxel=0.1) for c in dims]
    mats = [[material(10.0 ** rng.uniform(6.0, 8.0), rng.uniform(0.25, 0.45))] for _ in dims]
    check(stepped(meshes, mats, precision, tolerance, "auto"), tolerance)


# 5,832 nodes; 6,710, slender; 9,261 nodes (48,000 tets)
@pytest.mark.parametrize("cells,youngs", [((17, 17, 17), 1e7), ((9, 60, 10), 1e8), ((20, 20, 20), 1e8)])
@pytest.mark.parametrize("law", [tb.COROTATED, tb.NEO_HOOKEAN])
@pytest.mark.parametrize("precision,tolerance", TOLERANCES)
def test_one_stiff_body(cells, youngs, law, precision, tolerance):
    mesh = tb.box_mesh(cells, voxel=0.1)
    check(stepped(mesh, [material(youngs)], precision, tolerance, "auto", law), tolerance)


@pytest.mark.parametrize("precision,tolerance", [(tb.FP32_MIXED, 1e-5), (tb.FP32_MIXED, 1e-6), (tb.FP64, 1e-8),
                                                 (tb.FP64, 1e-11)])
def test_layered_body(precision, tolerance):
    """A stiff layer over a soft one, 1e4 apart: the residual rises and falls by as much on the way."""
    mesh = tb.box_mesh((18, 17, 17), voxel=0.1)
    top = mesh.rest_positions[mesh.tet_nodes.astype(np.int64)][:, :, 1].mean(1) > 0.85
    reports = stepped(mesh, [material(1e5, 0.3)], precision, tolerance, "auto", youngs=np.where(top, 1e9, 1e5))
    check(reports, tolerance)


@pytest.mark.parametrize("precision,tolerance", [(tb.FP32_MIXED, 1e-5), (tb.FP32_MIXED, 1e-6), (tb.FP64, 1e-8),
                                                 (tb.FP64, 1e-12)])
def test_lockstep_pipelined_batch(precision, tolerance):
    """The lockstep pipelined order: bodies replace their recurrences in different phases, beside others that update,
    stop early or fill less than a tile."""
    meshes = [tb.box_mesh(c, voxel=0.1) for c in ((12, 11, 10), (3, 30, 4), (2, 2, 2), (9, 20, 9), (7, 7, 3))]
    mats = [[material(e, 0.35)] for e in (1e8, 3e7, 1e5, 1e8, 1e6)]
    check(stepped(meshes, mats, precision, tolerance, "assembled-pipelined"), tolerance)


def test_floating_body_at_the_default_settings():
    """A floating body solves to 1e-5 whatever the settings ask, in FP32-mixed too."""
    mesh = tb.box_mesh((17, 17, 17), voxel=0.1, jitter=0.01, seed=4, anchor_axis=3)
    check(stepped(mesh, [material(1e8)], tb.FP32_MIXED, 1e-3, "auto"), 1e-5)


@pytest.mark.parametrize("precision,tolerance", [(tb.FP32_MIXED, 1e-6), (tb.FP64, 1e-11)])
def test_yielding_body(precision, tolerance):
    """The plastic Newton loop's solves, with the consistent operator among them."""
    mesh, mat = plastic_block((18, 17, 17), speed=4.0)
    s = tb.System(mesh, [mat], precision)
    s.set_state(tb.rest_state(mesh))
    reports = [s.step(tb.Settings(tolerance=tolerance, cg_iterations=4000), GRAVITY, DT) for _ in range(3)]
    s.close()
    assert any(r[0].cg_tangent_iterations > 0 for r in reports)
    check(reports, tolerance)
