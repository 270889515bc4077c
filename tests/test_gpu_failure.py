"""Failure detection on the GPU without a GPU fault.

Every spin in the persistent kernels is bounded (2 s on the grid barrier);
when it runs out the kernel records TL_ERR_TIMEOUT in a status word the host
reads, and the context stays usable.  tl_ctx_check_wait_limit makes that wait
run out: one block waits at the barrier for an arrival that never comes.
Afterwards the same context steps a body normally.  The host-side failure
paths (a rank that raises, never joins) are covered with gloo ranks in
test_shard.
"""
import ctypes as C
import time

import numpy as np
import pytest

import talus_b200 as tb
from talus_b200 import _capi as capi
from tests.helpers import DT, GRAVITY, elastic_block

pytestmark = pytest.mark.gpu


def test_bounded_wait_runs_out_with_a_status_and_the_context_stays_usable():
    ctx = tb.Context(0)
    began = time.perf_counter()
    rc = capi.lib().tl_ctx_check_wait_limit(ctx.handle)
    waited = time.perf_counter() - began
    assert rc == capi.TL_ERR_TIMEOUT
    assert 1.5 < waited < 30.0
    assert b"bounded wait" in capi.lib().tl_ctx_last_error(ctx.handle)
    mesh, mat = elastic_block((4, 4, 4), seed=6)
    system = tb.System(mesh, [mat], tb.FP64, context=ctx)
    system.set_state(tb.rest_state(mesh))
    report = system.step(tb.Settings(), GRAVITY, DT)[0]
    assert report.cg_iterations > 0
    assert np.isfinite(system.get_state().position).all()
    system.close()
    ctx.close()


@pytest.mark.parametrize("solve", [0, 1])
def test_a_wait_that_runs_out_in_an_early_solve_is_reported_at_the_step_end(solve):
    """The elastic step runs three PCG solves.  When the barrier wait of an
    early one runs out, the later solves of the same step must not erase the
    record: the step returns TL_ERR_TIMEOUT.  The next step runs normally."""
    mesh, mat = elastic_block((4, 4, 4), seed=6)
    system = tb.System(mesh, [mat], tb.FP64)
    system.set_state(tb.rest_state(mesh))
    assert capi.lib().tl_system_expire_wait(system.handle, solve) == capi.TL_OK
    reports = (tb.StepReport * 1)()
    g = np.asarray(GRAVITY, np.float64)
    rc = capi.lib().tl_step(system.handle, C.byref(tb.Settings()._c()), g.ctypes.data, DT, reports)
    assert rc == capi.TL_ERR_TIMEOUT
    system.set_state(tb.rest_state(mesh))
    report = system.step(tb.Settings(), GRAVITY, DT)[0]
    assert report.cg_iterations > 0
    assert np.isfinite(system.get_state().position).all()
    system.close()


@pytest.mark.parametrize("solve", [0, 2])
def test_factored_solve_reports_an_expired_wait(solve):
    """The same host-armed expiry on a system with a solver state: the
    factored PCG (kPcgFactor, whose grid barriers and supernode waits are
    bounded the same way) leaves at its first barrier, the step returns
    TL_ERR_TIMEOUT, and the next step runs normally with the factor."""
    mesh, mat = elastic_block((4, 4, 4), seed=6)
    system = tb.System(mesh, [mat], tb.FP64)
    system.use_factor(True, 32)
    system.set_state(tb.rest_state(mesh))
    system.step(tb.Settings(), GRAVITY, DT)
    assert capi.lib().tl_system_expire_wait(system.handle, solve) == capi.TL_OK
    reports = (tb.StepReport * 1)()
    g = np.asarray(GRAVITY, np.float64)
    rc = capi.lib().tl_step(system.handle, C.byref(tb.Settings()._c()), g.ctypes.data, DT, reports)
    assert rc == capi.TL_ERR_TIMEOUT
    system.set_state(tb.rest_state(mesh))
    report = system.step(tb.Settings(), GRAVITY, DT)[0]
    assert report.cg_iterations > 0
    assert np.isfinite(system.get_state().position).all()
    assert system.factor_stats()["ready"] == 1
    system.close()


def _expired_step(system, solve):
    assert capi.lib().tl_system_expire_wait(system.handle, solve) == capi.TL_OK
    reports = (tb.StepReport * len(system.meshes))()
    g = np.asarray(GRAVITY, np.float64)
    return capi.lib().tl_step(system.handle, C.byref(tb.Settings()._c()), g.ctypes.data, DT, reports)


# one body over many blocks of kPcgSell; bodies of one block each; one of several beside one of one
@pytest.mark.parametrize("cells", [[(16, 16, 17)], [(3, 3, 3), (2, 5, 3), (4, 4, 4)], [(12, 11, 10), (2, 2, 2)]])
@pytest.mark.parametrize("precision", [tb.FP64, tb.FP32_MIXED])
def test_every_solve_of_a_step_leaves_after_an_expired_wait(cells, precision):
    """kPcgSell over one body and over a batch's queue: a wait that ran out before the first solve ends all solves of
    the step, those of bodies that meet no barrier too, so no acceleration of a body at rest changes.  The next step
    runs normally."""
    meshes = [tb.box_mesh(c, voxel=0.1, jitter=0.01, seed=6) for c in cells]
    mats = [[tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3)] for _ in meshes]
    system = tb.System(meshes, mats, precision)
    for i, m in enumerate(meshes):
        system.set_state(tb.rest_state(m), i)
    assert _expired_step(system, 0) == capi.TL_ERR_TIMEOUT
    for i in range(len(meshes)):
        assert not system.get_state(i).acceleration.any(), i
    for i, m in enumerate(meshes):
        system.set_state(tb.rest_state(m), i)
    reports = system.step(tb.Settings(), GRAVITY, DT)
    assert all(r.cg_iterations > 0 for r in reports)
    for i in range(len(meshes)):
        assert np.isfinite(system.get_state(i).position).all()
    system.close()


@pytest.mark.parametrize("solve", [0, 2])
def test_the_lean_factored_solve_reports_an_expired_wait(solve):
    mesh, mat = elastic_block((4, 4, 4), seed=6)
    system = tb.System(mesh, [mat], tb.FP64)
    capi.check(capi.lib().tl_system_use_factor(system.handle, 2, 32), system.context.handle)
    system.set_state(tb.rest_state(mesh))
    system.step(tb.Settings(), GRAVITY, DT)
    assert _expired_step(system, solve) == capi.TL_ERR_TIMEOUT
    system.set_state(tb.rest_state(mesh))
    assert system.step(tb.Settings(), GRAVITY, DT)[0].cg_iterations > 0
    assert system.factor_stats()["ready"] == 1
    system.close()
