"""The assembled operator's closed-form element blocks, the neo-Hookean law's and
stiffness damping's, against the element-by-element operator: more corners of a
node than one group of the gather holds, fewer, and none left over."""
import pytest

import talus_b200 as tb
from tests.helpers import DT, GRAVITY, relative_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (3, 2, 4), (12, 11, 10)])
@pytest.mark.parametrize("law", ["neo-hookean", "damped", "damped plastic"])
@pytest.mark.parametrize("precision,solve,tol", [(tb.FP64, 1e-11, 1e-8), (tb.FP32_MIXED, 1e-6, 1e-5)])
def test_blocks_match_the_element_operator(cells, law, precision, solve, tol):
    mesh = tb.box_mesh(cells, voxel=0.1, jitter=0.01, seed=5)
    settings = tb.Settings(law=tb.NEO_HOOKEAN if law == "neo-hookean" else tb.COROTATED, tolerance=solve)
    kind = {} if law == "neo-hookean" else dict(stiffness_damping=0.03)
    if law == "damped plastic":
        kind["yield_stress"] = 1e3
    mat = tb.PhysicalMaterial(density=1000.0, youngs_modulus=1e6, poissons_ratio=0.3, **kind)
    out = {}
    for form in ("assembled", "elementwise"):
        s = tb.System(mesh, [mat], precision)
        s.set_solver(form)
        s.set_state(tb.rest_state(mesh))
        for _ in range(3):
            s.step(settings, GRAVITY, DT)
        out[form] = s.get_state().position
        s.close()
    assert relative_error(out["assembled"], out["elementwise"], mesh.rest_positions) <= tol
