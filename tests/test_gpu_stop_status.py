"""The status after a call that stops early: figures of the last step done."""
import numpy as np
import pytest

from conftest import rel_l2
from fea_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 60, 110])  # one block, a cluster, a device-wide grid
@pytest.mark.parametrize("prec", [0, 1])
def test_blow_up_inside_a_call(fea, n, prec):
    """Explicit advection far above its stability limit passes 1e4 after some steps."""
    xyz, tri = mg.jittered_grid(n, seed=1)
    tol = 1e-10 if prec else 1e-6
    p = fea.default_params(equation=fea.ADVECTION_DIFFUSION, advection_scheme=1, advdiff_time_step=1e-2,
                           advdiff_c=0.01, velocity_mode=1, cg_tolerance=tol)
    vel = np.tile(np.array([30.0, 20.0, 0.0], np.float32), (len(tri), 1))
    u = np.random.default_rng(n).uniform(0, 1, len(xyz)).astype(np.float32)
    got = []
    for variant in (14, None):
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        s.set_element_fields(velocity=vel)
        if variant:
            s.set_cg_variant(variant)
        s.set_values(u)
        s.advance_time(60)
        got.append((s.status(), s.get_values()))
    (a, x), (b, y) = got
    assert a.flags == b.flags == 1 and 0 < a.steps_done < 60
    assert b.steps_done == a.steps_done
    assert a.last_iterations[0] > 0 and abs(b.last_iterations[0] - a.last_iterations[0]) <= 2
    for st in (a, b):
        assert 0 < st.last_rel_residual[0] < tol
    assert rel_l2(y, x) < (1e-6 if prec else 1e-3)  # (the errors of the solves grow with the field)
