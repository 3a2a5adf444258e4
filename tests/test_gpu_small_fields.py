"""Fields close to the smallest normal numbers: a plate that cools to zero.

The solve's threshold is at least the smallest normal number of the handle's
type for |r|^2, so the CG scalars gamma = r.D^-1 r and delta reach denormals
while a solve still iterates.  Their quotients are ordinary numbers all the
way down; no solve there is a breakdown.
"""
import numpy as np
import pytest

from fea_gb300 import meshgen as mg
from test_gpu_stiff import CELLS, flattened

pytestmark = pytest.mark.gpu


def _set(s, u):
    import torch
    dt = torch.float64 if s.precision == 1 else torch.float32
    t = torch.tensor(u, dtype=dt, device="cuda")
    z = torch.zeros_like(t)
    torch.cuda.synchronize()
    s.set_fields_device(t.data_ptr(), z.data_ptr())


def _mesh(name):
    if name == "stiff":
        return flattened(68, 0.02, CELLS)
    return mg.jittered_grid(int(name), seed=3)


# one block, a cluster, a device-wide grid, stiff groups
@pytest.mark.parametrize("mesh", ["18", "60", "110", "stiff"])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("variant", [None, 14])
def test_heat_to_zero_raises_no_flag(fea, mesh, prec, variant):
    xyz, tri = _mesh(mesh)
    p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=20.0,
                           cg_tolerance=1e-10 if prec else 1e-6)
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.DIRICHLET, precision=prec, params=p)
    if variant:
        s.set_cg_variant(variant)
    u = np.random.default_rng(1).uniform(0.5, 1.0, s.info.num_unknowns)
    start = range(-150, -165, -1) if prec else range(-10, -25, -1)
    for e in start:  # each from one magnitude on, two decay steps and more
        _set(s, u * 10.0 ** e)
        s.advance_time(6)
        st = s.status()
        assert st.flags == 0 and st.steps_done == 6, (e, st.flags)
