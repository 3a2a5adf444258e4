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


@pytest.mark.parametrize("variant", [None, 14])
@pytest.mark.parametrize("prec", [0, 1])
def test_stiff_loop_stops_at_the_smallest_normal_number(fea, variant, prec):
    """With stiff groups a loop stops at an eighth of the tolerance, but never asks |r|^2
    below the smallest normal number: the same solve scaled up by a power of two, with
    the tolerance at that point, does as many iterations."""
    xyz, tri = flattened(68, 0.02, CELLS)
    its = []
    rng = np.random.default_rng(2)
    tiny = 2.0 ** -1022 if prec else 2.0 ** -126
    scale = 2.0 ** -495 if prec else 2.0 ** -54
    u = None
    for small in (True, False):
        p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0, cg_refine=0,
                               cg_tolerance=1e-10 if prec else 1e-6)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        if variant:
            s.set_cg_variant(variant)
        if u is None:
            u = rng.uniform(0.5, 1.0, s.info.num_unknowns).astype(s.real).astype(np.float64)
            # |b|^2 of b = (M/dt) u, up to a few per cent
            rp, col, M, _ = s.matrix(fea.MASS)
            rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
            b = np.bincount(rows, weights=np.asarray(M, np.float64) * u[col], minlength=len(u)) / 1e-3
            bb = float(b @ b)
        if not small:
            p.cg_tolerance = 8.0 * np.sqrt(tiny / scale ** 2 / bb)
            assert p.cg_tolerance > 100 * (1e-10 if prec else 1e-6)
            s.set_params(p)
        _set(s, u * scale if small else u)
        s.advance_time(1)
        st = s.status()
        assert st.flags == 0
        its.append(st.total_iterations)
    # (squares of denormal size carry three digits: the count may move a little; a factor
    # of eight in |r| is more)
    assert abs(its[0] - its[1]) <= 2, its
