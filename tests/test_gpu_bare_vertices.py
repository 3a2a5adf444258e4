"""Vertices that no triangle names.

Their rows of every matrix are empty.  Under the reference's nodal reaction
(mode 0) such an unknown's equation reads 0 = reaction: no solution, and the
value runs away until the call stops on it, whatever kernel runs.  Under the
other equations its right-hand side is 0 and the other vertices' values do not
depend on it.
"""
import numpy as np
import pytest

from conftest import rel_l2
from fea_gb300 import meshgen as mg
from test_gpu_stiff import CELLS, flattened

pytestmark = pytest.mark.gpu


def _mesh(name, extra):
    xyz, tri = flattened(68, 0.02, CELLS) if name == "stiff" else mg.jittered_grid(int(name), seed=1)
    if extra:
        xyz = np.vstack([xyz, [[0.5, 0.5, 0.3], [2, 2, 2]]]).astype(np.float32)
    return xyz, tri


def _fields(n):
    r = np.random.default_rng(3)
    return (1 - 0.5 * r.uniform(size=n)).astype(np.float32), (0.25 * r.uniform(size=n)).astype(np.float32)


# one block, a cluster, a device-wide grid, stiff groups
@pytest.mark.parametrize("mesh", ["20", "70", "110", "stiff"])
@pytest.mark.parametrize("prec", [0, 1])
def test_nodal_reaction_reports_it(fea, mesh, prec):
    xyz, tri = _mesh(mesh, True)
    p = fea.default_params(equation=fea.REACTION_DIFFUSION, cg_tolerance=1e-10 if prec else 1e-6)
    out = []
    for variant in (11, None, 14):  # variant 11 iterates on the full layout
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        if variant:
            s.set_cg_variant(variant)
        s.set_fields(*_fields(len(xyz)))
        s.advance_time(8)
        st = s.status()
        out.append((st.flags, st.steps_done))
    for flags, done in out:
        assert flags & 1 and done < 8, out


@pytest.mark.parametrize("mesh", ["20", "70", "stiff"])
@pytest.mark.parametrize("mode", [1, "heat"])
def test_other_vertices_do_not_see_it(fea, mesh, mode):
    out = []
    for extra in (False, True):
        xyz, tri = _mesh(mesh, extra)
        n = len(xyz) - (2 if extra else 0)
        if mode == "heat":
            p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0, cg_tolerance=1e-12)
        else:
            p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_time_step=1.0, rd_Du=2e-4, rd_Dv=1e-4,
                                   reaction_mode=1, cg_tolerance=1e-12)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=fea.FP64, params=p)
        u, v = _fields(n)
        pad = np.full(2 if extra else 0, 0.5, np.float32)
        s.set_fields(np.concatenate([u, pad]), np.concatenate([v, pad]))
        s.advance_time(3)
        assert s.status().flags == 0
        out.append([f[:n] for f in s.get_fields()])
    assert rel_l2(out[1][0], out[0][0]) < 1e-7  # float32 node values of two solves to 1e-12
    assert mode == "heat" or rel_l2(out[1][1], out[0][1]) < 1e-7
