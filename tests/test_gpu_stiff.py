"""Solves in the stiff groups' basis (csrc/stiff.cu) against the FP64 oracle.

Grids with some cells flattened: one corner of a triangle sits `eps` cell
sizes from the opposite edge, which ties its three vertices together.  One
lies at the grid's corner, some are neighbours (groups that share vertices
and meet the limit of four), one is at the far end, the rest (enough for the
groups to be used) is spread over the grid.  Every equation whose
operator the groups change, both precisions and boundary conditions; the
iteration count against a kernel family without groups.
"""
import numpy as np
import pytest

from conftest import rel_l2
from fea_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def flattened(n, eps, cells):
    xyz, tri = mg.jittered_grid(n, seed=n, jitter=0.1)
    h = 1.0 / (n - 1)
    for j, i in cells:
        k = 2 * (j * (n - 1) + i)
        a, b, c = tri[k]  # (v00, v10, v11) or (v00, v10, v01)
        p, q = (a, c) if np.linalg.norm(xyz[c] - xyz[a]) > np.linalg.norm(xyz[c] - xyz[b]) else (b, c)
        m = b if p == a else a
        d = xyz[q] - xyz[p]
        nrm = np.array([-d[1], d[0], 0.0]) / np.linalg.norm(d)
        side = np.sign(np.dot(xyz[m] - xyz[p], nrm))
        xyz[m] = (0.55 * xyz[p] + 0.45 * xyz[q] + side * eps * h * nrm).astype(np.float32)
    return xyz, tri


CELLS = [(4, 4), (4, 5), (5, 4), (0, 0), (35, 36)] + [(j, i) for j in range(8, 36, 4) for i in range(2, 36, 5)]
EQS = {
    "heat": dict(equation="HEAT", heat_time_step=1e-3, heat_conductivity=1.0),
    "explicit": dict(equation="ADVECTION_DIFFUSION", advdiff_time_step=1e-3, advdiff_c=0.25, advection_scheme=1),
    "wave": dict(equation="WAVE", wave_time_step=2e-2, wave_c=1.0, wave_scheme=0),
    "newmark": dict(equation="WAVE", wave_time_step=2e-2, wave_c=1.0, wave_scheme=1),
    "gs": dict(equation="REACTION_DIFFUSION", rd_time_step=1.0, rd_Du=2e-3, rd_Dv=1e-3, rd_feed_rate=0.037,
               rd_kill_rate=0.06, reaction_mode=1),
}


@pytest.mark.parametrize("eq", list(EQS))
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("prec", [0, 1])
def test_steps_match_oracle(fea, oracle_mod, eq, bc, prec):
    O = oracle_mod
    xyz, tri = flattened(68, 0.02, CELLS)
    kw = dict(EQS[eq])
    p = fea.default_params(**{**kw, "equation": getattr(fea, kw["equation"])}, cg_tolerance=1e-12 if prec else 1e-7)
    s = fea.CUDASolver(xyz, tri, boundary_condition=bc, precision=prec, params=p)
    assert s.info.rows_per_warp_lanes == 14
    rng = np.random.default_rng(3)
    u0 = (0.5 + 0.3 * np.sin(5 * xyz[:, 0]) * np.cos(4 * xyz[:, 1])).astype(np.float32)
    v0 = (0.2 + 0.1 * np.cos(3 * xyz[:, 0])).astype(np.float32)
    u0 += rng.uniform(-0.01, 0.01, len(u0)).astype(np.float32)
    s.set_fields(u0, v0)
    s.advance_time(3)
    assert s.status().flags == 0
    S = O.System(xyz, tri, bc=bc)
    name = kw["equation"]
    if name == "HEAT":
        po = O.params(O.HEAT, p.heat_time_step, kappa=p.heat_conductivity, tol=1e-15)
    elif name == "ADVECTION_DIFFUSION":
        po = O.params(O.ADVECTION_DIFFUSION, p.advdiff_time_step, kappa=p.advdiff_c, adv_scheme=p.advection_scheme,
                      adv_sign=p.advection_sign, tol=1e-15)
    elif name == "WAVE":
        po = O.params(O.WAVE, p.wave_time_step, kappa=p.wave_c, wave_scheme=p.wave_scheme, tol=1e-15)
    else:
        po = O.params(O.REACTION_DIFFUSION, p.rd_time_step, Du=p.rd_Du, Dv=p.rd_Dv, F=p.rd_feed_rate,
                      k=p.rd_kill_rate, reaction_mode=p.reaction_mode, tol=1e-15)
    a = S.newmark_init(po, S.gather(u0)) if eq == "newmark" else None
    uo, vo, *_ = S.step(po, S.gather(u0), S.gather(v0), a, nsteps=3)
    ug, vg = s.get_fields()
    # node values travel as float32; the wave's velocity carries the acceleration's error (1e-4 as elsewhere)
    bar = 1e-7 if prec else 1e-5
    assert rel_l2(ug, S.scatter(uo)) < bar
    if name in ("REACTION_DIFFUSION", "WAVE"):
        assert rel_l2(vg, S.scatter(vo)) < (bar if prec or name != "WAVE" else 1e-4)


@pytest.mark.parametrize("n,eps", [(68, 0.02), (97, 1e-3), (130, 0.01)])
def test_fewer_iterations(fea, n, eps):
    xyz, tri = flattened(n, eps, CELLS + [(n - 3, n - 4)])
    its, out = [], []
    for variant in (11, 14):
        p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0, cg_tolerance=1e-10)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=fea.FP64, params=p)
        s.set_cg_variant(variant)
        u0 = np.random.default_rng(5).uniform(0, 1, len(xyz)).astype(np.float32)
        s.set_values(u0)
        s.advance_time(2)
        assert s.status().flags == 0
        its.append(s.status().total_iterations)
        out.append(s.get_values())
    assert rel_l2(out[1], out[0]) < 1e-7  # float32 node values of two solves to 1e-10
    assert its[1] < its[0], its
