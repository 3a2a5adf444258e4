"""Stiff groups against the caller's settings: the iteration limit, autotuning,
refinement modes and the extrapolated start, in the resident launch and on the
step graph's own kernels."""
import numpy as np
import pytest

from conftest import f32, rel_l2
from test_gpu_stiff import CELLS, flattened

pytestmark = pytest.mark.gpu


def _heat(fea, prec, **kw):
    return fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0, **kw)


def _noise(n, seed=5):
    return np.random.default_rng(seed).uniform(0, 1, n).astype(np.float32)


@pytest.mark.parametrize("variant", [None, 14])
@pytest.mark.parametrize("prec", [0, 1])
def test_limit_is_judged_by_the_callers_tolerance(fea, variant, prec):
    """A solve that meets cg_tolerance when the limit ends it has converged."""
    xyz, tri = flattened(68, 0.02, CELLS)
    tol = 1e-10 if prec else 1e-5

    def run(tolerance, limit):
        p = _heat(fea, prec, cg_tolerance=tolerance, cg_refine=0, cg_max_iterations=limit)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        if variant:
            s.set_cg_variant(variant)
        s.set_values(_noise(len(xyz)))
        s.advance_time(1)
        return s.status()

    reach, past = run(8 * tol, 0).total_iterations, run(tol, 0).total_iterations
    assert reach < past
    for limit in range(reach, past):
        st = run(tol, limit)
        assert st.total_iterations == limit
        if st.last_rel_residual[0] < tol:
            assert st.flags == 0, (limit, reach, past)
        else:
            assert st.flags == 4, (limit, reach, past)
    assert run(tol, past - 1).last_rel_residual[0] < tol  # the case this is about occurred
    st = run(tol, max(1, reach // 2))
    assert st.flags == 4 and st.last_rel_residual[0] > tol


@pytest.mark.parametrize("variant", [None, 14])
def test_limit_two_fields(fea, variant):
    """Per field: one field within the tolerance at the limit and one not is not converged."""
    xyz, tri = flattened(68, 0.02, CELLS)
    flags = []
    for limit in range(1, 60):
        p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_time_step=1.0, rd_Du=2e-3, rd_Dv=1e-3,
                               rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_tolerance=1e-5, cg_refine=0,
                               cg_max_iterations=limit)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, params=p)
        if variant:
            s.set_cg_variant(variant)
        s.set_fields(1 - 0.5 * _noise(len(xyz)), 0.25 * _noise(len(xyz), 6))
        s.advance_time(1)
        st = s.status()
        assert (st.flags == 4) == (max(st.last_rel_residual) >= 1e-5), (limit, list(st.last_rel_residual))
        flags.append(st.flags)
        if st.total_iterations < limit:
            break
    assert flags[0] == 4 and flags[-1] == 0


@pytest.mark.parametrize("n", [68, 130, 300])
@pytest.mark.parametrize("prec", [0, 1])
def test_autotune_keeps_the_groups(fea, n, prec):
    """The variant autotuning leaves behind takes no more iterations than the default."""
    xyz, tri = flattened(n, 0.02, CELLS)
    its = []
    for tune in (False, True):
        p = _heat(fea, prec, cg_tolerance=1e-10 if prec else 1e-6)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        if tune:
            s.autotune()
        s.set_values(_noise(len(xyz)))
        s.advance_time(2)
        assert s.status().flags == 0
        its.append(s.status().total_iterations)
    assert its[1] <= its[0] + 2, (its, s.info.rows_per_warp_lanes)


@pytest.mark.parametrize("variant", [None, 14, 15])
@pytest.mark.parametrize("refine", [0, 1, 2])
@pytest.mark.parametrize("guess", [0, 1])
def test_gray_scott_matches_oracle(fea, oracle_mod, variant, refine, guess):
    O = oracle_mod
    xyz, tri = flattened(68, 0.02, CELLS)
    p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_time_step=1.0, rd_Du=2e-3, rd_Dv=1e-3,
                           rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_tolerance=1e-7, cg_refine=refine,
                           cg_initial_guess=guess)
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, params=p)
    if variant:
        s.set_cg_variant(variant)
    u0, v0 = 1 - 0.5 * _noise(len(xyz)), 0.25 * _noise(len(xyz), 6)
    s.set_fields(u0, v0)
    s.advance_time(3)
    S = O.System(xyz, tri, bc=O.NEUMANN)
    po = O.params(O.REACTION_DIFFUSION, 1.0, Du=f32(2e-3), Dv=f32(1e-3), F=f32(0.037), k=f32(0.06), reaction_mode=1,
                  tol=1e-15)
    uo, vo, *_ = S.step(po, S.gather(u0), S.gather(v0), nsteps=3)
    ug, vg = s.get_fields()
    assert s.status().flags == 0
    assert rel_l2(ug, S.scatter(uo)) < 1e-5 and rel_l2(vg, S.scatter(vo)) < 1e-5  # float32 fields, as elsewhere
