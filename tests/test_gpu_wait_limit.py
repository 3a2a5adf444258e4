"""A wait of the resident launch that expires (csrc/resident.cu).

FEA_WAIT_CLOCKS bounds every wait of a launch.  With one clock the first word
that has not arrived yet expires it: the call reports FEA_STATUS_BREAKDOWN,
no block waits any longer, the call's later launches do nothing, and the
handle steps as a new one does once the limit is back.
"""
import numpy as np
import pytest

from fea_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

BREAKDOWN = 8


@pytest.mark.parametrize("n", [48, 100, 250])  # a cluster, a device-wide grid, several tiles a block
@pytest.mark.parametrize("prec", [0, 1])
def test_expired_wait_reports_and_recovers(fea, monkeypatch, n, prec):
    xyz, tri = mg.cylinder(n, n)
    p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_time_step=1.0, rd_Du=2e-4, rd_Dv=1e-4,
                           rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_initial_guess=1,
                           cg_tolerance=1e-10 if prec else 1e-6)
    rng = np.random.default_rng(n)
    u = (1 - 0.5 * rng.uniform(size=len(xyz))).astype(np.float32)
    v = (0.25 * rng.uniform(size=len(xyz))).astype(np.float32)

    def fresh():
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        s.set_fields(u, v)
        return s

    ref = fresh()
    ref.advance_time(8)
    s = fresh()
    s.advance_time(2)  # the epochs are under way
    assert s.status().flags == 0
    monkeypatch.setenv("FEA_WAIT_CLOCKS", "1")
    s.advance_time(600)  # three launches
    st = s.status()
    assert st.flags & BREAKDOWN
    assert st.steps_done < 256  # the launches after the expired one did nothing
    monkeypatch.delenv("FEA_WAIT_CLOCKS")
    s.clear_values()
    s.set_fields(u, v)
    s.advance_time(8)
    st = s.status()
    assert st.flags == 0 and st.steps_done == 8
    assert all(np.array_equal(a, b) for a, b in zip(s.get_fields(), ref.get_fields()))


@pytest.mark.parametrize("eq", ["advdiff", "gs"])
def test_expired_wait_in_an_adjoint_is_an_error(fea, monkeypatch, eq):
    """The sweep's later solves do not hide it: no loss and no gradient come back."""
    import torch
    xyz, tri = mg.jittered_grid(100, seed=2)
    if eq == "advdiff":
        p = fea.default_params(equation=fea.ADVECTION_DIFFUSION, advection_scheme=1, advdiff_time_step=1e-2,
                               advdiff_c=0.1, cg_tolerance=1e-10)
    else:
        p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_Du=2e-4, rd_Dv=1e-4, rd_time_step=1.0,
                               rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_tolerance=1e-10)
    f = torch.tensor(np.random.default_rng(0).uniform(0.2, 0.8, (4, len(xyz))), dtype=torch.float64, device="cuda")
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=fea.FP64, params=p)

    def sweep():
        if eq == "advdiff":
            return s.adjoint_advdiff_device(f[0], f[1], 6, 3)
        return s.adjoint_gray_scott_device(f[0], f[1], f[2], f[3], 6, 3)

    ref = sweep()
    monkeypatch.setenv("FEA_WAIT_CLOCKS", "1")
    with pytest.raises(fea.FeaError) as err:
        sweep()
    assert err.value.code == -9
    monkeypatch.delenv("FEA_WAIT_CLOCKS")
    again = sweep()
    assert again[0] == ref[0]
    assert all(torch.equal(torch.as_tensor(a), torch.as_tensor(b)) for a, b in zip(again[1:], ref[1:]))


def test_expired_wait_in_the_starting_acceleration_is_kept(fea, monkeypatch):
    """Newmark's first call runs two launches; the second does not clear the first's word."""
    xyz, tri = mg.cylinder(100, 100)
    p = fea.default_params(equation=fea.WAVE, wave_time_step=2e-3, wave_c=1.0, wave_scheme=1, cg_tolerance=1e-6)
    u = np.random.default_rng(0).uniform(size=len(xyz)).astype(np.float32)
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, params=p)
    s.set_fields(u, u)
    monkeypatch.setenv("FEA_WAIT_CLOCKS", "1")
    s.advance_time(1)
    assert s.status().flags & BREAKDOWN
    monkeypatch.delenv("FEA_WAIT_CLOCKS")
    s.clear_values()
    assert s.status().flags == 0
    s.set_fields(u, u)
    s.advance_time(3)
    ref = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, params=p)
    ref.set_fields(u, u)
    ref.advance_time(3)
    assert s.status().flags == 0
    assert all(np.array_equal(a, b) for a, b in zip(s.get_fields(), ref.get_fields()))
