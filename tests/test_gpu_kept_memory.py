"""Device memory a handle keeps between calls: the adjoint's states are given
back when they are large, the work arrays of the mesh's size are kept."""
import numpy as np
import pytest

from fea_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

KEPT = 64 << 20  # checkpoints and segment states a handle may keep


@pytest.mark.parametrize("eq", ["advdiff", "gs"])
def test_adjoint_gives_large_states_back(fea, eq):
    import torch
    xyz, tri = mg.jittered_grid(400, seed=0)
    n, steps = len(xyz), 80 if eq == "advdiff" else 40
    dt = torch.float64
    f = torch.tensor(np.random.default_rng(0).uniform(0.2, 0.8, (4, n)), dtype=dt, device="cuda")
    if eq == "advdiff":
        p = fea.default_params(equation=fea.ADVECTION_DIFFUSION, advection_scheme=1, advdiff_time_step=1e-3,
                               advdiff_c=0.1, cg_tolerance=1e-10)
    else:
        p = fea.default_params(equation=fea.REACTION_DIFFUSION, rd_Du=2e-5, rd_Dv=1e-5, rd_time_step=1.0,
                               rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_tolerance=1e-10)
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=fea.FP64, params=p)

    def sweep(k):
        if eq == "advdiff":
            return s.adjoint_advdiff_device(f[0], f[1], k, 1)
        return s.adjoint_gray_scott_device(f[0], f[1], f[2], f[3], k, 1)

    before = s.info.device_bytes
    first = sweep(4)
    work = s.info.device_bytes - before  # the work arrays and small states stay
    states = (steps + 2) * n * 8 * (1 if eq == "advdiff" else 2)
    assert states > KEPT + work
    sweep(steps)
    assert s.info.device_bytes - before <= work + KEPT
    again = sweep(4)  # and the next sweep finds what it needs
    assert first[0] == again[0]
    assert all(torch.equal(torch.as_tensor(a), torch.as_tensor(b)) for a, b in zip(first[1:], again[1:]))
