"""The device-built ordering and tile-ELL layout at their edges.

A fan (one hub joined to every rim vertex) puts n columns in the hub's row, so
its tile's halo list grows with n: below the small hash set's limit (768), at
and past it (the large set), and past what the operand budget of the layout
holds (the CSR kernels take over).  Vertices are numbered at random, so the
ordering's sort moves them all.  One heat step against the FP64 oracle.
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def fan(n, seed):
    th = 2 * np.pi * np.arange(n) / n
    xyz = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(th), np.sin(th)], 1)])
    xyz = np.concatenate([xyz, np.zeros((n + 1, 1))], 1).astype(np.float32)
    i = np.arange(n)
    tri = np.stack([np.zeros(n, int), 1 + i, 1 + (i + 1) % n], 1)
    perm = np.random.default_rng(seed).permutation(n + 1)  # old -> new number
    out = np.empty_like(xyz)
    out[perm] = xyz
    return out, perm[tri].astype(np.uint32)


@pytest.mark.parametrize("n,fp64", [(3, 0), (255, 0), (256, 0), (257, 0), (1023, 0), (1024, 0), (1100, 0),
                                    (5000, 0), (6200, 1)])
def test_fan_heat_step(fea, oracle_mod, n, fp64):
    xyz, tri = fan(n, seed=n)
    p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1e-3, cg_tolerance=1e-7)
    s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=fea.FP64 if fp64 else fea.FP32,
                       params=p)
    if fp64:  # 96 KiB of (u, v) pairs less the tile's 256 rows: 5888 halo columns at most
        assert s.info.rows_per_warp_lanes == 8
    u0 = np.random.default_rng(1).uniform(0.5, 1.5, n + 1).astype(np.float32)
    s.set_values(u0)
    s.advance_time(1)
    assert s.status().flags == 0
    S = oracle_mod.System(xyz, tri, bc=oracle_mod.NEUMANN)
    po = oracle_mod.params(oracle_mod.HEAT, float(np.float32(1e-3)), kappa=float(np.float32(1e-3)), tol=1e-14)
    uo, *_ = S.step(po, S.gather(u0), np.zeros(S.N))
    assert rel_l2(s.get_values(), S.scatter(uo)) < 1e-5


@pytest.mark.parametrize("n", [63, 64, 65, 91])  # 3969 to 8281 rows: the one-block sort ends at 4096
def test_shuffled_grid_heat_step(fea, oracle_mod, n):
    from fea_gb300 import meshgen as mg
    xyz, tri = mg.jittered_grid(n, seed=n)
    perm = np.random.default_rng(n).permutation(len(xyz))
    out = np.empty_like(xyz)
    out[perm] = xyz
    tri = perm[tri].astype(np.uint32)
    p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0, cg_tolerance=1e-7)
    s = fea.CUDASolver(out, tri, boundary_condition=fea.NEUMANN, params=p)
    u0 = np.random.default_rng(1).uniform(0.5, 1.5, len(out)).astype(np.float32)
    s.set_values(u0)
    s.advance_time(1)
    S = oracle_mod.System(out, tri, bc=oracle_mod.NEUMANN)
    po = oracle_mod.params(oracle_mod.HEAT, float(np.float32(1e-3)), kappa=1.0, tol=1e-14)
    uo, *_ = S.step(po, S.gather(u0), np.zeros(S.N))
    assert rel_l2(s.get_values(), S.scatter(uo)) < 1e-5
