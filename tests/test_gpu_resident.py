"""The resident launch (csrc/resident.cu) against the step graph and the oracle.

The step graph runs the same recurrences (variant 14, chosen explicitly), so
the two agree to the rounding of their sums.  Sizes at the edges of the launch
shapes: one tile, two tiles in one block, a cluster's first and last sizes,
the cooperative grid's first, and several tiles per block.
"""
import threading

import numpy as np
import pytest

from conftest import rel_l2
from fea_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def _params(fea, eq, prec, grid):
    tol = 1e-12 if prec else 1e-6
    if eq == "heat":
        return fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=0.5, cg_tolerance=tol)
    if eq in ("advdiff", "explicit"):
        return fea.default_params(equation=fea.ADVECTION_DIFFUSION, advdiff_time_step=1e-3, advdiff_c=0.25,
                                  advection_scheme=int(eq == "explicit"), cg_tolerance=tol)
    if eq in ("wave", "newmark"):
        return fea.default_params(equation=fea.WAVE, wave_time_step=2e-3, wave_c=1.0, wave_scheme=int(eq == "newmark"),
                                  cg_tolerance=tol)
    return fea.default_params(equation=fea.REACTION_DIFFUSION, rd_time_step=1.0, rd_Du=2e-4, rd_Dv=1e-4,
                              rd_feed_rate=0.037, rd_kill_rate=0.06, reaction_mode=1, cg_tolerance=tol,
                              cg_initial_guess=int(eq == "gs1"))


def _both(fea, xyz, tri, bc, prec, p, steps, fields, calls=2):
    out = []
    for explicit in (True, False):
        s = fea.CUDASolver(xyz, tri, boundary_condition=bc, precision=prec, params=p)
        if explicit:
            s.set_cg_variant(14)
        s.set_fields(*fields)
        for _ in range(calls):
            s.advance_time(steps)
        st = s.status()
        out.append((s.get_fields(), st.total_iterations, st.flags, st.steps_done, list(st.last_rel_residual)))
    return out


# rows: one tile, its edges, two tiles, three (a cluster), a cluster's last (FP64
# 4096 rows, FP32 8192) and the grid's first, one and two tiles per block, more
SIZES = [(5, 3), (16, 16), (17, 16), (32, 16), (33, 16), (64, 64), (65, 64), (128, 64), (129, 64), (128, 128),
         (129, 128), (300, 260)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("eq", ["heat", "gs1"])
def test_sizes_match_step_graph(fea, nx, ny, prec, eq):
    xyz, tri = mg.cylinder(nx, ny)
    rng = np.random.default_rng(nx)
    u = (1 - 0.5 * rng.uniform(0, 1, len(xyz))).astype(np.float32)
    v = (0.25 * rng.uniform(0, 1, len(xyz))).astype(np.float32)
    a, b = _both(fea, xyz, tri, 1, prec, _params(fea, eq, prec, False), 3, (u, v))
    # two solves to the tolerance: 1e-12 (then float32 node values), 1e-6
    bar = 1e-7 if prec else 1e-5
    assert rel_l2(b[0][0], a[0][0]) < bar
    if eq != "heat":
        assert rel_l2(b[0][1], a[0][1]) < bar
    assert b[2] == a[2] == 0 and b[3] == a[3] == 3
    assert abs(b[1] - a[1]) <= 6 + a[1] // 50  # a solve may stop an iteration earlier or later


# three, four and five passes of a block's thread groups (on 152 SMs)
@pytest.mark.parametrize("nx,ny,prec,eq", [(400, 480, 0, "gs1"), (400, 480, 1, "heat"), (500, 480, 0, "gs1"),
                                           (500, 480, 1, "heat"), (500, 480, 0, "heat"), (600, 600, 0, "heat")])
def test_many_tiles_per_block(fea, nx, ny, prec, eq):
    test_sizes_match_step_graph(fea, nx, ny, prec, eq)


@pytest.mark.parametrize("eq", ["heat", "advdiff", "explicit", "wave", "newmark", "gs0", "gs1"])
@pytest.mark.parametrize("n", [40, 150])  # 7 tiles (cluster) and 88 (grid)
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("refine", [0, 1, 2])
def test_equations_match_step_graph(fea, eq, n, bc, refine):
    xyz, tri = mg.cylinder(n, n)
    p = _params(fea, eq, 0, False)
    p.cg_refine = refine
    u = (1 - 0.4 * np.exp(-np.sum((xyz - xyz[7]) ** 2, 1) / 0.1)).astype(np.float32)
    v = (0.2 * np.exp(-np.sum((xyz - xyz[-9]) ** 2, 1) / 0.2)).astype(np.float32)
    a, b = _both(fea, xyz, tri, bc, 0, p, 4, (u, v))
    assert rel_l2(b[0][0], a[0][0]) < 1e-5
    if eq in ("wave", "newmark", "gs0", "gs1"):
        assert rel_l2(b[0][1], a[0][1]) < 1e-5
    assert b[2] == a[2]
    assert all(abs(x - y) <= 1e-5 for x, y in zip(a[4], b[4]))


def test_many_steps_and_calls(fea):
    """More steps than one launch holds (256), the same in several calls, bit for bit."""
    xyz, tri = mg.icosphere(3)
    u, v = mg.sphere_patches(xyz, seed=2, n_patches=5, radius=0.4)
    p = _params(fea, "gs1", 0, False)
    out = []
    for calls in ([600], [256, 344], [1] * 3 + [597]):
        s = fea.CUDASolver(xyz, tri, boundary_condition=1, params=p)
        s.set_fields(u, v)
        for n in calls:
            s.advance_time(n)
            assert s.status().steps_done == n
        out.append((s.get_fields(), s.status().total_iterations))
    for o in out[1:]:
        assert np.array_equal(o[0][0], out[0][0][0]) and np.array_equal(o[0][1], out[0][0][1])
        assert o[1] == out[0][1]


def test_stops_on_blow_up(fea):
    """A state above 1e4 stops the stepping in every block, as the step graph does."""
    xyz, tri = mg.cylinder(60, 60)
    u = np.ones(len(xyz), np.float32)
    u[1234] = 2e4
    a, b = _both(fea, xyz, tri, 1, 0, _params(fea, "heat", 0, False), 300, (u, u), calls=1)
    assert a[2] == b[2] and a[3] == b[3] == 0
    assert np.array_equal(a[0][0], b[0][0])


def test_iteration_limit_and_zero_field(fea):
    xyz, tri = mg.cylinder(40, 30)
    p = _params(fea, "heat", 0, False)
    p.cg_max_iterations = 2
    p.cg_tolerance = 1e-12
    u = np.random.default_rng(0).uniform(size=len(xyz)).astype(np.float32)
    a, b = _both(fea, xyz, tri, 1, 0, p, 2, (u, u))
    assert a[1] == b[1] and a[2] == b[2] == 4
    assert rel_l2(b[0][0], a[0][0]) < 1e-6
    a, b = _both(fea, xyz, tri, 1, 0, _params(fea, "gs0", 0, False), 2, (u, 0 * u))
    assert rel_l2(b[0][0], a[0][0]) < 1e-5 and np.all(b[0][1] == 0) and np.all(a[0][1] == 0)


def test_handles_on_several_threads(fea):
    """Handles stepped at once from threads of their own (one block, a cluster, two
    device-wide grids and the step graph) give what each gives alone."""
    shapes = [(10, 10, 0, "heat"), (64, 60, 0, "gs1"), (128, 129, 1, "heat"), (251, 251, 0, "gs1"), (251, 251, 0, "heat")]
    handles, fields = [], []
    for nx, ny, prec, eq in shapes:
        xyz, tri = mg.cylinder(nx, ny)
        handles.append(fea.CUDASolver(xyz, tri, boundary_condition=1, precision=prec, params=_params(fea, eq, prec, False)))
        w = np.random.default_rng(nx).uniform(size=(2, len(xyz)))
        fields.append(np.stack([1 - 0.5 * w[0], 0.25 * w[1]]).astype(np.float32))
    handles[-1].set_cg_variant(14)

    def work(i, out):
        s = handles[i]
        s.clear_values()
        s.set_fields(*fields[i])
        for _ in range(5):
            s.advance_time(4)
        st = s.status()
        out[i] = (s.get_fields(), st.flags, st.steps_done)

    alone, together = {}, {}
    for i in range(len(shapes)):
        work(i, alone)
    threads = [threading.Thread(target=work, args=(i, together)) for i in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(len(shapes)):
        assert together[i][1:] == alone[i][1:] == (0, 4)
        assert all(np.array_equal(a, b) for a, b in zip(together[i][0], alone[i][0]))
