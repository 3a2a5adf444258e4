"""Meshes whose stiff groups widen the tiles (csrc/stiff.cu, tile_ell.cu).

The rows of A' = Q^T A Q are longer than A's.  Where they do not fit a ring
variant's stages, that variant runs without the groups: the groups never cost
a mesh its kernel, and no variant is refused for them.
"""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_stiff import flattened

pytestmark = pytest.mark.gpu


# (grid, every k-th cell of the first m x m flattened): FP64 rows past three stages, past four
@pytest.mark.parametrize("n,k,m", [(68, 2, 24), (130, 2, 40), (68, 3, 40), (68, 5, 64)])
@pytest.mark.parametrize("prec", [0, 1])
def test_dense_groups_keep_the_ring_variants(fea, n, k, m, prec):
    cells = [(j, i) for j in range(2, min(m, n - 3), k) for i in range(2, min(m, n - 3), k)]
    xyz, tri = flattened(n, 0.02, cells)
    u = np.random.default_rng(4).uniform(0, 1, len(xyz)).astype(np.float32)
    out = {}
    for variant in (None, 11, 14, 15, "autotune"):
        p = fea.default_params(equation=fea.HEAT, heat_time_step=1e-3, heat_conductivity=1.0,
                               cg_tolerance=1e-10 if prec else 1e-7)
        s = fea.CUDASolver(xyz, tri, boundary_condition=fea.NEUMANN, precision=prec, params=p)
        assert s.info.rows_per_warp_lanes == 14
        if variant == "autotune":
            s.autotune()
        elif variant:
            s.set_cg_variant(variant)
            assert s.time_spmv(reps=1) > 0
        s.set_values(u)
        s.advance_time(2)
        assert s.status().flags == 0
        out[variant] = s.get_values()
    for v in out.values():  # solves to 1e-10 in float32 node values, to 1e-7
        assert rel_l2(v, out[11]) < (1e-7 if prec else 1e-5)
