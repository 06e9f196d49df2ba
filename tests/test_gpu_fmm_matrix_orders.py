"""FP64 M2L at the largest order of the matrix form (23) and above it (24, the
scalar form), at the level with most of the links, against the per-target
translations. Both use the same tables, so they differ by rounding alone, which
has to stay below the truncation the orders stand for."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,order", [(100.0, 23), (105.0, 24)])
def test_the_largest_matrix_order(k, order):
    mesh = meshes.icosphere(3)
    rng = np.random.default_rng(order)
    p = rng.normal(size=mesh.vertex_count) + 1j * rng.normal(size=mesh.vertex_count)
    numerics, tolerance = hs.BemNumerics(), 1e-10
    with hs.CudaBemSolver(mesh) as solver:
        solver.set_plane_wave_threshold(1e9)  # every level rotational
        grouped, _, _, levels = solver.debug_fmm_far(numerics, k, tolerance, p)
        solver.set_fmm_grouped_m2l(False)
        per_target, _, _, _ = solver.debug_fmm_far(numerics, k, tolerance, p)
    assert levels[np.argmax(levels[:, 3]), 1] == order
    assert np.linalg.norm(grouped - per_target) < tolerance * np.linalg.norm(per_target)
