"""FP64 M2L as matrix products at the order where its tile shape changes (15 to
16 at every level: below k r = 1 the order is ceil(1.3 d) + 1 for d digits)
against the per-target translations. Both use the same tables, so they differ by
rounding alone, which has to stay below the truncation the orders stand for."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("digits,order", [(10.7, 15), (11.5, 16)])
def test_matrix_m2l_where_its_tiles_change(digits, order):
    mesh = meshes.icosphere(3)
    rng = np.random.default_rng(order)
    p = rng.normal(size=mesh.vertex_count) + 1j * rng.normal(size=mesh.vertex_count)
    numerics, k, tolerance = hs.BemNumerics(), 5.0, 10.0 ** -digits
    with hs.CudaBemSolver(mesh) as solver:
        grouped, _, _, levels = solver.debug_fmm_far(numerics, k, tolerance, p)
        solver.set_fmm_grouped_m2l(False)
        per_target, _, _, _ = solver.debug_fmm_far(numerics, k, tolerance, p)
    assert len(levels) and (levels[:, 1] == order).all()
    assert np.linalg.norm(grouped - per_target) < tolerance * np.linalg.norm(per_target)
