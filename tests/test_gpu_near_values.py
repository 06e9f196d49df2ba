"""Near-field values of the fast-multipole form with near lists of one tile and
of several (2048 trial panels a tile): a solve with large leaves, whose near
lists pass 2048 panels on this mesh, meets the dense solution like one with the
usual leaves. The solves stop at a relative residual of 1e-7; the equilibrated
Burton-Miller system of a sphere has a condition number below a hundred."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity,precision", [(16, "fp64"), (256, "fp64"), (256, "mixed")])
def test_large_leaves_match_the_dense_solution(capacity, precision):
    mesh = meshes.icosphere(4)

    def solve(acceleration, form):
        numerics = hs.BemNumerics(acceleration=acceleration, precision=form, relative_residual_tolerance=1e-7,
                                  fast_multipole=hs.FastMultipoleSettings(leaf_support_capacity=capacity))
        with hs.CudaBemSolver(mesh) as solver:
            r = solver.solve(hs.BemRequest(frequencies=[900.0], numerics=numerics,
                                           excitations=[hs.BemExcitation("u", [hs.FaceVelocity(1, 1.0)])]))
        return r.frequencies[0].excitations[0].boundary.pressure_trace

    dense, fast = solve("dense", "fp64"), solve("fast_multipole", precision)
    assert np.linalg.norm(fast - dense) <= 1e-5 * np.linalg.norm(dense)
