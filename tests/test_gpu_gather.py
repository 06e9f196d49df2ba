"""Dense matrices of meshes whose columns are gathered in two passes (above
4266 triangles): every remainder of the vertex count by the four columns a
thread takes, and a mesh above 10,000 triangles, whose rule bins are counted
before they are filled. The dense solution meets the fast-multipole one, which
uses neither gather. The iterative solves stop at a relative residual of 1e-7
and the equilibrated Burton-Miller system of a sphere has a condition number
below a hundred: 1e-5, and 3e-5 more where the samples are FP32 (6e-8, a few of
them, times that condition number)."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,remainder,precision", [(.0076, 0, "fp64"), (.0074, 1, "fp64"), (.0074, 1, "mixed"),
                                                   (.00745, 2, "fp64"), (.005, 3, "fp64"), (.005, 3, "mixed")])
def test_two_pass_gather_meets_the_fast_multipole_solution(h, remainder, precision):
    mesh = meshes.revolved_sphere(h=h)
    assert mesh.triangle_count > 4266 and mesh.vertex_count % 4 == remainder

    def solve(acceleration, form):
        numerics = hs.BemNumerics(acceleration=acceleration, precision=form, relative_residual_tolerance=1e-7)
        with hs.CudaBemSolver(mesh) as solver:
            r = solver.solve(hs.BemRequest(frequencies=[900.0], numerics=numerics,
                                           excitations=[hs.BemExcitation("u", [hs.FaceVelocity(1, 1.0)])]))
        return r.frequencies[0].excitations[0].boundary.pressure_trace

    dense, fast = solve("dense", precision), solve("fast_multipole", "fp64")
    bound = 1e-5 if precision == "fp64" else 4e-5
    assert np.linalg.norm(fast - dense) <= bound * np.linalg.norm(dense)
