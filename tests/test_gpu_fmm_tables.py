"""The fast-multipole operator with its point tables, without them, and where
their allocation fails: then the leaves evaluate their points on the fly, in the
apply that met the failure and in the captured ones after it, and the next
operator has tables again. Table and on-the-fly evaluation differ by rounding,
which has to stay below the truncation the expansion orders stand for."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu
MESH = meshes.icosphere(3)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_application_without_room_for_its_tables(precision):
    rng = np.random.default_rng(4)
    p = rng.normal(size=MESH.vertex_count) + 1j * rng.normal(size=MESH.vertex_count)
    numerics, tolerance = hs.BemNumerics(precision=precision), 1e-6

    with hs.CudaBemSolver(MESH) as solver:
        def far():
            return solver.debug_fmm_far(numerics, 15.0, tolerance, p)[0]

        tables = far()
        solver.debug_fmm_tables(refused=True)
        refused = far()
        solver.debug_fmm_tables(0)
        on_the_fly = far()
        solver.debug_fmm_tables()
        again = far()
    assert np.array_equal(refused, on_the_fly) and np.array_equal(again, tables)
    assert not np.array_equal(tables, on_the_fly)  # two evaluations, not one twice
    assert np.linalg.norm(tables - on_the_fly) < tolerance * np.linalg.norm(on_the_fly)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_solve_without_room_for_its_tables(precision):
    numerics = hs.BemNumerics(acceleration="fast_multipole", precision=precision,
                              fast_multipole=hs.FastMultipoleSettings(leaf_support_capacity=16))
    request = hs.BemRequest(frequencies=[700.0, 900.0], numerics=numerics,
                            excitations=[hs.BemExcitation(n, [hs.FaceVelocity(1, v)]) for n, v in (("a", 1.0), ("b", 1j))])

    def traces(solver):
        return np.array([[e.boundary.pressure_trace for e in f.excitations] for f in solver.solve(request).frequencies])

    with hs.CudaBemSolver(MESH) as solver:
        solver.set_fmm_audit("expansion")  # re-prepared operators and other panel rules on the way
        solver.debug_fmm_tables(0)
        on_the_fly = traces(solver)
        solver.debug_fmm_tables(refused=True)
        assert np.array_equal(traces(solver), on_the_fly)
        solver.debug_fmm_tables()
        tables = traces(solver)
    # both solves stop at the default relative residual; the sphere's condition number is below a hundred
    assert np.linalg.norm(tables - on_the_fly) <= 100 * 2 * hs.BemNumerics().relative_residual_tolerance * np.linalg.norm(tables)
