"""Far fields about an origin so far away that the phases leave the range of the
short sine and cosine. The mesh lies below the spacing of doubles there, so every
panel has the same phase, k times a power of two, in the kernel of many directions
as in the per-output kernel: both give the same values. (Between 2^25 and 2^53
the rounded phases differ from panel to panel, and the field's rules do not agree.)"""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [20, 60, 90])
def test_a_distant_origin(exponent):
    mesh = meshes.octahedral_sphere(3)
    axes = np.concatenate([np.eye(3), -np.eye(3)])
    distance = 2.0 ** exponent

    def solve(solver, where):
        request = hs.BemRequest(frequencies=[500.0, 1700.0], observers=where,
                                excitations=[hs.BemExcitation("u", [hs.FaceVelocity(1, 1.0 + 0.5j)])],
                                far_field=hs.FarFieldObservation((distance, distance, distance), 1.0))
        return np.array([f.excitations[0].observer_pressure for f in solver.solve(request).frequencies])

    with hs.CudaBemSolver(mesh) as solver:
        where = distance + distance * axes  # observers one distance from the origin along its axes
        few, many = solve(solver, where), solve(solver, np.tile(where, (40, 1)))
    # nearer than 2^53 the kernels round a point's position (up to one spacing of its phase) and its phase
    # (half a spacing in one, twice half in the other) differently
    phase = 2 * np.pi * 1700.0 / 343.0 * distance
    bound = 1e-13 + (4 * np.spacing(phase) if exponent < 53 else 0.0)
    assert np.max(np.abs(many - np.tile(few, 40))) <= bound * np.max(np.abs(few))
    assert np.all(np.isfinite(many)) and np.max(np.abs(many)) > 0
