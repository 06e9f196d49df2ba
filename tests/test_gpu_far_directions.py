"""Far-field directions by the many-direction kernel (32 directions on) against
the per-output kernel, which serves fewer: the same directions of one request
asked for in small groups. Both sum the same rule points in FP64 in another
order, so they agree to a few hundred roundings of the largest value."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


def _cabinet(drivers):
    base = meshes.icosphere(2)  # 320 triangles: two panel tiles, the second one partial
    faces = 1 + np.arange(base.triangle_count) % drivers
    return meshes.SurfaceMesh(base.vertices, base.triangles, faces, base.boundary)


# edges of the direction blocks (64) and of the excitation pairs; frequencies reach the rules of 6, 12, 16 and 49 points
@pytest.mark.parametrize("directions,drivers", [(32, 1), (63, 2), (65, 3), (129, 1)])
def test_many_directions_match_few(directions, drivers):
    mesh = _cabinet(drivers)
    rng = np.random.default_rng(directions)
    where = rng.normal(size=(directions, 3)) + [0.0, 0.0, 0.2]

    def request(points):
        return hs.BemRequest(frequencies=[300.0, 1500.0, 3200.0], observers=points,
                             excitations=[hs.BemExcitation(f"d{d}", [hs.FaceVelocity(d + 1, 1.0 - 0.3j * d)])
                                          for d in range(drivers)],
                             far_field=hs.FarFieldObservation((0.01, -0.02, 0.03), 2.0))

    with hs.CudaBemSolver(mesh) as solver:
        many = solver.solve(request(where))
        few = [solver.solve(request(where[i:i + 16])) for i in range(0, directions, 16)]
    for f in range(3):
        for e in range(drivers):
            got = many.frequencies[f].excitations[e].observer_pressure
            want = np.concatenate([r.frequencies[f].excitations[e].observer_pressure for r in few])
            assert got.shape == (directions,)
            assert np.max(np.abs(got - want)) <= 1e-13 * np.max(np.abs(want))
