"""Pressure samples are linear in the traces: amplitudes scaled by a power of two
give the same statuses and pressures scaled by it, bit for bit, as far as the
traces and pressures themselves are normal numbers. The test points run from
3 mm off the surface, where panels are divided, to far away."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-900, -540, -500, -100, 100, 490, 900])
def test_amplitudes_do_not_matter(exponent):
    mesh = meshes.icosphere(2)
    rng = np.random.default_rng(6)
    trace = np.exp(3j * mesh.vertices[:, 0] / 0.1) + 0.3
    slope = rng.normal(size=mesh.triangle_count) + 1j * rng.normal(size=mesh.triangle_count)
    direction = rng.normal(size=(200, 3))
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    points = direction * 0.1 * (1 + np.geomspace(0.03, 1e4, 200))[:, None]

    def samples(solver, unit):
        solution = hs.BemExcitationResult("u", np.zeros(0), [], 0, 0.0, 0, 0, 0.0,
                                          hs.BemBoundaryData(unit * trace[mesh.triangles].mean(1), unit * trace,
                                                             unit * slope))
        found = solver.pressure_field(1500.0, solution, points)
        return np.array([int(s.status) for s in found]), np.array([s.pressure for s in found])

    with hs.CudaBemSolver(mesh) as solver:
        status, pressure = samples(solver, 1.0)
        scaled_status, scaled = samples(solver, 2.0 ** exponent)
    assert (status == int(hs.FieldPointStatus.AIR)).sum() > 150
    assert np.array_equal(scaled_status, status)
    assert np.array_equal(scaled, pressure * 2.0 ** exponent)
