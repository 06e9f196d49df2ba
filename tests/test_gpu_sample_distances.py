"""Pressure samples from the source to where its panels are one point and k r
leaves the range of the short sine and cosine. Within 1e10 m the pressure falls
as 1 / r. From 1e20 m on every rule point of every panel has the same distance,
an axis coordinate, to the last bit: the rules agree, the sample is in the air,
and its modulus is that of the panels' integrals in plain FP64 (a thousand
roundings of their sum)."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu
FREQUENCY = 1500.0


def test_samples_at_every_distance():
    mesh = meshes.icosphere(2)
    k = 2 * np.pi * FREQUENCY / 343.0
    rng = np.random.default_rng(6)
    corner = mesh.vertices[mesh.triangles]
    trace = np.exp(3j * mesh.vertices[:, 0]) + 0.3
    slope = rng.normal(size=mesh.triangle_count) + 1j * rng.normal(size=mesh.triangle_count)
    solution = hs.BemExcitationResult("u", np.zeros(0), [], 0, 0.0, 0, 0, 0.0,
                                      hs.BemBoundaryData(trace[mesh.triangles].mean(1), trace, slope))
    axes = np.concatenate([np.eye(3), -np.eye(3)])
    near, far = [1e3, 1e6, 1e8, 1e10], [1e20, 1e40, 1e100]
    with hs.CudaBemSolver(mesh) as solver:
        at = {r: solver.pressure_field(FREQUENCY, solution, r * axes) for r in near + far}
    for r in near + far:
        assert all(s.status == hs.FieldPointStatus.AIR for s in at[r]), r
    modulus = {r: np.array([abs(s.pressure) * r for s in at[r]]) for r in at}
    for r in near[1:]:  # 1/r up to 0.1 m / r of the next order, and the phase's spacing of k r
        assert np.max(np.abs(modulus[r] / modulus[near[0]] - 1)) <= 2e-2
    cross = np.cross(corner[:, 1] - corner[:, 0], corner[:, 2] - corner[:, 0])
    area = np.linalg.norm(cross, axis=1) / 2
    projected = axes @ (cross / 2).T  # (x - y) . n / r, times the area
    want = np.abs(projected @ (1j * k * trace[mesh.triangles].mean(1)) - area @ slope) / (4 * np.pi)
    for r in far:
        assert np.max(np.abs(modulus[r] - want)) <= 1e-13 * np.max(want)


def test_a_distant_point_changes_no_other():
    """The samples of a call with a point beyond the short functions' range equal those of a call without."""
    mesh = meshes.icosphere(2)
    trace = np.exp(3j * mesh.vertices[:, 0]) + 0.3
    solution = hs.BemExcitationResult("u", np.zeros(0), [], 0, 0.0, 0, 0, 0.0,
                                      hs.BemBoundaryData(trace[mesh.triangles].mean(1), trace,
                                                         np.full(mesh.triangle_count, 1.0 - 2.0j)))
    points = np.random.default_rng(8).normal(size=(65, 3))
    with hs.CudaBemSolver(mesh) as solver:
        alone = solver.pressure_field(FREQUENCY, solution, points)
        mixed = solver.pressure_field(FREQUENCY, solution, np.concatenate([points, [[1e30, 0.0, 0.0]]]))
    assert alone == mixed[:65] and mixed[65].status == hs.FieldPointStatus.AIR
