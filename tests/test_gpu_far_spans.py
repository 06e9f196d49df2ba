"""Far fields of many directions: the kernel that shares a panel's data among
directions runs over spans of 8 to 256 panels, chosen from the sizes. Every span
against the per-output kernel, which serves fewer than 32 directions (the same
rule points in another order: a few hundred roundings of the largest value),
alone and in a batch (bit for bit), and a polar plot's time, which must not be
that of a thread's walk over a whole tile."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


def _request(frequencies, where, drivers, raster=()):
    return hs.BemRequest(frequencies=list(frequencies), observers=where, interaction_plan_frequencies=list(raster),
                         excitations=[hs.BemExcitation(f"d{d}", [hs.FaceVelocity(d + 1, 1.0 - 0.3j * d)])
                                      for d in range(drivers)],
                         far_field=hs.FarFieldObservation((0.01, -0.02, 0.03), 2.0))


def _drivers(base, drivers):
    return meshes.SurfaceMesh(base.vertices, base.triangles, 1 + np.arange(base.triangle_count) % drivers, base.boundary)


def _observed(result):
    return np.array([[e.observer_pressure for e in f.excitations] for f in result.frequencies])


# spans of 8, 8, 16, 32, 64 and 128 panels; the ring meshes' triangle counts are no multiples of them
@pytest.mark.parametrize("mesh,directions,drivers", [
    (lambda: meshes.icosphere(2), 192, 1), (lambda: meshes.icosphere(2), 193, 3),
    (lambda: meshes.revolved_sphere(h=.0145), 1500, 1), (lambda: meshes.revolved_sphere(h=.0145), 2664, 1),
    (lambda: meshes.revolved_sphere(h=.0145), 2600, 3), (lambda: meshes.icosphere(3), 2664, 7)])
def test_spans_match_the_per_output_kernel(mesh, directions, drivers):
    mesh = _drivers(mesh(), drivers)
    rng = np.random.default_rng(directions)
    where = rng.normal(size=(directions, 3)) + [0.0, 0.0, 0.2]
    frequencies = [300.0, 1500.0, 2200.0]
    with hs.CudaBemSolver(mesh) as solver:
        many = _observed(solver.solve(_request(frequencies, where, drivers)))
        for part in (slice(0, 16), slice(56, 72), slice(directions - 16, directions)):
            few = _observed(solver.solve(_request(frequencies, where[part], drivers)))
            assert np.max(np.abs(many[:, :, part] - few)) <= 1e-13 * np.max(np.abs(many))


def test_whole_tiles_of_a_large_mesh():
    """5120 triangles, 2664 directions, three excitations: spans of 256 panels."""
    mesh = _drivers(meshes.icosphere(4), 3)
    where = np.random.default_rng(1).normal(size=(2664, 3))
    with hs.CudaBemSolver(mesh) as solver:
        many = _observed(solver.solve(_request([900.0], where, 3)))
        few = _observed(solver.solve(_request([900.0], where[-16:], 3)))
    assert np.max(np.abs(many[:, :, -16:] - few)) <= 1e-13 * np.max(np.abs(many))


@pytest.mark.parametrize("directions", [72, 720])
def test_a_batch_changes_no_bit(directions):
    mesh = _drivers(meshes.icosphere(3), 2)
    where = np.random.default_rng(directions).normal(size=(directions, 3))
    frequencies = [400.0, 800.0, 1300.0, 1900.0, 2500.0]
    with hs.CudaBemSolver(mesh) as solver:
        together = _observed(solver.solve(_request(frequencies, where, 2, frequencies)))
        alone = [_observed(solver.solve(_request([f], where, 2, frequencies)))[0] for f in frequencies]
    assert np.array_equal(together, np.array(alone))


def test_a_polar_plot_does_not_wait_for_one_thread():
    """80 directions against the 31 of the per-output kernel at one frequency: at most four
    times the device time (2.6 times the outputs); a walk over 256 panels took 23 times."""
    mesh = meshes.icosphere(3)
    where = np.random.default_rng(3).normal(size=(80, 3))

    def milliseconds(solver, count):
        request, times = _request([1500.0], where[:count], 1), []
        for _ in range(7):
            solver.set_profiling(False)
            solver.set_profiling(True)
            solver.solve(request)
            times.append(solver.profile()["field"][0])
        return np.median(times)

    with hs.CudaBemSolver(mesh) as solver:
        solver.solve(_request([1500.0], where, 1))
        assert milliseconds(solver, 80) <= 4 * milliseconds(solver, 31)
