"""The lists that are read in tiles or filled after counting, with the sizes that
reach those forms asserted: near lists of more than one tile of 2048 trial panels
(the fast-multipole near values) and more than 10,000 triangles (the rule bins of
the dense assembly). The solves stop at a relative residual of 1e-7; the
equilibrated Burton-Miller system of a sphere has a condition number below a
hundred."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu
TILE, COUNTED = 2048, 10000


def _trace(mesh, **numerics):
    with hs.CudaBemSolver(mesh) as solver:
        r = solver.solve(hs.BemRequest(frequencies=[900.0],
                                       numerics=hs.BemNumerics(relative_residual_tolerance=1e-7, **numerics),
                                       excitations=[hs.BemExcitation("u", [hs.FaceVelocity(1, 1.0)])]))
    return r.frequencies[0].excitations[0].boundary.pressure_trace


def _longest_near_list(mesh, settings):
    """A panel's near list holds at least the panels of the vertices near one of its vertices."""
    numerics = hs.BemNumerics(acceleration="fast_multipole", fast_multipole=settings)
    with hs.CudaBemSolver(mesh) as solver:
        _, row, cols, _ = solver.debug_fmm_far(numerics, 1.0, 1e-4, np.ones(mesh.vertex_count))
    near = np.zeros(mesh.vertex_count, bool)
    at = int(np.argmax(np.diff(row.astype(np.int64))))
    near[cols[row[at]:row[at + 1]]] = True
    return int(near[mesh.triangles].any(1).sum())


@pytest.mark.parametrize("capacity,tiles", [(16, 1), (256, 2)])
def test_near_lists_of_one_tile_and_more(capacity, tiles):
    mesh = meshes.icosphere(4)
    settings = hs.FastMultipoleSettings(leaf_support_capacity=capacity)
    longest = _longest_near_list(mesh, settings)
    assert (longest > TILE) == (tiles > 1)
    dense, fast = _trace(mesh), _trace(mesh, acceleration="fast_multipole", fast_multipole=settings)
    assert np.linalg.norm(fast - dense) <= 1e-5 * np.linalg.norm(dense)


def test_counted_bins():
    mesh = meshes.revolved_sphere(h=.005)
    assert mesh.triangle_count > COUNTED
    dense, fast = _trace(mesh), _trace(mesh, acceleration="fast_multipole")
    assert np.linalg.norm(fast - dense) <= 1e-5 * np.linalg.norm(dense)
