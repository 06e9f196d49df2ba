"""Admission of fast-multipole requests and their point tables (128 KB a
triangle and operator): a serving budget that holds the tables reserves them,
one that does not serves the request without them, so the tables refuse no
request. Either way the result is that of a session with or without tables, bit
for bit: the choice follows from the sizes and the budget."""
import numpy as np
import pytest
import torch

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu
PLAN_HZ = 1000.0


@pytest.mark.parametrize("precision,operators", [("fp64", 1), ("mixed", 2)])
def test_a_budget_without_room_for_the_tables_still_serves(precision, operators):
    mesh = meshes.icosphere(4)
    tables = operators * mesh.triangle_count * 128 * 1024
    numerics = hs.BemNumerics(acceleration="fast_multipole", precision=precision,
                              fast_multipole=hs.FastMultipoleSettings(leaf_support_capacity=16))
    request = hs.BemRequest(frequencies=[900.0], numerics=numerics, interaction_plan_frequencies=[900.0, PLAN_HZ],
                            excitations=[hs.BemExcitation("u", [hs.FaceVelocity(1, 1.0)])])

    def trace(result):
        return result.frequencies[0].excitations[0].boundary.pressure_trace

    def served(fraction):
        with hs.BemServer(hs.ServeOptions(workers=1, memory_fraction=fraction, planning_frequency=PLAN_HZ)) as server:
            result, timing = server.wait(server.submit(mesh, request))
        return trace(result), timing.footprint_bytes

    with hs.CudaBemSolver(mesh) as solver:
        with_tables = trace(solver.solve(request))
        solver.debug_fmm_tables(0)
        without = trace(solver.solve(request))
    assert not np.array_equal(with_tables, without)
    wide, footprint = served(0.6)
    assert np.array_equal(wide, with_tables)
    free, _ = torch.cuda.mem_get_info()
    narrow, small = served((footprint - tables + tables / 16) / free)
    assert small == footprint - tables
    assert np.array_equal(narrow, without)
