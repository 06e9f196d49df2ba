"""FP64 touching pairs at the smallest singular orders, an odd one and a large
one: the tabulated tuples and the warp's split of them over its lanes depend on
the order. Entry by entry against the oracle's FP64 assembly, to the tolerance
of the assembly parity (1e-12 of the largest entry)."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 3, 7, 16])
def test_touching_pairs_at_every_kind_of_order(order):
    mesh = meshes.octahedral_sphere(1)
    k = 2 * np.pi * 900.0 / 343.0
    q = np.linspace(1.0, 2.0, mesh.triangle_count) * (1 + 0.5j)
    with hs.CudaBemSolver(mesh) as solver:
        A, b = solver.debug_assemble(hs.BemNumerics(singular_order=order), k, k, q)
    Ao, bo = O.assemble(mesh, O.Numerics.default(singular_order=order), k, k, q)
    assert np.max(np.abs(A - Ao)) <= 1e-12 * np.max(np.abs(Ao))
    assert np.max(np.abs(b - bo)) <= 1e-12 * np.max(np.abs(bo))
