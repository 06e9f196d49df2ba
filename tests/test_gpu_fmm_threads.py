"""Fast-multipole applications of low and high order on several threads at once,
each with its own session: the kernels, and their shared-memory limits, are
common to all of them. Every result is bitwise that of a thread alone (the sums
have a fixed order)."""
import threading

import numpy as np
import pytest

import hornsculpt_b200 as hs
from hornsculpt_b200 import meshes

pytestmark = pytest.mark.gpu


def test_orders_of_other_threads_do_not_matter():
    mesh = meshes.icosphere(3)
    rng = np.random.default_rng(2)
    p = rng.normal(size=mesh.vertex_count) + 1j * rng.normal(size=mesh.vertex_count)
    settings = [(5.0, 1e-3), (5.0, 1e-12)]  # orders 5 and 17: every kernel at two sizes of shared memory
    failures = []

    def work(k, tolerance, want, rounds):
        try:
            with hs.CudaBemSolver(mesh) as solver:
                for _ in range(rounds):
                    far = solver.debug_fmm_far(hs.BemNumerics(), k, tolerance, p)[0]
                    if want is None:
                        return far
                    assert np.array_equal(far, want)
        except Exception as error:  # reported by the main thread
            failures.append(error)

    alone = [work(k, tolerance, None, 1) for k, tolerance in settings]
    assert not failures
    threads = [threading.Thread(target=work, args=(*settings[i % 2], alone[i % 2], 150)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
