"""Meshes of few elements take another launch shape as variant 0.  Every shape keeps a number
there, the large default too, and the sizes between the lines give the same bits."""
import numpy as np
import pytest

from nekwave_b200 import DgSolver
from nekwave_b200.pool import CavityPool
from oracle import oracle as O
from tests.gpu_helpers import random_state, rel_l2, rel_max, solver_for

pytestmark = pytest.mark.gpu

# more elements than the last line of each order (NWB_SMALL)
LARGE = {2: (13, 12, 12), 3: (13, 13, 13), 4: (3, 2, 2), 5: (19, 18, 18), 6: (15, 14, 15), 7: (7, 7, 7),
         8: (3, 2, 2), 9: (6, 5, 5), 10: (11, 11, 10)}


def shapes(N, nel):
    s = DgSolver("fp64")
    s.initializeBox(N, nel, (0, 0, 0), (1, 1, 1), 1.0)
    out = []
    for v in range(s.info()["variant_count"]):
        s.setVariant(v)
        i = s.info()
        out.append(tuple(i[k] for k in ("ks", "epb", "threads_per_block", "smem_bytes", "ksmem", "minb")))
    s.finalize()
    return out


@pytest.mark.parametrize("N", range(2, 11))
def test_every_shape_has_a_number_on_small_and_large_meshes(gpu, N):
    small, large = shapes(N, (2, 2, 2)), shapes(N, LARGE[N])
    assert sorted(small) == sorted(large)
    assert large[0] in small and small[0] in large


@pytest.mark.parametrize("N,nel", [(2, (13, 12, 12)), (3, (13, 13, 13)), (5, (20, 18, 17)), (10, (11, 11, 10))])
def test_default_shape_beyond_the_line(gpu, N, nel):
    """The large default of the orders whose other tests stay below the line, against the
    oracle (bounds as in the other parity tests: rounding and FMA contraction only)."""
    m = O.box_mesh(N, nel, (0, 0, 0), (1, 1.5, 1), (True, False, False))
    s = solver_for(m, 1.0)
    u = random_state(m, 11)
    s.uploadState(u)
    assert rel_max(s.evalRhs(), O.rhs(m, 1.0, u)) < 1e-12
    dt = 0.1 * O.dxmin(m)
    s.steps(dt, 2)
    assert rel_l2(s.downloadState(), O.step(m, 1.0, dt, 2, u)[0]) < 1e-12
    s.finalize()


@pytest.mark.parametrize("nel", [(6, 7, 7), (7, 7, 7), (14, 15, 14)])
def test_six_point_pools_on_both_sides_of_the_first_line(gpu, nel):
    """6 points has two lines (296 and 2960 elements): 294, 343 and 2940 elements with a small
    cavity beside them, each as alone bit for bit."""
    pulses = [(0.5 + 0.1 * c, 0.3, 0.4, 0.5, 0.2) for c in range(6)]
    nels, dt = [nel, (2, 1, 1)], 1e-3
    pool = CavityPool(1 << 30, max_slots=2)
    slots = [pool.add_box(6, n, (0, 0, 0), (1, 1, 1), 1.0, dt, 3) for n in nels]
    for q in slots:
        pool.init_pulse(q, pulses)
    pool.step(3)
    for q, n in zip(slots, nels):
        s = DgSolver("fp64")
        s.initializeBox(6, n, (0, 0, 0), (1, 1, 1), 1.0)
        s.initPulse(pulses)
        s.steps(dt, 3)
        np.testing.assert_array_equal(pool.results(q, energy=False, probes=False)["state"], s.downloadState())
        s.finalize()
    pool.close()
