"""Where the axis-aligned class ends: meshes with diagonal metrics whose normals are not along
the axes keep the general flux, in solver and pool; elements so thin that rounding turns
their normals are axis-aligned in both, with the same bits.

Bound: 1e-12 against the oracle as in the other parity tests (rounding and FMA contraction
only)."""
import numpy as np
import pytest

from nekwave_b200 import DgSolver
from nekwave_b200.pool import CavityPool
from oracle import oracle as O
from tests.gpu_helpers import random_state, rel_l2, solver_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", range(2, 11))
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_pool_computes_normals_off_the_axes(gpu, N, mode, precision):
    """Turned by 0.1: not rounding.  Beside it an ordinary cavity of the same order, whose
    bits do not change, and the oblique one again after the first was removed."""
    m = O.box_mesh(N, (3, 2, 2), (0, 0, 0), (1, 1, 1))
    t = 0.1
    m.nx, m.ny = np.cos(t) * m.nx - np.sin(t) * m.ny, np.sin(t) * m.nx + np.cos(t) * m.ny
    dt = 0.1 * O.dxmin(m)
    u = random_state(m, N)
    want = O.step(m, 1.0, dt, 3, u)[0]
    pulses = [(0.5 + 0.1 * c, 0.3, 0.4, 0.5, 0.2) for c in range(6)]
    alone = CavityPool(64 << 20, max_slots=1, precision=precision)
    alone.set_mode(mode)
    alone.init_pulse(alone.add_box(N, (3, 2, 2), (0, 0, 0), (1, 1, 1), 1.0, dt, 3), pulses)
    alone.step(3)
    plain = alone.results(0, energy=False, probes=False)["state"]
    alone.close()
    keep = solver_for(m, 1.0)
    pool = CavityPool(256 << 20, max_slots=3, precision=precision)
    pool.set_mode(mode)
    a = pool.add(keep._keep_mesh, 1.0, dt, 3)
    pool.upload(a, u)
    pool.step(3)  # alone: no ordinary tile of its order
    assert rel_l2(pool.results(a)["state"], want) < 1e-12
    b = pool.add_box(N, (3, 2, 2), (0, 0, 0), (1, 1, 1), 1.0, dt, 3)
    for again in range(2):
        pool.init_pulse(b, pulses)
        pool.upload(a, u)
        pool.step(3)
        r = pool.results(a, probes=False)
        assert rel_l2(r["state"], want) < 1e-12 and np.all(np.isfinite(r["energy"]))
        np.testing.assert_array_equal(pool.results(b, energy=False, probes=False)["state"], plain)
        pool.remove(a)
        a = pool.add(keep._keep_mesh, 1.0, dt, 3)
    pool.close()
    keep.finalize()


@pytest.mark.parametrize("N", [3, 5, 6, 8, 10])
@pytest.mark.parametrize("height", [1e-5, 1e-6])
def test_thin_elements_are_axis_aligned_in_solver_and_pool(gpu, N, height):
    lo, hi, nel = (100.0, -300.0, 200.0), (1100.0, 900.0, 200.0 + 1000.0 * height), (3, 2, 2)
    m = O.box_mesh(N, nel, lo, hi)
    u = random_state(m, N)
    dt = 0.1 * O.dxmin(m)
    s = DgSolver("fp64")
    s.initializeBox(N, nel, lo, hi, 1.0)
    assert s.info()["geometry"] == 0
    s.uploadState(u)
    s.steps(dt, 3)
    pool = CavityPool(64 << 20, max_slots=1)
    q = pool.add_box(N, nel, lo, hi, 1.0, dt, 3)
    pool.upload(q, u)
    pool.step(3)
    np.testing.assert_array_equal(pool.results(q)["state"], s.downloadState())
    pool.close()
    s.finalize()
