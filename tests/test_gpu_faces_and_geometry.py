"""The reduced faces of axis-aligned elements, the launch shapes of the general
geometry classes and the LSRK register's skipped accesses, against the oracle.

Bounds: FP64 right-hand sides to 1e-12 of the largest value and states after a few
steps to 1e-12 in relative L2, as in the other parity tests (the kernels differ from the
oracle by rounding and by FMA contraction only)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_helpers import random_state, rel_l2, rel_max, solver_for

from nekwave_b200 import DgSolver
from nekwave_b200.pool import CavityPool

pytestmark = pytest.mark.gpu


def half_turned_box(N, nel):
    """A box mesh whose every other element is turned 180 degrees about z: still
    axis-aligned (negative metrics), but its faces meet with reversed points."""
    corners, fk, fb, ff = O.box_corners(nel, (0, 0, 0), (1.0, 1.2, 0.8), (False, False, False))
    turned = np.arange(corners.shape[0]) % 2 == 1
    face = np.array([2, 3, 0, 1, 4, 5])
    c2, fk2, fb2, ff2 = corners.copy(), fk.copy(), fb.copy(), ff.copy()
    for e in np.nonzero(turned)[0]:
        c2[e] = corners[e][[2, 3, 0, 1, 6, 7, 4, 5]]
        fk2[e, face] = fk[e]
        fb2[e, face] = fb[e]
        ff2[e, face] = ff[e]
    has = fb2 >= 0
    nb = np.zeros_like(has)
    nb[has] = turned[fb2[has]]
    ff2[nb] = face[ff2[nb]]
    return O.hex_mesh(N, c2, fk2, fb2, ff2)


@pytest.mark.parametrize("N", range(2, 11))
def test_half_turned_elements(gpu, N):
    m = half_turned_box(N, (3, 2, 3))
    s = solver_for(m, 0.7)
    assert s.info()["geometry"] == 0 and s.info()["structured"] == (0, 0, 0)
    u = random_state(m, N)
    for v in range(s.info()["variant_count"]):
        s.setVariant(v)
        s.uploadState(u)
        assert rel_max(s.evalRhs(), O.rhs(m, 0.7, u)) < 1e-12, v
    s.finalize()


@pytest.mark.parametrize("N", [3, 6, 8])
def test_normals_off_the_axes_leave_the_axis_aligned_class(gpu, N):
    """Axis-aligned metrics with normals that are not: the general flux applies."""
    m = O.box_mesh(N, (2, 2, 2), (0, 0, 0), (1, 1, 1))
    t = 0.1
    m.nx, m.ny = np.cos(t) * m.nx - np.sin(t) * m.ny, np.sin(t) * m.nx + np.cos(t) * m.ny
    s = solver_for(m, 1.0)
    assert s.info()["geometry"] == 1
    u = random_state(m, N)
    s.uploadState(u)
    assert rel_max(s.evalRhs(), O.rhs(m, 1.0, u)) < 1e-12
    s.finalize()


def test_pool_takes_normals_off_the_axes_by_rounding(gpu):
    """1e-11 moves one right-hand side by about as much relative to its largest entry."""
    m = O.box_mesh(4, (2, 2, 2), (0, 0, 0), (1, 1, 1))
    t = 1e-11
    m.nx, m.ny = m.nx - t * m.ny, t * m.nx + m.ny
    dt = 0.1 * O.dxmin(m)
    u = random_state(m, 4)
    pool = CavityPool(64 << 20, max_slots=2)
    s = pool.add(solver_for(m, 1.0)._keep_mesh, 1.0, dt, 3)
    pool.upload(s, u)
    pool.step(3)
    assert rel_l2(pool.results(s, energy=False, probes=False)["state"], O.step(m, 1.0, dt, 3, u)[0]) < 1e-9
    pool.close()


@pytest.mark.parametrize("N", range(2, 11))
@pytest.mark.parametrize("kind", ["affine", "nodal"])
def test_general_shapes_with_ragged_tiles(gpu, N, kind):
    nel = (5, 3, 3)  # 45 elements: a partial last tile for every shape of several elements
    if kind == "affine":
        m = O.warped_box_mesh(N, nel, linear=[[1.0, 0.3, 0.1], [-0.2, 1.1, 0.05], [0.1, 0.2, 0.9]])
    else:
        m = O.warped_box_mesh(N, nel, warp=0.04)
    s = solver_for(m, 1.0)
    assert s.info()["geometry"] == (1 if kind == "affine" else 2)
    u = random_state(m, N)
    s.uploadState(u)
    assert rel_max(s.evalRhs(), O.rhs(m, 1.0, u)) < 1e-12
    dt = 0.1 * O.dxmin(m)
    s.steps(dt, 3)
    assert rel_l2(s.downloadState(), O.step(m, 1.0, dt, 3, u)[0]) < 1e-12
    s.finalize()


@pytest.mark.parametrize("N", range(2, 11))
@pytest.mark.parametrize("warp", [0.0, 0.04])
def test_the_register_of_an_earlier_run_does_not_enter_a_step(gpu, N, warp):
    """The first stage of a step multiplies the register by zero; it is not read, so what
    an earlier state left there (here NaN) does not matter."""
    m = O.warped_box_mesh(N, (2, 3, 2), warp=warp) if warp else O.box_mesh(N, (2, 3, 2), (0, 0, 0), (1, 1, 1))
    dt = 0.1 * O.dxmin(m)
    u = random_state(m, N)
    s = solver_for(m, 1.0)
    s.uploadState(np.full_like(u, np.nan))
    s.steps(dt, 2)
    s.uploadState(u)
    assert rel_max(s.evalRhs(), O.rhs(m, 1.0, u)) < 1e-12
    s.uploadState(np.full_like(u, np.nan))
    s.step(dt)
    s.uploadState(u)
    s.steps(dt, 2)
    assert rel_l2(s.downloadState(), O.step(m, 1.0, dt, 2, u)[0]) < 1e-12
    s.finalize()


# elements up to which an order takes the shapes for few elements, and a size beyond it
LARGE = {2: (13, 12, 12), 3: (13, 13, 13), 4: (5, 4, 3), 5: (19, 18, 18), 6: (15, 14, 15), 7: (7, 7, 7),
         8: (5, 4, 3), 9: (6, 5, 5), 10: (11, 11, 10)}


@pytest.mark.parametrize("N", range(2, 11))
def test_few_and_many_elements_give_a_cavity_the_same_bits(gpu, N):
    """The launch shape follows the number of elements of an order (single solver: of its
    mesh; pool: of all its cavities).  A small cavity alone, in a pool of its own (shapes
    for few elements) and beside a large one (the other shape) ends in the same bits."""
    small, dt = (3, 2, 2), 1e-3
    pulses = [(0.5 + 0.1 * c, 0.3, 0.4, 0.5, 0.2) for c in range(6)]
    s = DgSolver("fp64")
    s.initializeBox(N, small, (0, 0, 0), (1, 1, 1), 1.0)
    s.initPulse(pulses)
    s.steps(dt, 3)
    want = s.downloadState()
    s.finalize()
    for nels in ([small], [small, LARGE[N]], [LARGE[N], small]):
        pool = CavityPool(1 << 30, max_slots=4)
        slots = [pool.add_box(N, nel, (0, 0, 0), (1, 1, 1), 1.0, dt, 3) for nel in nels]
        for q in slots:
            pool.init_pulse(q, pulses)
        pool.step(3)
        np.testing.assert_array_equal(pool.results(slots[nels.index(small)])["state"], want)
        if LARGE[N] in nels:
            s = DgSolver("fp64")
            s.initializeBox(N, LARGE[N], (0, 0, 0), (1, 1, 1), 1.0)
            s.initPulse(pulses)
            s.steps(dt, 3)
            np.testing.assert_array_equal(pool.results(slots[nels.index(LARGE[N])])["state"], s.downloadState())
            s.finalize()
        pool.close()


@pytest.mark.parametrize("periodic", [(True, True, True), (True, False, True), (False, False, False)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_pool_and_solver_find_the_same_neighbours(gpu, periodic, precision):
    """Boxes one element wide, periodic and closed, structured in solver and pool: the same bits."""
    pulses = [(1.0 - 0.2 * c, 0.4, 0.6, 0.5, 0.2 + 0.05 * c) for c in range(6)]
    boxes = [(N, nel) for N in (3, 4, 6, 8, 9) for nel in ((1, 1, 1), (1, 3, 2), (2, 1, 5), (3, 2, 1))]
    pool = CavityPool(256 << 20, max_slots=len(boxes), precision=precision)
    slots = [pool.add_box(N, nel, (0, 0, 0), (1, 1, 1), 1.0, 1e-3, 3, periodic=periodic) for N, nel in boxes]
    for q in slots:
        pool.init_pulse(q, pulses)
    pool.step(3)
    for q, (N, nel) in zip(slots, boxes):
        s = DgSolver(precision)
        s.initializeBox(N, nel, (0, 0, 0), (1, 1, 1), 1.0, periodic=periodic)
        s.initPulse(pulses)
        s.steps(1e-3, 3)
        np.testing.assert_array_equal(pool.results(q, energy=False, probes=False)["state"], s.downloadState())
        s.finalize()
    pool.close()


def test_pool_takes_a_table_that_is_no_structured_box(gpu):
    m = half_turned_box(5, (3, 2, 2))
    dt = 0.1 * O.dxmin(m)
    u = random_state(m, 5)
    pool = CavityPool(64 << 20, max_slots=2)
    s = pool.add(solver_for(m, 1.0)._keep_mesh, 1.0, dt, 3)
    pool.upload(s, u)
    pool.step(3)
    assert rel_l2(pool.results(s, energy=False, probes=False)["state"], O.step(m, 1.0, dt, 3, u)[0]) < 1e-12
    pool.close()
