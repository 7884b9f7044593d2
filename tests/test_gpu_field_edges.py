"""Outputs at the edges of their launches: problem counts around the groups that
the Kochin and free-surface kernels sum at once, panel counts around their
panel chunks, impulse responses around a CTA's times and pair chunks, and
finite-depth wave terms beyond the tabulated range (k R above 99.7), between
bodies and at field points. Bounds are those of the parity tests of the same
outputs: 1e-9 of a problem's largest value, 1e-12 for the impulse responses."""
import numpy as np
import pytest

import nemoh_b200 as nb
import oracle_lib as O
from nemoh_b200 import cases as C

pytestmark = pytest.mark.gpu


def _both(solver, mesh, depth):
    solver.set_mesh(mesh.nodes, mesh.panels, mesh.isym, 1000.0, 9.81, depth)
    return O.Oracle(mesh.nodes, mesh.panels, mesh.isym, 1000.0, 9.81, depth, cache_s=True)


def _strengths(rng, n, nprob):
    return rng.standard_normal((n, nprob)) + 1j * rng.standard_normal((n, nprob))


@pytest.fixture(scope="module")
def solver():
    with nb.Solver(0, nb.FP64) as s:
        yield s


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("nprob", [1, 2, 7, 8, 9, 15, 16, 17])
def test_problem_counts(solver, half, nprob):
    mesh = C.box_mesh(20.0, 8.0, 4.0, nx=6, ny=2 if half else 4, nz=3, half=half)
    o = _both(solver, mesh, 30.0)
    rng = np.random.default_rng(nprob)
    zigb = _strengths(rng, mesh.npanels, nprob)
    zigs = _strengths(rng, mesh.npanels, nprob) if half else np.zeros_like(zigb)
    theta = np.linspace(0.0, 3.0, 5)
    xy = rng.uniform(-60.0, 60.0, (130, 2))
    for got, want in ((solver.kochin(6.0, theta, zigb, zigs, 0.5, 0.0),
                       o.kochin(6.0, theta, zigb, zigs if half else None, 0.5, 0.0)),
                      (solver.free_surface(6.0, xy, zigb, zigs), o.free_surface(6.0, xy, zigb, zigs))):
        assert (np.abs(got - want) / np.abs(want).max(axis=0)).max() < 1e-9


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129])
def test_panel_counts(solver, n):
    full = C.cylinder_mesh(3.0, 5.0, 16, 6, 4)
    mesh = C.Mesh(full.nodes, full.panels[:n], isym=0)
    o = _both(solver, mesh, 0.0)
    rng = np.random.default_rng(n)
    z = _strengths(rng, n, 3)
    theta = np.linspace(-1.0, 2.0, 4)
    xy = rng.uniform(-40.0, 40.0, (33, 2))
    for got, want in ((solver.kochin(5.0, theta, z), o.kochin(5.0, theta, z)),
                      (solver.free_surface(5.0, xy, z), o.free_surface(5.0, xy, z))):
        assert (np.abs(got - want) / np.abs(want).max(axis=0)).max() < 1e-9


@pytest.mark.parametrize("ntime", [2, 128, 129, 130, 258])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 1, 3), (129, 1, 4), (5, 5, 1)])
def test_impulse_responses(solver, shape, ntime):
    rng = np.random.default_rng(ntime)
    w = np.sort(rng.uniform(0.05, 3.0, shape[0]))
    damping, added = rng.standard_normal(shape), rng.standard_normal(shape) + 2.0
    K, ainf = solver.irf(w, damping, added, ntime, 0.1)
    Ko, ao = O.irf(w, damping, added, ntime, 0.1)
    assert np.abs(K - Ko).max() <= 1e-12 * max(np.abs(Ko).max(), 1e-300)
    assert np.abs(ainf - ao).max() <= 1e-12 * np.abs(ao).max()


@pytest.mark.parametrize("half", [False, True])
def test_far_finite_depth(solver, half):
    """k R on both sides of 99.7 (k = 0.35 1/m, up to 600 m apart)."""
    a = C.box_mesh(20.0, 8.0, 4.0, nx=5, ny=2 if half else 3, nz=2, half=half)
    mesh = C.merge_meshes([a, C.Mesh(a.nodes + np.array([290.0, 0.0, 0.0]), a.panels, a.isym)])
    o = _both(solver, mesh, 50.0)
    w = np.sqrt(9.81 * 0.35)
    T = 2 * np.pi / w
    rng = np.random.default_rng(5)
    nv = rng.standard_normal(mesh.npanels * (2 if half else 1)) + 0j
    got, want = solver.solve_potential(T, nv), o.solve_problem(T, nv)
    assert np.abs(got["zpb"] - want["zpb"]).max() <= 1e-9 * np.abs(want["zpb"]).max()


@pytest.mark.parametrize("half", [False, True])
def test_far_field_points(solver, half):
    """Field points on both sides of k R = 99.7 (k = 0.3 1/m)."""
    mesh = C.box_mesh(20.0, 8.0, 4.0, nx=5, ny=2 if half else 3, nz=2, half=half)
    o = _both(solver, mesh, 50.0)
    rng = np.random.default_rng(6)
    z = _strengths(rng, mesh.npanels, 2)
    zs = _strengths(rng, mesh.npanels, 2) if half else np.zeros_like(z)
    xy = rng.uniform(150.0, 350.0, (200, 2))
    T = 2 * np.pi / np.sqrt(9.81 * 0.3 * np.tanh(15.0))
    got, want = solver.free_surface(T, xy, z, zs), o.free_surface(T, xy, z, zs)
    assert (np.abs(got - want) / np.abs(want).max(axis=0)).max() < 1e-9
