"""Precision of the FP64 LU's trailing update on the tensor cores, where the
forces of a hull can't show it: the update alone against exact products, one
entry at a time; sources of whole solves, one entry at a time, against the same
solves with the update on the FP64 pipe; and the routes the update takes
(captured, merged over panel pairs in a ragged batch, left to the FP64 pipe)."""
import ctypes
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import nemoh_b200 as nb
from nemoh_b200 import cases as C

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
EPS = 2.0 ** -53


def _update(a, orders, panels):
    """a: list of square matrices, largest first; the updated matrices."""
    f = nb.load_library().nemoh_b200_diag_fp64_update
    d, i = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, i, ctypes.c_int, d]
    n = len(a[0])
    buf = np.zeros((len(a), n * n), dtype=np.complex128)
    for s, m in enumerate(a):
        buf[s, :m.size] = m.ravel(order="F")
    o = np.array([len(m) for m in a], dtype=np.int32)
    st = f(0, n, len(a), o.ctypes.data_as(i) if orders else None, panels, buf.ctypes.data_as(d))
    assert st == 0
    return [buf[s, :m.size].reshape(m.shape, order="F") for s, m in enumerate(a)]


def _mul(x, y):
    return x.astype(np.clongdouble) @ y.astype(np.clongdouble)


def _scale(x, axis):
    """The power of two above the largest component of each row (axis 1) or column (0)."""
    m = np.maximum(np.abs(x.real), np.abs(x.imag)).max(axis=axis, keepdims=True)
    return np.exp2(np.frexp(m)[1].astype(float))


def _cancelling(rng, n, panels):
    """A matrix whose panels' products almost cancel: column 64 + k of a panel
    repeats column k, row 64 + k is row k negated but for 2^-30 of it. The products
    are so small that FP64 holds them to 2^-53 of a small number, and every digit
    of the operands still counts; rows and columns reach over 2^40."""
    a = np.zeros((n, n), dtype=np.complex128)
    half = lambda *s: rng.uniform(-1, 1, s) + 1j * rng.uniform(-1, 1, s)  # noqa: E731
    for p in range(panels):
        k, r = 128 * p, n - 128 * (p + 1)
        col, row = half(r, 64), half(64, r)
        col *= np.exp2(rng.integers(-20, 20, (r, 1)))
        row *= np.exp2(rng.integers(-20, 20, (1, r)))
        a[k + 128:, k:k + 64] = a[k + 128:, k + 64:k + 128] = col
        a[k:k + 64, k + 128:] = row
        a[k + 64:k + 128, k + 128:] = -row * (1 + rng.uniform(-1, 1, row.shape) * 2.0 ** -30)
    return a


# edges of the 128 x 64 tiles, one and several systems, uniform and ragged
SHAPES = [[129], [130, 130], [191], [192, 192], [193], [255], [256], [257], [320, 320, 320], [385], [500, 130, 129, 90],
          [449, 448, 321, 320, 257, 256, 200]]


@pytest.mark.parametrize("orders", SHAPES, ids=str)
def test_one_update_digit_by_digit(orders):
    rng = np.random.default_rng(sum(orders))
    a = [_cancelling(rng, n, 1) if n > 128 else rng.standard_normal((n, n)) + 0j for n in orders]
    got = _update(a, len(set(orders)) > 1, 1)
    for m, g in zip(a, got):
        assert np.array_equal(g[:128], m[:128]) and np.array_equal(g[:, :128], m[:, :128])
        if len(m) <= 128:
            continue
        L, U = m[128:, :128], m[:128, 128:]
        err = (g[128:, 128:] - (m[128:, 128:] - _mul(L, U))).astype(complex)
        s = _scale(L, 1) * _scale(U, 0)
        # Dropped are the digit products of i + j >= 8: 7 pairs of digits of root mean
        # square 74 (balanced base 256), two real products, 128 k, 2^-76 of the scales a unit:
        # sqrt(7 * 256) 74^2 2^-76 = 2^-58.2, and 2^-55 is nine times that. One pair of
        # i + j = 7 left out would be 16 * 74^2 * 2^-68 = 2^-51.6.
        worst = np.maximum(np.abs(err.real), np.abs(err.imag)) / s
        assert worst.max() <= 2.0 ** -55, np.log2(worst.max())


@pytest.mark.parametrize("orders", [[257], [300, 300], [384, 384], [385], [600, 400, 385, 384, 300, 257, 256, 200, 129]],
                         ids=str)
def test_merged_pair_digit_by_digit(orders):
    """The first panel's products into the next panel's rows and columns, then
    both panels' into the rest; the scales of the two differ."""
    rng = np.random.default_rng(sum(orders))
    a = []
    for n in orders:
        m = _cancelling(rng, n, 1)
        if n > 256:   # the second panel's operands are what the first update leaves of these
            m[128:, 128:] += _cancelling(rng, n - 128, 1)
        a.append(m)
    got = _update(a, len(set(orders)) > 1, 2)
    for m, g in zip(a, got):
        L, U = m[128:, :128], m[:128, 128:]
        one = (m[128:, 128:] - _mul(L, U))
        s0 = _scale(L, 1) * _scale(U, 0)
        nc = min(128, len(one))
        c = g[128:, 128:]   # the corner: one update, its entries held in FP64
        for part in (np.s_[:, :nc], np.s_[:nc, :]):
            e = (c[part] - one[part]).astype(complex)
            bound = 2.0 ** -55 * s0[part] + 2 * EPS * np.abs(one[part]).astype(float)
            assert (np.maximum(np.abs(e.real), np.abs(e.imag)) <= bound).all()
        if len(one) <= 128:
            continue
        L1, U1 = c[128:, :128], c[:128, 128:]
        two = one[128:, 128:] - _mul(L1, U1)
        s1 = _scale(L1, 1) * _scale(U1, 0)
        e = (c[128:, 128:] - two).astype(complex)
        # both panels' dropped digits, and the rounding of the sums: eight drains of each panel
        size = np.abs(_mul(L, U)[128:, 128:]).astype(float) + np.abs(_mul(L1, U1)).astype(float)
        bound = 2.0 ** -55 * (s0[128:, 128:] + s1) + 16 * EPS * size + 2 * EPS * np.abs(two).astype(float)
        assert (np.maximum(np.abs(e.real), np.abs(e.imag)) <= bound).all()


def test_nan_and_infinity_stay_in_their_rows_and_columns():
    rng = np.random.default_rng(9)
    m = rng.standard_normal((300, 300)) + 1j * rng.standard_normal((300, 300))
    m[200, 5], m[7, 250] = np.nan, np.inf
    g, = _update([m], False, 1)
    bad = ~np.isfinite(g[128:, 128:])
    want = np.zeros_like(bad)
    want[200 - 128, :] = want[:, 250 - 128] = True
    assert np.array_equal(bad, want)


# ---------------------------------------------------------------------------
# whole solves
# ---------------------------------------------------------------------------
def _case(mesh, w, depth=0.0):
    return C.Case(mesh, np.array([w]), np.array([0.0]), C.six_dofs(), C.six_dofs(), depth=depth)


def _solves():
    """(mesh, w): hulls whose far entries are smallest against the near ones, at both ends of the frequencies."""
    box, cyl = C.box_mesh(100.0, 20.0, 10.0, 64, 10, 7), C.cylinder_mesh(5.0, 10.0, 56, 22, 10, 28)
    return [(box, 2.5), (box, 0.3), (cyl, 2.5)]


def _sources():
    out = []
    with nb.Solver(0, nb.FP64) as s:
        for mesh, w in _solves():
            c = _case(mesh, w)
            s.set_case(c)
            nv = C.body_conditions(c)
            out.append([s.solve_potential(2 * np.pi / w, nv[:, j])["zigb"] for j in (0, 3)])
        return out, s.tensor_updates()


def test_sources_entry_by_entry():
    """Each source's error relative to itself, against sources refined in 80-bit
    arithmetic: no larger than with the updates on the FP64 pipe (quantiles; by a
    quarter at most, the two forms' errors being different samples)."""
    from scipy.linalg import lu_factor, lu_solve
    code = ("import sys, json; sys.path[:0] = %r; import test_gpu_fp64_precision as t; z, u = t._sources(); "
            "print(json.dumps([u, [[[list(x.real), list(x.imag)] for x in p] for p in z]]))" % [HERE, os.path.dirname(HERE)])
    env = dict(os.environ, NEMOH_B200_TC="0")
    ran = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert ran.returncode == 0, ran.stderr[-2000:]
    updates, pipe = json.loads(ran.stdout.strip().splitlines()[-1])
    assert updates == 0
    tensor, updates = _sources()
    assert updates >= 3
    for (mesh, w), zt, zp in zip(_solves(), tensor, pipe):
        c = _case(mesh, w)
        nv = C.body_conditions(c)
        with nb.Solver(0, nb.FP64) as s:
            s.set_case(c)
            (D, _, _, _), _ = s.assemble(2 * np.pi / (2 * np.pi / w))
        f, DL = lu_factor(D), D.astype(np.clongdouble)
        for x, y, b in zip(zt, zp, (nv[:, 0], nv[:, 3])):
            y = np.array(y[0]) + 1j * np.array(y[1])
            z = lu_solve(f, b).astype(np.clongdouble)
            for _ in range(3):
                z = z + lu_solve(f, (b - DL @ z).astype(np.complex128))
            et, ep = (np.abs(v - z).astype(float) / np.abs(z).astype(float) for v in (x, y))
            for q in (0.5, 0.9, 0.99):
                assert np.quantile(et, q) <= 1.25 * np.quantile(ep, q), (w, q, np.quantile(et, q), np.quantile(ep, q))
            assert np.abs(x - z).max() <= 1e-14 * np.abs(z).max()


def test_captured_updates():
    """A batch above the rule's line: direct, captured and replayed launches give the same forces."""
    rng = np.random.default_rng(1)
    c = _case(C.cylinder_mesh(6.0, 12.0, 28, 13, 6, 16), 1.0)   # 460 panels
    n, count = c.mesh.npanels, 24
    nv = [np.asfortranarray(rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))) for _ in range(count)]
    om, body = np.linspace(0.4, 1.6, count), np.zeros(count, np.int32)
    with nb.Solver(0, nb.FP64) as s:
        s.add_body(c)
        s.set_graphs(True)
        runs, issued = [], []
        for _ in range(4):
            runs.append(s.solve_bodies(body, om, nv))
            issued.append(s.tensor_updates())
        assert s.graph_stats() == (1, 2)
        assert 0 < issued[0] and issued[1] == 2 * issued[0] == issued[2] == issued[3]
    for got in runs[1:]:
        for g, r in zip(got, runs[0]):
            assert np.abs(g - r).max() <= 1e-13 * np.abs(r).max()   # the sums of the sources differ in their order


def test_ragged_batch_with_merged_pairs():
    """Twelve systems of 1,000 merge their panel pairs; others end in the first
    or second panel of a pair, or at its edge. Against each body alone, whose
    update is too small for the tensor cores: potentials of all panels."""
    orders = [1000, 700, 513, 512, 400, 385, 384, 300, 257, 256, 200, 129, 128, 100]
    full = C.cylinder_mesh(6.0, 12.0, 44, 19, 9, 24)
    assert full.npanels >= 1000
    cases = [_case(C.Mesh(full.nodes, full.panels[-n:], 0), 1.0) for n in orders]
    rng = np.random.default_rng(2)
    body = np.array([0] * 12 + list(range(1, len(orders))), np.int32)
    nv = [np.asfortranarray(rng.standard_normal((orders[b], 1)) + 1j * rng.standard_normal((orders[b], 1))) for b in body]
    om = np.linspace(0.5, 1.5, len(body))
    with nb.Solver(0, nb.FP64) as s:
        for c in cases:
            s.add_body(c, nds=np.eye(c.mesh.npanels))
        got = s.solve_bodies(body, om, nv)
        updates = s.tensor_updates()
        assert updates > 0
        for i in list(range(2)) + list(range(12, len(body))):
            alone, = s.solve_bodies(body[i:i + 1], om[i:i + 1], nv[i:i + 1])
            # two backward-stable solves of systems whose condition is some tens
            assert np.abs(got[i] - alone).max() <= 5e-14 * np.abs(alone).max(), (i, orders[body[i]])
        assert s.tensor_updates() == updates


@pytest.mark.parametrize("mixed_numbering", [False, True])
def test_hulls_taking_turns_stay_on_the_fp64_pipe(mixed_numbering):
    """A 1:20 pair of hulls 200 m apart: in body order the tensor cores update all
    panels but the one that both share; with the hulls' panels taking turns none."""
    a = C.cylinder_mesh(6.0, 12.0, 52, 22, 10, 28)
    both = C.merge_meshes([a, C.Mesh(a.nodes * 0.05 + np.array([200.0, 0.0, 0.0]), a.panels, 0)])
    panels = both.panels
    if mixed_numbering:
        panels = panels.reshape(2, a.npanels, 4).transpose(1, 0, 2).reshape(-1, 4)
    c = _case(C.Mesh(both.nodes, panels, 0), 1.0)
    with nb.Solver(0, nb.FP64) as s:
        s.set_case(c)
        s.solve_potential(2 * np.pi, C.body_conditions(c)[:, 0])
        assert (s.tensor_updates() > 0) != mixed_numbering
