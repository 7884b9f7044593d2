"""The FP64 LU's trailing update on the tensor cores (integer slices, exact
products): the sources of FP64 solves against numpy's LU of the assembled
matrix, at orders around its tiles (128 rows, 64 columns) and its panel pairs,
for batches large enough to take that path, uniform and ragged."""
import os
import re

import numpy as np
import pytest

import nemoh_b200 as nb
from nemoh_b200 import cases as C

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = 2.0 ** -53


def _hull(n):
    """A hull of exactly n panels: a cylinder whose wall and bottom are cut to the count."""
    f = max(1.0, np.sqrt(n / 300.0))
    m = C.cylinder_mesh(6.0, 12.0, 2 * round(12 * f), round(10 * f) + 1, round(5 * f), 2 * round(6 * f) + 2)
    assert m.npanels >= n
    return C.Mesh(m.nodes, m.panels[-n:], 0)


def _case(n, nomega):
    return C.Case(_hull(n), np.linspace(0.5, 1.1, nomega), np.array([0.0]), C.six_dofs(), C.six_dofs(), depth=0.0)


def _sources(mats, nvel):
    return np.linalg.solve(mats, nvel)


def _forces(case, D, S, nvel, nds, w):
    z = S @ _sources(D, nvel)
    return -nds @ (case.rho * 1j * w * z)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nomega", [(385, 64), (449, 48), (513, 32), (640, 20), (769, 14), (1027, 7), (1281, 4)])
def test_forces_of_tensor_core_updates(n, nomega):
    case = _case(n, nomega)
    assert (n - 128) ** 2 * nomega >= 4.2e6   # the batch takes the path
    nv = C.body_conditions(case).reshape(n, 7, nomega, order="F")
    nds = C.generalised_normals(case)
    with nb.Solver(0, nb.FP64) as s:
        s.set_case(case)
        F = s.solve_frequencies(case.omegas, np.asfortranarray(nv), nds)
        for i in (0, nomega - 1):
            w = 2 * np.pi / (2 * np.pi / case.omegas[i])
            (D, _, S, _), _ = s.assemble(w)
            ref = _forces(case, D, S, nv[:, :, i], nds, w)
            # backward-stable solves: n eps cond(D) at most, and these hulls' cond is a few tens
            assert np.abs(F[:, :, i] - ref).max() <= 50 * n * EPS * np.abs(ref).max()


@pytest.mark.gpu
def test_ragged_batch_of_tensor_core_updates():
    orders = [129, 257, 300, 450, 641, 900, 1100]
    cases = [_case(n, 3) for n in orders]
    with nb.Solver(0, nb.FP64) as s:
        ids = [s.add_body(c) for c in cases]
        bodies = np.repeat(np.array(ids, dtype=np.int32), 3)
        om = np.concatenate([c.omegas for c in cases])
        nv = [C.body_conditions(c)[:, 7 * j:7 * j + 7] for c in cases for j in range(3)]
        assert len(bodies) * (1100 - 128) ** 2 >= 4.2e6
        F = s.solve_bodies(bodies, om, nv)
        for i, c in enumerate(cases):
            s.set_case(c)
            (D, _, S, _), _ = s.assemble(2 * np.pi / (2 * np.pi / om[3 * i]))
            ref = _forces(c, D, S, nv[3 * i], C.generalised_normals(c), om[3 * i])
            assert np.abs(F[3 * i] - ref).max() <= 50 * orders[i] * EPS * np.abs(ref).max()


def test_images_are_in_the_graph_key():
    """A captured batch holds the addresses of the operand images."""
    src = os.path.join(ROOT, "nemoh_b200", "csrc")
    api = open(os.path.join(src, "api.cu")).read()
    key = api[api.index("std::vector<long long> sig = {"):]
    key = key[:key.index("};")]
    body = open(os.path.join(src, "oz_gemm.cuh")).read()
    body = body[body.index("struct OzWork {"):]
    ptrs = re.findall(r"^\s*(?:unsigned char|double)\* (\w+) = nullptr;", body[:body.index("\n};")], re.M)
    assert ptrs == ["a", "b", "sc"]
    assert all("c->oz.%s" % p in key for p in ptrs)
