"""Mixed-precision solves must not depend on what their workspace held before.

A process that has allocated and freed device memory gets it back with its old
contents, small blocks above all. The block panel forms only the triangles of
W = inv(L11) and V = inv(U11); their images must be zero outside them whatever
the scratch holds. Here many small blocks full of NaN are freed before a
context with a few systems is made, so that its small buffers are cut from
them."""
import numpy as np
import pytest

import gpu_cases as G
import nemoh_b200 as nb
from nemoh_b200 import cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("panels", [(12, 10, 5, 6), (16, 12, 6, 8), (10, 9, 2, 6)])
@pytest.mark.parametrize("nomega", [1, 2, 4])
def test_mixed_solve_after_freed_nan_blocks(panels, nomega):
    import torch
    nt, nz, nr, ns = panels
    mesh = C.cylinder_mesh(5.0, 10.0, 2 * nt, nz, nr, 2 * ns)   # 420, 576 and 204 panels: two to five LU panels
    case = C.Case(mesh, np.linspace(0.4, 1.4, nomega), np.array([0.0]), C.six_dofs(), C.six_dofs(), depth=0.0)
    nvel, nds, _ = G.problems(case)
    with nb.Solver(0, nb.FP64) as s:
        s.set_case(case)
        ref = s.solve_frequencies(case.omegas, nvel, nds)
    for _ in range(3):
        blocks = [torch.full((1 << 17,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(64)]
        torch.cuda.synchronize()
        del blocks
        torch.cuda.empty_cache()
        with nb.Solver(0, nb.MIXED) as s:
            s.set_case(case)
            got = s.solve_frequencies(case.omegas, nvel, nds)
            assert s.last_refinement()[0] > 0
        # the refinement's tolerance, 1e-12 of the right-hand side, over these well-conditioned hulls
        assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
