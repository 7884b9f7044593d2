"""The blocks of the LU panels (the 32 x 32 factor with both inverses, the
32 x 32 tiles of a step, the 128 x 128 block of the mixed path) at orders
around their widths, on general dense systems whose pivots reach far up and
down the exponent range: a pivot's reciprocal is formed by scaling."""
import ctypes

import numpy as np
import pytest

import nemoh_b200 as nb
from nemoh_b200 import cases as C

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _entry():
    f = nb.load_library().nemoh_b200_factor_solve_device_noalloc
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                  ctypes.c_void_p, ctypes.c_char_p, ctypes.c_int]
    return f


def _systems(rng, n, nsys, scale):
    a = rng.standard_normal((nsys, n, n)) + 1j * rng.standard_normal((nsys, n, n))
    a = 0.3 / np.sqrt(n) * a + np.exp(2j * np.pi * rng.uniform(size=(nsys, 1, n))) * np.eye(n)
    return a * scale   # diagonally dominant: no pivoting needed, condition of a few units


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 32, 33, 63, 64, 65, 95, 127, 130, 161])
@pytest.mark.parametrize("scale", [1e-18, 1.0, 1e160])
def test_factor_solve_orders_and_scales(n, scale):
    import torch
    rng = np.random.default_rng(n)
    nsys, nrhs = 3, 2
    a = _systems(rng, n, nsys, scale)
    x = rng.standard_normal((nsys, nrhs, n)) + 1j * rng.standard_normal((nsys, nrhs, n))
    ad = torch.from_numpy(np.ascontiguousarray(a.transpose(0, 2, 1))).cuda()   # column-major
    xd = torch.from_numpy(x.copy()).cuda()
    torch.cuda.synchronize()
    st = _entry()(0, n, nsys, ad.data_ptr(), nrhs, xd.data_ptr(), torch.cuda.current_stream().cuda_stream, None, 0)
    assert st == 0
    got = xd.cpu().numpy()
    for s in range(nsys):
        ref = np.linalg.solve(a[s] / scale, x[s].T).T / scale
        # backward-stable elimination without growth: n eps times the condition (below 10)
        assert np.abs(got[s] - ref).max() <= 30 * (n + 10) * EPS * np.abs(ref).max()


def test_singular_pivot_is_reported():
    import torch
    a = np.eye(40, dtype=complex)
    a[37, 37] = 1e-21
    ad, xd = torch.from_numpy(a).cuda(), torch.ones(1, 1, 40, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    st = _entry()(0, 40, 1, ad.data_ptr(), 1, xd.data_ptr(), torch.cuda.current_stream().cuda_stream, None, 0)
    assert st == 3


@pytest.mark.parametrize("n", [31, 96, 127, 128, 130, 160, 191, 255, 290, 353])
def test_mixed_block_panels(n):
    """The mixed path's sources at orders that end in every part of a panel block."""
    f = max(1.0, np.sqrt(n / 300.0))
    m = C.cylinder_mesh(6.0, 12.0, 2 * round(12 * f), round(10 * f) + 1, round(5 * f), 2 * round(6 * f) + 2)
    c = C.Case(C.Mesh(m.nodes, m.panels[-n:], 0), np.array([0.5, 0.9]), np.array([0.0]), C.six_dofs(), C.six_dofs(),
               depth=0.0)
    nv = C.body_conditions(c)
    with nb.Solver(0, nb.MIXED) as s:
        s.set_case(c)
        for i, w in enumerate(c.omegas):
            T = 2 * np.pi / w
            (D, _, _, _), _ = s.assemble(2 * np.pi / T)
            for j in (0, 3):
                b = nv[:, 7 * i + j]
                x = np.linalg.solve(D, b)
                got = s.solve_potential(T, b)["zigb"]
                it, _ = s.last_refinement()
                assert 0 < it <= 5   # FP32 factors of a well-conditioned hull
                # refined to 1e-12 of the right-hand side, condition below 10
                assert np.abs(got - x).max() <= 1e-11 * np.abs(x).max()
