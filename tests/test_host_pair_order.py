"""CPU check of a pair of submerged panels in the order in which the wave pass
evaluates it: in finite depth the exponential images first, the tabulated part
added to them. Against the oracle's influence matrices at the parity tests'
tolerances (1e-12 of each row's largest entry in deep water, 1e-10 in finite
depth), with wave terms of the tables and of the asymptotic form (k R above
99.7)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import gpu_cases as G
from nemoh_b200 import build as B
from nemoh_b200 import cases as C

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nemoh_b200", "csrc")
SRC = [os.path.join(HERE, "host_pairs", f) for f in ("host_order.cu", "host_pairs.cu")]
LIB = os.path.join(HERE, "host_pairs", "_build", "libhost_order.so")
DEPS = SRC + [os.path.join(CSRC, f) for f in ("common.cuh", "green.cuh", "assembly.cuh", "freesurface.cuh",
                                              "kochin.cuh", "preproc.cuh", "fd_setup.cpp", "fd_setup.h")]
_d, _i = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)


def _far(half):
    a = C.box_mesh(20.0, 8.0, 4.0, nx=4, ny=2, nz=2, half=half)
    mesh = C.merge_meshes([a, C.Mesh(a.nodes + np.array([290.0, 0.0, 0.0]), a.panels, a.isym)])
    c = C.Case(mesh, np.sqrt(9.81 * np.array([0.32, 0.36])), np.array([0.0]), C.six_dofs(), C.six_dofs(), depth=50.0)
    c.name = "far_half" if half else "far"
    return c


CASES = G.small_cases() + [_far(False), _far(True)]


@pytest.mark.parametrize("case", CASES, ids=[c.name for c in CASES])
def test_pairs_in_the_wave_pass_order(case):
    if not os.path.exists(LIB) or any(os.path.getmtime(p) > os.path.getmtime(LIB) for p in DEPS):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run([B.NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler",
                        "-fPIC,-ffp-contract=off", "-shared", "-o", LIB, SRC[0], os.path.join(CSRC, "fd_setup.cpp")],
                       check=True)
    f = ctypes.CDLL(LIB).host_order_assemble
    f.argtypes = [ctypes.c_int] * 3 + [_d, _i, _d, ctypes.c_double, _d] + [ctypes.c_double] * 3 + [_i, _i] + [_d] * 4
    m = case.mesh
    n = m.npanels
    o = G.oracle_for(case)
    geo, zer = o.geometry()
    _, _, apd = o.tables()
    geo, apd = np.ascontiguousarray(geo), np.ascontiguousarray(apd.transpose(0, 2, 1)).ravel()
    p = lambda a: a.ctypes.data_as(_d)  # noqa: E731
    nq, mode = ctypes.c_int(0), ctypes.c_int()
    for w in case.omegas:
        mats = [np.zeros((n, n), dtype=np.complex128, order="F") for _ in range(4)]
        st = f(len(m.nodes), n, m.isym, p(m.nodes), m.panels.ctypes.data_as(_i), p(geo), zer, p(apd), case.g,
               case.depth, w, ctypes.byref(nq), ctypes.byref(mode), *[p(a) for a in mats])
        assert st == 0
        ref, mode_o, _ = o.assemble(w)
        assert mode.value == mode_o
        for a, b in zip(mats, ref):
            err = np.abs(a - b) / np.abs(b).max(axis=1, keepdims=True)
            assert err.max() < (1e-10 if mode_o else 1e-12), (w, err.max())
