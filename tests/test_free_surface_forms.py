"""Elevations at the frequencies where the bodies' finite-depth wave number
lies above the field points' limit. For K h from about 16 to 20 (K = w^2 / g)
the reference solves with the finite-depth forms, whose root search returns an
AMH above 20, and evaluates the field points with the deep-water forms, whose
wave number is w^2 / g and not AMH / h. Bound: the parity tests' 1e-9 of a
problem's largest |ETA|."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle_lib as O
from nemoh_b200 import build as B
from nemoh_b200 import cases as C

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nemoh_b200", "csrc")
SRC = [os.path.join(HERE, "host_pairs", f) for f in ("host_forms.cu", "host_pairs.cu")]
LIB = os.path.join(HERE, "host_pairs", "_build", "libhost_forms.so")
DEPS = SRC + [os.path.join(CSRC, f) for f in ("common.cuh", "green.cuh", "assembly.cuh", "freesurface.cuh",
                                              "kochin.cuh", "preproc.cuh", "fd_setup.cpp", "fd_setup.h")]
DEPTH, G = 50.0, 9.81
KH = [12.0, 15.0, 16.5, 17.5, 19.0, 21.0]


def _case(half):
    mesh = C.box_mesh(20.0, 8.0, 4.0, nx=5, ny=2 if half else 3, nz=2, half=half)
    rng = np.random.default_rng(6)
    z = rng.standard_normal((mesh.npanels, 2)) + 1j * rng.standard_normal((mesh.npanels, 2))
    zs = rng.standard_normal(z.shape) + 1j * rng.standard_normal(z.shape) if half else np.zeros_like(z)
    # near the hull (tabulated wave terms) and far from it (asymptotic ones)
    xy = np.concatenate([rng.uniform(12.0, 40.0, (20, 2)), rng.uniform(150.0, 350.0, (20, 2))])
    o = O.Oracle(mesh.nodes, mesh.panels, mesh.isym, 1000.0, G, DEPTH, cache_s=True)
    return mesh, z, zs, xy, o


def _period(kh):
    return 2 * np.pi / np.sqrt(G * kh / DEPTH)


def _close(eta, ref):
    assert (np.abs(eta - ref) / np.abs(ref).max(axis=0)).max() < 1e-9


@pytest.mark.parametrize("kh", KH)
@pytest.mark.parametrize("half", [False, True])
def test_host_forms(half, kh):
    if not os.path.exists(LIB) or any(os.path.getmtime(p) > os.path.getmtime(LIB) for p in DEPS):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run([B.NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler",
                        "-fPIC,-ffp-contract=off", "-shared", "-o", LIB, SRC[0], os.path.join(CSRC, "fd_setup.cpp")],
                       check=True)
    f = ctypes.CDLL(LIB).host_forms_free_surface
    d, i = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    f.argtypes = [ctypes.c_int] * 3 + [d, i, d, ctypes.c_double, d] + [ctypes.c_double] * 3 + \
                 [ctypes.c_int, d, ctypes.c_int, d, d, d, i]
    mesh, z, zs, xy, o = _case(half)
    geo, zer = o.geometry()
    _, _, apd = o.tables()
    p = lambda a: np.ascontiguousarray(a).ctypes.data_as(d)  # noqa: E731
    geo, apd = np.ascontiguousarray(geo), np.ascontiguousarray(apd.transpose(0, 2, 1)).ravel()
    zf, zsf = np.asfortranarray(z), np.asfortranarray(zs)
    eta = np.zeros((len(xy), 2), dtype=np.complex128, order="F")
    finite = ctypes.c_int()
    T = _period(kh)
    st = f(len(mesh.nodes), mesh.npanels, mesh.isym, p(mesh.nodes), mesh.panels.ctypes.data_as(i), p(geo), zer, p(apd),
           G, DEPTH, T, len(xy), p(xy), 2, zf.ctypes.data_as(d), zsf.ctypes.data_as(d), eta.ctypes.data_as(d),
           ctypes.byref(finite))
    assert st == 0
    _close(eta, o.free_surface(T, xy, z, zs))
    amh = O.x0(kh) if kh < 20 else kh   # kwave h, at 20 and above
    assert finite.value == (amh < 20)


@pytest.mark.gpu
@pytest.mark.parametrize("kh", KH)
@pytest.mark.parametrize("half", [False, True])
def test_elevation_and_kochin(half, kh):
    import nemoh_b200 as nb
    mesh, z, zs, xy, o = _case(half)
    T = _period(kh)
    theta = np.linspace(0.0, 3.0, 7)
    with nb.Solver(0, nb.FP64) as s:
        s.set_mesh(mesh.nodes, mesh.panels, mesh.isym, 1000.0, G, DEPTH)
        _close(s.free_surface(T, xy, z, zs), o.free_surface(T, xy, z, zs))
        _close(s.kochin(T, theta, z, zs), o.kochin(T, theta, z, zs if half else None))
