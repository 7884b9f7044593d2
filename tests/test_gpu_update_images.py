"""Operand images of the FP64 LU's tensor-core updates when device memory is
short: they are had for a whole batch before anything of it is launched, or the
update runs on the FP64 pipe, also in batches that are captured into graphs;
what a shortage leaves allocated is given back; and a mixed-precision context,
in which only the FP64 fallback takes images, doesn't count them as room for
its batches. Memory is made short by allocating the rest of the device."""
import contextlib

import numpy as np
import pytest

import nemoh_b200 as nb
from nemoh_b200 import cases as C

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _hull(n):
    """A hull of exactly n panels: a cylinder whose wall and bottom are cut to the count."""
    f = max(1.0, np.sqrt(n / 300.0))
    m = C.cylinder_mesh(6.0, 12.0, 2 * round(12 * f), round(10 * f) + 1, round(5 * f), 2 * round(6 * f) + 2)
    return C.Mesh(m.nodes, m.panels[-n:], 0)


def _body(n):
    return C.Case(_hull(n), np.array([0.8]), np.array([0.0]), C.six_dofs(), C.six_dofs(), depth=0.0)


def _items(rng, n, count):
    nv = rng.standard_normal((count, n, 2)) + 1j * rng.standard_normal((count, n, 2))
    return np.linspace(0.5, 1.2, count), [np.asfortranarray(v) for v in nv]


def _free():
    import torch
    return torch.cuda.mem_get_info(0)[0]


@contextlib.contextmanager
def _only(room):
    """All of the device but `room` bytes allocated."""
    import torch
    held = []
    try:
        for size in (1 << 33, 1 << 30, 1 << 27, 1 << 24, 1 << 22):
            while _free() > room + size:
                try:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("room", [20 * MB, 60 * MB])   # none of the images fits; the first of them does
def test_captured_batch_without_room_for_images(room):
    rng = np.random.default_rng(1)
    n, count = 400, 21
    om, nv = _items(rng, n, count)
    om_a, nv_a = _items(rng, 200, 200)
    with nb.Solver(0, nb.FP64) as s:
        s.add_body(_body(n))
        ref = s.solve_bodies(np.zeros(count, np.int32), om, nv)
        assert s.tensor_updates() > 0   # with room the batch takes them
    with nb.Solver(0, nb.FP64) as s:
        s.add_body(_body(n))
        s.add_body(_body(200))
        s.prepare_bodies()
        s.set_graphs(True)
        # a batch of many small systems provides every other buffer
        for _ in range(2):
            s.solve_bodies(np.ones(200, np.int32), om_a, nv_a)
        assert s.tensor_updates() == 0
        captures, replays = s.graph_stats()
        with _only(room):
            before = _free()
            runs = [s.solve_bodies(np.zeros(count, np.int32), om, nv) for _ in range(4)]
            after = _free()
        assert s.tensor_updates() == 0
        assert s.graph_stats() == (captures + 1, replays + 2)
        assert before - after < 16 * MB   # no part of the images is kept
        runs.append(s.solve_bodies(np.zeros(count, np.int32), om, nv))   # with room again
        assert s.tensor_updates() > 0
    for got in runs:
        for g, r in zip(got, ref):
            # both are backward-stable solves of well-conditioned systems
            assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()


def test_ragged_images_grow_with_headroom():
    """A stream of batches that each need a little more reallocates the images
    rarely (a reallocation synchronises the device), as its other buffers."""
    rng = np.random.default_rng(2)
    with nb.Solver(0, nb.FP64) as s:
        s.add_body(_body(400))
        s.prepare_bodies()
        free = []
        for count in range(40, 48):   # images of 192 to 226 MB
            om, nv = _items(rng, 400, count)
            s.solve_bodies(np.zeros(count, np.int32), om, nv)
            free.append(_free())
        assert s.tensor_updates() > 0
    assert len(set(free)) == 1, free


@pytest.mark.parametrize("ragged", [False, True])
def test_mixed_batches_after_a_fallback_in_short_memory(ragged, monkeypatch):
    """The fallback of 40 systems leaves images of 183 MB; with 100 MB free a
    larger mixed call is solved, in as many batches as fit."""
    rng = np.random.default_rng(3)
    n = 400
    case = _body(n)
    nds = C.generalised_normals(case)
    om, nv = _items(rng, n, 72)

    def solve(s, count):
        if ragged:
            return np.stack(s.solve_bodies(np.zeros(count, np.int32), om[:count], nv[:count]), axis=2)
        return s.solve_frequencies(om[:count], np.asfortranarray(np.stack(nv[:count], axis=2)), nds)

    with nb.Solver(0, nb.MIXED) as s:
        s.add_body(case)
        s.set_case(case)
        ref = solve(s, 72)
    with nb.Solver(0, nb.MIXED) as s:
        s.add_body(case)
        s.set_case(case)
        s.prepare_bodies()
        monkeypatch.setenv("NEMOH_B200_REFINE_MAX_IT", "1")
        solve(s, 40)
        monkeypatch.delenv("NEMOH_B200_REFINE_MAX_IT")
        assert s.tensor_updates() > 0
        with _only(100 * MB):
            for count in (44, 48, 52, 56, 60, 64, 68, 72):
                got = solve(s, count)
                # refined to 1e-12 of the right-hand side on either side
                assert np.abs(got - ref[:, :, :count]).max() <= 1e-10 * np.abs(ref).max()


def _ragged(s, ids, counts):
    rng = np.random.default_rng(4)
    bodies, nv = [], []
    for b, (n, count) in zip(ids, counts):
        bodies += [b] * count
        nv += _items(rng, n, count)[1]
    s.solve_bodies(np.array(bodies, np.int32), np.linspace(0.5, 1.2, len(bodies)), nv)


@pytest.mark.parametrize("counts,updates", [
    ([(700, 1), (200, 40)], (0, 0)),     # 0.54 M trailing entries after the first panel, in 41 systems
    ([(1100, 2), (200, 20)], (1, 4)),    # 1.99 M after the first panel (an update per stream group), 1.42 M after it
    ([(1100, 4), (300, 4)], (3, 10)),    # 3.9, 2.9, 2.1 and 1.4 M: three panels
])
def test_ragged_batches_count_the_systems_that_go_on(counts, updates):
    """The tensor-core update is for batches of 1.5 M trailing entries, counted
    over the systems that have some."""
    with nb.Solver(0, nb.FP64) as s:
        ids = [s.add_body(_body(n)) for n, _ in counts]
        _ragged(s, ids, counts)
        assert updates[0] <= s.tensor_updates() <= updates[1]


def test_small_systems_are_not_charged_for_images(monkeypatch):
    """64 items of 100 panels (about 0.7 MB each) fit a budget of 64 MB in one
    batch: systems of one panel have no trailing update and no images."""
    om, nv = _items(np.random.default_rng(5), 100, 64)

    def launches(s):
        before = s.launches
        s.solve_bodies(np.zeros(64, np.int32), om, nv)
        return s.launches - before

    with nb.Solver(0, nb.FP64) as s:
        s.add_body(_body(100))
        s.prepare_bodies()
        whole = launches(s)
        monkeypatch.setenv("NEMOH_B200_BATCH_BYTES", str(64 * MB))
        assert launches(s) == whole


def test_batches_of_one_call_share_the_room_for_images(monkeypatch):
    """A call of two batches, the small hulls' second: their matrices are smaller and
    their images larger than those of the first, and the buffers keep their size, so that
    images for a whole budget of small hulls don't fit beside them. The batch is cut to
    the room, both take the tensor cores, and every call finds the buffers where the last
    one left them: its batches replay."""
    monkeypatch.setenv("NEMOH_B200_BATCH_BYTES", str(400 * MB))
    rng = np.random.default_rng(6)
    om_a, nv_a = _items(rng, 1400, 5)     # 62 MB of matrices and 14 MB of images each
    om_b, nv_b = _items(rng, 400, 36)     # 5 MB and 5 MB
    body = np.array([0] * 5 + [1] * 36, np.int32)
    om, nv = np.concatenate([om_a, om_b]), nv_a + nv_b

    def bodies(s):
        s.add_body(_body(1400))
        s.add_body(_body(400))
        s.prepare_bodies()

    with nb.Solver(0, nb.FP64) as s:
        bodies(s)
        ref = [s.solve_bodies(body[:5], om[:5], nv[:5]), s.solve_bodies(body[5:], om[5:], nv[5:])]
        ref = ref[0] + ref[1]
        large = s.tensor_updates()
        s.solve_bodies(body[:5], om[:5], nv[:5])
        large = s.tensor_updates() - large
    with nb.Solver(0, nb.FP64) as s:
        bodies(s)
        s.solve_bodies(body[6:7], om[6:7], nv[6:7])   # kernels loaded
        before = s.tensor_updates()
        with _only(490 * MB):
            runs = [s.solve_bodies(body, om, nv)]     # the buffers grow from batch to batch
            assert s.tensor_updates() - before > large > 0
            s.set_graphs(True)   # one call directly, one captured, two replayed
            runs += [s.solve_bodies(body, om, nv) for _ in range(4)]
        captures, replays = s.graph_stats()
        assert captures >= 2 and replays == 2 * captures
    for got in runs:
        for g, r in zip(got, ref):
            # both are backward-stable solves of well-conditioned systems
            assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()


def test_mixed_batches_that_fall_back_replay(monkeypatch):
    """The FP64 fallback of a mixed batch runs outside the captured sequence: its
    images, which another batch's fallback has moved, are no reason to capture anew."""
    rng = np.random.default_rng(7)
    om_a, nv_a = _items(rng, 1000, 20)   # images of 210 MB
    om_b, nv_b = _items(rng, 300, 60)    # of 236 MB; of the other buffers the fallback's are smaller
    with nb.Solver(0, nb.MIXED) as s:
        s.add_body(_body(1000))
        s.add_body(_body(300))
        s.prepare_bodies()
        s.solve_bodies(np.ones(60, np.int32), om_b, nv_b)
        assert s.fallback_count()[0] == 0
        monkeypatch.setenv("NEMOH_B200_REFINE_MAX_IT", "1")   # every system falls back
        s.solve_bodies(np.zeros(20, np.int32), om_a, nv_a)
        s.set_graphs(True)
        for _ in range(2):
            s.solve_bodies(np.zeros(20, np.int32), om_a, nv_a)
        assert s.graph_stats() == (1, 0)
        updates = s.tensor_updates()
        s.solve_bodies(np.ones(60, np.int32), om_b, nv_b)
        assert s.tensor_updates() > updates
        s.solve_bodies(np.zeros(20, np.int32), om_a, nv_a)
        assert s.fallback_count()[0] == 5
        assert s.graph_stats() == (1, 1)
