"""The FP64 update's schedule on the CPU: a producer that loads slices into
eight slots, two issuers that take the slice products of a tile in four phases
and an epilogue that drains the accumulators in pairs, each waiting only where
the kernel waits. Whatever the interleaving, every kept product is formed once,
from the slices it names, into the accumulator of its diagonal; no slot is
loaded while an issuer may read it; and all of them reach the end."""
import ctypes
import os
import random
import subprocess

import pytest

from nemoh_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nemoh_b200", "csrc")
SRC = os.path.join(HERE, "host_pairs", "host_schedule.cu")
LIB = os.path.join(HERE, "host_pairs", "_build", "libhost_schedule.so")
DEPS = [SRC] + [os.path.join(CSRC, f) for f in ("common.cuh", "linalg.cuh", "tc_gemm.cuh", "oz_gemm.cuh")]
SLICES, SLOTS, TILES = 8, 8, 4
CHUNK, LOW = (0, 1, 0, 1), (False, False, True, True)   # of the phases


@pytest.fixture(scope="module")
def schedule():
    if not os.path.exists(LIB) or any(os.path.getmtime(p) > os.path.getmtime(LIB) for p in DEPS):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run([B.NVCC] + B.COMMON + ["-O1", "-shared", "-cudart", "static", "-o", LIB, SRC], check=True)
    L = ctypes.CDLL(LIB)
    buf = (ctypes.c_int * 4096)()
    rows = lambda n, w: [tuple(buf[w * k:w * k + w]) for k in range(n)]  # noqa: E731
    loads = rows(L.host_schedule_loads(buf), 3)
    return loads, [rows(L.host_schedule_steps(w, buf), 10) for w in (0, 1)]


def _run(loads, plans, pick):
    fills, frees, content = [0] * SLOTS, [0] * SLOTS, [None] * SLOTS
    waits, held, at = [[0] * SLOTS, [0] * SLOTS], [set(), set()], [0, 0]
    begun, full, drained, summed = [0] * 4, [0] * 4, [0] * 4, [0] * 4
    made, loaded, pair = {}, 0, 0

    def load():
        nonlocal loaded
        if loaded == TILES * len(loads):
            return False
        piece, q, chunk = loads[loaded % len(loads)]
        if fills[q] and frees[q] < 2 * fills[q]:
            return False
        assert q not in held[0] | held[1]
        fills[q] += 1
        content[q] = (piece, chunk, loaded // len(loads))
        loaded += 1
        return True

    def drain():
        nonlocal pair
        accs = (2 * (pair % 2), 2 * (pair % 2) + 1)   # (0, 1), (2, 3), (0, 1), (2, 3) of a tile
        if any(full[a] == drained[a] for a in accs):
            return False
        for a in accs:   # a diagonal d has d + 1 products per chunk
            assert summed[a] == 2 * (a + 1 if pair % 4 > 1 else 8 - a)
            drained[a] += 1
        pair += 1
        return True

    def issue(w):
        if at[w] == TILES * len(plans[w]):
            return False
        ph, i, j, qi, qj, acc, first, need, retire, done = plans[w][at[w] % len(plans[w])]
        tile = at[w] // len(plans[w])
        slots = [q for q in range(SLOTS) if need >> q & 1]
        if first and drained[acc] < begun[acc] or any(fills[q] == waits[w][q] for q in slots):
            return False
        begun[acc] += first
        summed[acc] = 1 if first else summed[acc] + 1
        for q in slots:
            waits[w][q] += 1
            assert waits[w][q] == fills[q] and q not in held[w]
            held[w].add(q)
        assert {qi, qj} <= held[w]
        assert content[qi] == (i, CHUNK[ph], tile) and content[qj] == (j, CHUNK[ph], tile)
        assert acc == (i + j if LOW[ph] else 7 - i - j)
        key = (tile, CHUNK[ph], i, j)
        made[key] = made.get(key, 0) + 1
        for q in range(SLOTS):
            if retire >> q & 1:
                held[w].remove(q)
                frees[q] += 1
        assert done in (0, 1 << acc)
        full[acc] += bool(done)
        at[w] += 1
        return True

    actors = [load, drain, lambda: issue(0), lambda: issue(1)]
    while any(a() for a in pick(actors)):
        pass
    assert loaded == TILES * len(loads) and at == [TILES * len(p) for p in plans]
    assert not held[0] | held[1] and drained == [2 * TILES] * 4
    assert made == {(t, c, i, j): 1 for t in range(TILES) for c in (0, 1)
                    for i in range(SLICES) for j in range(SLICES) if i + j < 8}


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 2, 1, 0), (2, 0, 1, 3), (3, 0, 1, 2), (1, 2, 3, 0)], ids=str)
def test_schedule_with_one_role_ahead(schedule, order):
    _run(*schedule, lambda actors: [actors[k] for k in order])


def test_schedule_in_any_interleaving(schedule):
    rng = random.Random(1)
    for _ in range(200):
        _run(*schedule, lambda actors: rng.sample(actors, len(actors)))
