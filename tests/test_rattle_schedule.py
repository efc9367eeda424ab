"""The schedule of the grouped RATTLE sweeps (csrc/rattle_schedule.h): run as the
kernel runs it, period by period and row by row, its visits see what those of
sweeps in list order see. Each visit reads and bumps a counter of both its
atoms; a visit's readings, sweep by sweep, are those of the sequential loop exactly
when every two visits that share an atom keep their order, and the rows are
race-free when the constraints of one share no atom."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sucrose_gb300", "csrc")


@pytest.fixture(scope="module")
def schedule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rattle_schedule")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text('#include "rattle_schedule.h"\n'
                   'extern "C" int schedule(int nc, const int* loc, int* lanes, int* slots) {\n'
                   '    std::vector<WaveSlot> l;\n'
                   '    for (int k = 0; k < nc; ++k) l.push_back({loc[2 * k], loc[2 * k + 1]});\n'
                   '    const WaveSchedule w = wave_schedule(l);\n    *lanes = w.lanes;\n'
                   '    for (size_t k = 0; k < w.slots.size(); ++k) { slots[2 * k] = w.slots[k].x; '
                   'slots[2 * k + 1] = w.slots[k].y; }\n    return w.period;\n}\n')
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                        str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(str(lib)).schedule

    def call(bonds):
        loc = np.ascontiguousarray(bonds, dtype=np.int32)
        slots, lanes = np.zeros(2 * 64 * 64, dtype=np.int32), C.c_int(0)
        period = fn(len(loc), loc.ctypes.data_as(C.c_void_p), C.byref(lanes), slots.ctypes.data_as(C.c_void_p))
        return slots[:2 * period * lanes.value].reshape(period, lanes.value, 2)
    return call


def chain(n):
    return [(k, k + 1) for k in range(n - 1)]


def graphs():
    rng = np.random.default_rng(11)
    yield from ([(0, 1)], chain(3), chain(32), [(0, 1), (1, 2), (2, 0)], [(0, 1), (0, 1)], [(0, k) for k in range(1, 10)],
                [(k, (k + 1) % 6) for k in range(6)], [(i, j) for i in range(4) for j in range(i + 1, 4)],
                chain(8) + [(k, 8 + k) for k in range(8)])
    for _ in range(200):
        n = int(rng.integers(3, 33))
        bonds = [(int(rng.integers(k)), k) for k in range(1, n)]   # a tree, and some rings
        bonds += [tuple(int(x) for x in rng.permutation(n)[:2]) for _ in range(int(rng.integers(0, 5)))]
        yield [bonds[k] if rng.integers(2) else bonds[k][::-1] for k in rng.permutation(len(bonds))]


def test_scheduled_visits_are_the_sequential_ones(schedule):
    sweeps = 5
    for bonds in graphs():
        rows = schedule(bonds)
        used = rows[rows[:, :, 0] >= 0]
        assert sorted(used[:, 1]) == list(range(len(bonds)))
        assert all((x & 255, x >> 8 & 255) == bonds[k] for x, k in used)
        for row in rows:
            atoms = [a for x, k in row if x >= 0 for a in bonds[k]]
            assert len(atoms) == len(set(atoms))
        want, count = {}, {}
        for s in range(sweeps):
            for k, b in enumerate(bonds):
                want[k, s] = tuple(count.get(a, 0) for a in b)
                for a in b:
                    count[a] = count.get(a, 0) + 1
        got, count = {}, {}
        for cycle in range(sweeps + 64):
            for row in rows:
                for x, k in row:
                    s = cycle - (x >> 16)
                    if x < 0 or not 0 <= s < sweeps:
                        continue
                    got[k, s] = tuple(count.get(a, 0) for a in bonds[k])
                    for a in bonds[k]:
                        count[a] = count.get(a, 0) + 1
        assert got == want
