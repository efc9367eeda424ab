"""When the captured step's calls make a graph of several steps (csrc/graph_steps.h):
not before the gaps it takes out have cost what making it costs, so that a
program that changes its configuration every few calls does not make one in vain,
and one that goes on has it soon."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sucrose_gb300", "csrc")
GAP, NODE, MOST = 4, 3, 16


@pytest.fixture(scope="module")
def call(tmp_path_factory):
    d = tmp_path_factory.mktemp("graph_steps")
    src, lib = d / "shim.cpp", d / "shim.so"
    # what sg_step does of it: graphs of several while they fit, then single steps
    src.write_text('#include "graph_steps.h"\n'
                   'extern "C" int call(int* steps, long long* gaps, int n, int kernels) {\n'
                   '    GraphSteps g;\n    g.steps = *steps;\n    g.gaps = *gaps;\n'
                   '    const int want = g.wanted(n, kernels);\n    if (want) g.made(want);\n'
                   '    g.gaps += g.launches(n);\n    *steps = g.steps;\n    *gaps = g.gaps;\n    return want;\n}\n')
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                        str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(lib)).call


def run(call, lengths, kernels):
    """Graphs made during calls of these lengths: (call, steps) each, and launches in all."""
    steps, gaps, made, total = C.c_int(0), C.c_longlong(0), [], 0
    for k, n in enumerate(lengths):
        want = call(C.byref(steps), C.byref(gaps), n, kernels)
        if want:
            made.append((k, want))
        s = steps.value
        total += n // s + n % s if s else n
    return made, total


@pytest.mark.parametrize("kernels", [4, 6, 14])
def test_few_calls_make_none(call, kernels):
    assert run(call, [20] * 2, kernels)[0] == []
    assert run(call, [10] * 3, kernels)[0] == []       # a box change every few calls
    assert run(call, [30], kernels)[0] == []
    assert run(call, [1] * 10000 + [0], kernels)[0] == []


@pytest.mark.parametrize("kernels", [4, 6, 14])
@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 30, 33, 100, 1000])
def test_it_is_made_when_the_gaps_have_cost_as_much(call, kernels, n):
    made, total = run(call, [n] * 4000, kernels)
    (k, steps), = made
    assert 2 <= steps <= min(n, MOST)
    cost = NODE * kernels * steps
    assert GAP * n * max(k, 1) >= cost and (k == 0 or GAP * n * (k - 1) < cost)
    assert total <= n * k + (4000 - k) * (n // steps + n % steps)


def test_a_longer_one_replaces_it_when_that_pays_too(call):
    made, _ = run(call, [3] * 100 + [100] * 100, 4)
    assert [m[1] for m in made] == [3, 14] and made[1][0] >= 100
    assert len(run(call, [3, 30] * 2000, 4)[0]) <= 2   # changing lengths do not make it over and over


@pytest.mark.gpu
def test_a_longer_graph_takes_over_from_a_shorter_one(lib):
    # rows add without atomics and NVE reads no sums: the same bits however launched
    import numpy as np
    from helpers import lj_fcc
    from sucrose_gb300 import GpuSystem, capi
    r, _, box, v = lj_fcc()
    out = []
    for lengths in ([3] * 12 + [100, 100, 5], [1] * 241):
        g = GpuSystem(len(r), box)
        g.upload(r=r, v=v)
        g.init_nlist(0.3, 2.5)
        g.configure_step(g.params(capi.LJ, cutoff=2.5), integrator=capi.INT_NVE, dt=0.004)
        for n in lengths:
            g.step(n)
        g.step_check()
        out.append((*g.download(), g.energies()))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
