"""The pair kernels' energy and virial sums lose nothing that double-float per
thread and FP64 per block hold. On a lattice of dyadic spacing the difference
vectors are exact, so that every pair of one difference has the same FP32
energy, of either sign by its length; a system of two particles with that
difference gives its value, and the sum of them over the lattice's pairs is
known exactly.

Bound: a thread adds up to some 130 terms; two-sum keeps each rounding error, and
those errors' own sum, at most 130 2^-24 of the terms' magnitudes, rounds at 2^-24
of itself: 5e-13 of the sum of magnitudes, taken as 1e-12."""
import itertools
import math

import numpy as np
import pytest

from sucrose_gb300 import GpuSystem, capi

pytestmark = pytest.mark.gpu


def vectors(reach):
    """Half of the lattice vectors no longer than reach: one of each pair +-v."""
    k = range(-int(reach), int(reach) + 1)
    return [v for v in itertools.product(k, k, k) if v > (0, 0, 0) and sum(x * x for x in v) <= reach * reach]


def lattice(cells, spacing, rng):
    g = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return (g[rng.permutation(len(g))] - cells // 2) * spacing, cells * spacing


def check(system, cutoff, kind, spacing, r, box, kw, both, setup=lambda g: None, launch=None):
    def call(n, pos, side, make=GpuSystem):
        g = make(n, side)
        setup(g)
        g.upload(r=np.asarray(pos, dtype=np.float64))
        if make is GpuSystem:
            g.init_nlist(0.3, cutoff)
        else:
            g.init_rep_nlist([0.3] * 3, [cutoff] * 3)
        if launch is not None:
            g.set_launch(kind, 256, launch)
        return g.pair_forces(g.params(kind, cutoff=cutoff, **kw), want_stats=True)
    two = [call(2, [[0, 0, 0], np.array(v) * spacing], (4 * cutoff,) * 3) for v in vectors((cutoff + 0.3) / spacing)]
    two = [(e, w) for e, w, st in two if st.solver_evals]
    e, w, st = call(len(r), r, (box,) * 3, system)
    assert st.solver_evals == len(r) * len(two)
    for got, terms in ((e, [x[0] for x in two]), (w, [x[1] for x in two]))[:2 if both else 1]:
        assert not both or min(terms) < 0 < max(terms)
        want, size = len(r) * math.fsum(terms), len(r) * math.fsum(map(abs, terms))
        assert abs(got - want) <= 1e-12 * size, (got / want - 1, size)


def replica(n, side):
    return GpuSystem.replicas([n], [side], [0])


@pytest.mark.parametrize("system", [GpuSystem, replica], ids=["rows", "spans"])
@pytest.mark.parametrize("cells", [12, 24, 34])   # sixteen and four lanes a row; entries as places
def test_lennard_jones(lib, system, cells):
    r, box = lattice(cells, 0.96875, np.random.default_rng(cells))
    check(system, 2.5, capi.LJ, 0.96875, r, box, {}, True)


@pytest.mark.parametrize("cells", [12, 20])
def test_gay_berne(lib, cells):
    spacing = 1.25
    r, box = lattice(cells, spacing, np.random.default_rng(cells))
    # parallel ellipsoids, none near contact: one sign, lengths and directions of unlike energy
    check(GpuSystem, 4.0, capi.GB, spacing, r, box, dict(mu=2, nu=1), False,
          setup=lambda g: g.set_particles(sig=(1.0, 1.0, 1.2), eps=(1.0, 1.0, 0.3)), launch=1)
