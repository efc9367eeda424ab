"""A position that is not finite leaves the other particles' forces alone: no
pair of that particle is in range, so everything is, bit for bit, as with the
particle out of reach of all that its rows list."""
import numpy as np
import pytest

from helpers import f32
from sucrose_gb300 import GpuSystem, capi

pytestmark = pytest.mark.gpu

KINDS = {capi.LJ: {}, capi.LJ12: {}, capi.LJW: dict(wf=0.1), capi.WCA: {},
         capi.MORSE: dict(dissoc=1.3, width=1.7, rmin=1.1), capi.DH: dict(db_len=1.0, dielectric=2.0),
         capi.COULOMB: dict(dielectric=1.5)}


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n", [2000, 12000, 40000])   # sixteen and four lanes a row; entries as places
@pytest.mark.parametrize("periodic", [True, False])
def test_other_particles_keep_their_forces(lib, n, bad, periodic):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    box = side * 1.12
    r = f32((grid + 0.5 + rng.uniform(-0.08, 0.08, grid.shape)) * 1.12 - box / 2)
    g = GpuSystem(n, (box,) * 3, periodic)
    g.set_charges(rng.choice([-1.0, 1.0], n))
    g.upload(r=r)
    g.init_nlist(0.3, 2.5)
    for k in (0, n // 2):
        moved = r.copy()
        moved[k, 0] += box / 2 if periodic else 4 * box   # further than list radius and cut-off from its neighbours
        lost = r.copy()
        lost[k, rng.integers(3)] = bad
        others = np.arange(n) != k
        for kind, kw in KINDS.items():
            out = []
            for x in (moved, lost):
                g.upload(r=x)   # the list stays
                g.zero_forces()
                pe, vir, st = g.pair_forces(g.params(kind, cutoff=2.5, **kw), want_stats=True)
                out.append((g.forces()[0], pe, vir, st.solver_evals))
            (f0, pe0, vir0, in0), (f1, pe1, vir1, in1) = out
            assert np.abs(f0).max() > 0 and not f0[k].any()
            assert np.array_equal(f0[others], f1[others]) and not f1[k].any(), kind
            assert (pe0, vir0, in0) == (pe1, vir1, in1)
