"""The bonded virial of the scheduled RATTLE sweeps is summed at least as well as
FP64 does it, as the kernel for single bonds sums it. Leaves on centres too heavy
to move: each bond's corrections are the same whether its centre has one leaf (a
molecule of its own, the single-bond kernel) or two (a scheduled molecule), so
both kernels add up the same FP32 products, all of one sign.

Bound: the sums of one sign over a tree round at 2^-53 of each partial sum, where
the last few levels' errors do not average out: some 2e-16 of the total a side, and
the step's scale as much again; 8e-16 is taken."""
import numpy as np
import pytest

from sucrose_gb300 import GpuSystem

pytestmark = pytest.mark.gpu


def bonded_virial(leaves, bonds, dt, velocities):
    rng = np.random.default_rng(1)
    u = rng.normal(size=(bonds, 3))
    u = (u / np.linalg.norm(u, axis=1, keepdims=True)).astype(np.float32).astype(np.float64)
    push = rng.uniform(0.002, 0.02, (bonds, 1))   # inwards
    k = np.arange(bonds)
    centre = k // leaves * (leaves + 1)
    leaf = centre + 1 + k % leaves
    n = bonds // leaves * (leaves + 1)
    r, v, mass = np.zeros((n, 3)), np.zeros((n, 3)), np.ones(n)
    mass[centre] = 1e30
    r[leaf] = u
    if velocities:
        v[leaf] = -50.0 * push * u
    g = GpuSystem(n, (40.0,) * 3)
    g.set_particles(mass=mass)
    g.upload(r=r, v=v)
    g.set_constraints(centre, leaf, np.linalg.norm(u, axis=1))
    g.constraints_save()
    if not velocities:
        r[leaf] = u * (1.0 - push)
        g.upload(r=r)
    g.zero_forces()
    (g.constraints_b if velocities else g.constraints_a)(dt)
    return g.thermo(3, 1.0)[1], g.constraint_stats()


@pytest.mark.parametrize("dt", [0.002, 0.0017, 0.003, 0.0041, 0.00123])
@pytest.mark.parametrize("velocities", [False, True])
def test_scheduled_sum_is_the_single_bonds(lib, dt, velocities):
    (one, s1), (two, s2) = (bonded_virial(k, 20000, dt, velocities) for k in (1, 2))
    done = "corrections_b" if velocities else "corrections_a"
    assert s1[done] == s2[done] >= 20000 and one > 0
    assert abs(two - one) <= 8e-16 * one
