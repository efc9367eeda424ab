"""A step with a pair kind that does not exist is refused, wherever the kind stands
among the step's pair sets (two neighbouring sets can run as one launch)."""
import pytest

from helpers import lj_fcc
from sucrose_gb300 import GpuSystem, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [[-1, capi.COULOMB], [-1, capi.MORSE], [capi.COULOMB, -1], [-1], [capi.WCA, 8],
                                   [capi.LJ, 99], [-1, capi.DIPOLE]])
def test_unknown_kind_is_refused(lib, kinds):
    r, _, box, v = lj_fcc()
    g = GpuSystem(len(r), box)
    g.upload(r=r, v=v)
    g.init_nlist(0.3, 2.5)
    g.configure_step_pairs([g.params(k, cutoff=2.5) for k in kinds], integrator=capi.INT_NVE, dt=0.001)
    with pytest.raises(capi.SgError) as e:
        g.step(1)
    assert e.value.code == capi.SG_EINVAL
