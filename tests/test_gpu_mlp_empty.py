"""Training samples of a list without pairs, or for no room: none, and no error."""
import ctypes as C

import pytest

from sucrose_gb300 import GpuSystem, capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("apart, capacity", [(9.0, 16), (9.0, 0), (2.5, 0)])
def test_no_samples(lib, apart, capacity):
    import torch
    g = GpuSystem(2, (20.0,) * 3)
    g.set_particles(sig=(3.0, 2.0, 1.0))
    g.upload(r=[[-apart / 2, 0, 0], [apart / 2, 0, 0]])
    g.init_nlist(0.3, 3.0)
    g.pair_forces(g.params(capi.ECPR, solver=capi.SOLVER_NEWTON))
    assert g.npairs() == (apart < 3.3)
    X = torch.zeros((16, 16), dtype=torch.bfloat16, device="cuda")
    y = torch.zeros(16, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    count = C.c_int64(-1)
    rc = g.L.sg_mlp_features(g.ctx, C.c_void_p(X.data_ptr()), C.c_void_p(y.data_ptr()), capacity, C.byref(count))
    assert rc == capi.SG_OK and count.value == 0
