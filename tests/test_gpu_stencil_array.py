"""TOPO_STENCIL of small levels, which the kernels hold in another form: the same values for a caller that asks before the
operators are built, after, again after a later update, and through a device pointer kept from before it."""
import numpy as np
import pytest

from topoptspline3d_gb300 import workloads
from tests.helpers import setup_gpu, setup_oracle, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ask_first", [False, True])
def test_stencil_follows_the_operators(oracle_mod, ask_first):
    import torch
    wl = workloads.cantilever(33, 17, 13, lattice=(9, 5, 4))
    g, o = setup_gpu(wl), setup_oracle(wl)
    n = g.size("stencil", 1)

    def view():
        a = type("View", (), {"__cuda_array_interface__": dict(shape=(n,), typestr="<f8", version=3,
                                                                data=(g.device_ptr("stencil", 1), False))})()
        return torch.as_tensor(a, device="cuda")

    kept = view() if ask_first else None
    for k in range(2):
        rho = np.random.default_rng(k).uniform(0.1, 1.0, wl.nx * wl.ny * wl.nz)
        for p in (g, o):
            p.put("rho", rho)
            p.update_operators()
        for level in range(1, g.num_levels()):
            assert rel(g.get("stencil", level), o.get("stencil", level)) < 1e-12
        kept = view() if kept is None else kept
        g.sync()
        assert np.array_equal(kept.cpu().numpy(), g.get("stencil", 1))
    g.close()
