"""Gauss-Seidel sweeps against the oracle at the sizes where their forms change:
level 1 with its largest colour just inside one cluster's share (378 vertices),
just above it (420), and odd; the fine colours with ragged groups of 32."""
import numpy as np
import pytest

from topoptspline3d_gb300 import workloads
from tests.helpers import setup_gpu, setup_oracle, rel, random_coeff, random_masked_u

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("size", [(64, 48, 40), (72, 52, 44), (61, 37, 29)])
def test_sweeps_match_oracle(oracle_mod, size, reverse):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=(nx // 4 + 1, ny // 4 + 1, nz // 4 + 1))
    coeff = random_coeff(int(np.prod([p + wl.order for p in wl.partition])), seed=3)
    g, o = setup_gpu(wl, coeff), setup_oracle(wl, coeff)
    rng = np.random.default_rng(4)
    u = random_masked_u(wl.nv, o.get("vmask"), 9) * 1e-6
    for p in (g, o):
        p.update_operators()
        p.put("u", u)
        p.smooth(0, 1, reverse=reverse)
    assert rel(g.get("u"), o.get("u")) < 1e-12
    n = g.size("u", 1)
    f1, u1 = rng.standard_normal(n), rng.standard_normal(n)
    for p in (g, o):
        p.put("f", f1, 1)
        p.put("u", u1, 1)
        p.smooth(1, 2, reverse=reverse)
    assert rel(g.get("u", 1), o.get("u", 1)) < 1e-11
