"""Restriction and prolongation against the oracle, by a factor of 4 (the smallest:
2), at rows that end on, before and after a warp's piece (96 fine vertices).
Random vectors; a restricted value has 343 terms whose weights' sum is 11 of
their norms, added in chains of at most 24: 24 x 11 x 2^-53 on either side."""
import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, setup_oracle, rel, random_masked_u

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(16, 8, 8), (95, 9, 13), (96, 10, 11), (125, 12, 9), (128, 8, 15), (193, 9, 8)])
def test_transfers_match_oracle(oracle_mod, size):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=(nx // 4 + 1, max(4, ny // 4 + 1), max(4, nz // 4 + 1)))
    g, o = setup_gpu(wl), setup_oracle(wl)
    rng = np.random.default_rng(7)
    r, uc = rng.standard_normal(3 * wl.nv), rng.standard_normal(g.size("u", 1))
    u = random_masked_u(wl.nv, o.get("vmask"), 9)
    for p in (g, o):
        p.update_operators()
        p.put("r", r)
        p.restrict(1)
        p.put("u", u)
        p.put("u", uc, 1)
        p.prolong(0)
    assert rel(g.get("f", 1), o.get("f", 1)) < 1e-13
    assert rel(g.get("u"), o.get("u")) < 1e-14


@pytest.mark.parametrize("size", [(48, 24, 24), (112, 96, 76), (112, 96, 80)])
def test_fp32_cycle_converges_as_fp64(size):
    """The FP32 restriction's forms (637, 14,500 and 15,225 coarse vertices: inside, just inside and outside the
    small grids' form) through the solves they precondition: rounding of 1e-7 in the cycle moves a CG's count by one at
    most, and both solves end below 1e-9 of the load, so their compliances agree to 1e-8."""
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(s // 4 + 1 for s in size))
    found = []
    for mode, prec in ((capi.SOLVE_PCG64, 1), (capi.SOLVE_MIXED, 2)):
        p = setup_gpu(wl)
        p.set_operator_precision(prec)
        p.update_operators()
        st = p.solve(mode=mode, smoother=capi.SMOOTH_CHEBYSHEV, pre=1, post=1, rtol=1e-9, max_iter=300, inner_max=1)
        found.append((st["iterations"], p.compliance()))
        p.close()
    (i64, c64), (i32, c32) = found
    assert abs(i64 - i32) <= 1
    assert abs(c64 - c32) < 1e-8 * c64
