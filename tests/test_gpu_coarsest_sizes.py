"""The coarsest inverse of the mixed path at sizes where its tiling changes: one
32-pivot tile, a last tile of a few rows, several tiles a CTA.  The design
iteration's compliance against FP64 MG-PCG with the FP64 inverse."""
import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, random_coeff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size, cap, n", [((4, 4, 4), 1, 24), ((8, 4, 4), 8, 36), ((16, 8, 8), 16, 135),
                                          ((48, 24, 24), 400, 336), ((16, 8, 8), 400, 675), ((77, 44, 42), 400, 1617)])
def test_compliance_with_either_inverse(size, cap, n):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(max(4, s // 4 + 1) for s in size))
    coeff = random_coeff(int(np.prod([p + wl.order for p in wl.partition])), seed=6, lo=0.2)
    c = []
    for mode, prec in ((capi.SOLVE_PCG64, 1), (capi.SOLVE_MIXED, 2)):
        p = capi.Problem(nx, ny, nz, max_coarse_elements=cap)
        p.set_bc(wl.fixed, wl.loads)
        p.set_spline(wl.order, wl.partition, *wl.spline_box())
        p.put("coeff", coeff)
        p.coeff_to_density()
        p.set_operator_precision(prec)
        assert p.size("u", p.num_levels() - 1) == n
        p.update_operators()
        p.solve(mode=mode, smoother=capi.SMOOTH_CHEBYSHEV, pre=1, post=1, rtol=1e-9, max_iter=300)
        c.append(p.compliance())
        p.close()
    assert abs(c[0] - c[1]) < 1e-8 * c[0]
