"""A slender beam whose FP32 coarsest matrix is not positive definite: its bending stiffness is below FP32's rounding of
the stencils (1e-8 of the diagonal), which shows at one of the last pivots.  Both inversions report it, from an operator
update and from a design iteration, where they run on a second stream, and the handle goes on with FP64 operators."""
import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size, n", [((1100, 8, 8), 1668), ((800, 12, 10), 2727)])
def test_indefinite_matrix_is_reported(size, n):
    """n = 1,668: k_gj_sweep; 2,727: beyond the SMs' shared memory, k_gj_blocked, whose CTAs all have to leave at once."""
    wl = workloads.cantilever(*size, lattice=tuple(max(4, s // 4 + 1) for s in size))
    p = capi.Problem(*size)
    p.set_bc(wl.fixed, wl.loads)
    p.set_spline(wl.order, wl.partition, *wl.spline_box())
    rng = np.random.default_rng(0)
    p.put("coeff", np.clip(0.5 + 0.2 * rng.standard_normal(p.num_coeffs()), 0.02, 1.0))
    p.coeff_to_density()
    level = p.num_levels() - 1
    assert p.size("u", level) == n
    p.set_operator_precision(2)
    solve = dict(mode=capi.SOLVE_MIXED, smoother=capi.SMOOTH_CHEBYSHEV, pre=1, post=1, max_iter=20, inner_max=4)
    for call in (p.update_operators, lambda: p.design_iteration(solve=solve, oc=dict(vgoal=0.5))):
        with pytest.raises(capi.TopoError) as e:
            call()
        assert e.value.code == capi.TOPO_E_SINGULAR
    p.set_operator_precision(1)
    p.update_operators()
    p.put("f", rng.standard_normal(n), level)
    p.coarsest_solve()
    assert np.isfinite(p.get("u", level)).all()
    p.close()
