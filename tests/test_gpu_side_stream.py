"""The FP64 coarsest inversion of a design iteration runs beside the solve's set-up."""
import time

import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


def test_inversion_beside_the_set_up_takes_no_longer_than_alone():
    """What FP64 operators add to an iteration (n = 1,617: their inversion, most of all) against the inversion in an
    operator update of its own: 7.1 against 8.7 ms when its CTAs lie evenly, 14.5 when the set-up came first."""
    nx, ny, nz = 77, 44, 42
    wl = workloads.half_mbb(nx, ny, nz, lattice=(20, 12, 11))
    kw = dict(solve=dict(mode=capi.SOLVE_MIXED, smoother=capi.SMOOTH_CHEBYSHEV, pre=1, post=1, max_iter=300, inner_max=4,
                         cheb_lo=0.1), oc=dict(vgoal=wl.vgoal))

    def median(f):
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return float(np.median(t))

    iteration, update = [], []
    for precision in (2, 3):
        p = capi.Problem(nx, ny, nz)
        p.set_bc(wl.fixed, wl.loads)
        p.set_spline(wl.order, wl.partition, *wl.spline_box())
        p.put("coeff", np.full(p.num_coeffs(), wl.coeff0))
        p.coeff_to_density()
        p.set_operator_precision(precision)
        for _ in range(3):
            p.design_iteration(**kw)
        rho, coeff, u = p.get("rho"), p.get("coeff"), p.get("u")

        def run():
            p.put("coeff", coeff)
            p.put("u", u)
            p.coeff_to_density()
            p.design_iteration(**kw)
            p.sync()

        iteration.append(median(run))
        for every in (1, 1000):  # with the inversion, and with the inverse kept
            p.set_coarse_refresh(every)

            def refresh():
                p.put("rho", rho)
                p.update_operators()
                p.sync()

            update.append(median(refresh))
        p.close()
    assert iteration[1] - iteration[0] < 1.2 * (update[2] - update[3])
