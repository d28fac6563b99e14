"""The forms of the fixed-point fine operator besides the single residual: materials from nearly incompressible to
strongly auxetic, neighbouring elements of very different displacements vertex by vertex, several right-hand sides,
the FP64 Chebyshev step with and without void planes, values that are not finite."""
import os
import subprocess
import sys

import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, rel, random_coeff, random_masked_u

pytestmark = pytest.mark.gpu

SIGN = np.array([[np.prod([(1 if a >> k & 1 else -1) if m >> k & 1 else 1 for k in range(3)]) for m in range(8)]
                 for a in range(8)])


def _exact(wl, rhop, vmask, u, nu, E=1e6):
    """K u in extended precision, and per vertex the sum over its elements of density, largest mode and stiffness: what
    their forces are rounded in proportion to."""
    L = np.longdouble
    nx, ny, nz = wl.nx, wl.ny, wl.nz
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    on = np.flatnonzero(rhop)
    z, y, x = on // (nx * ny), on // nx % ny, on % nx
    nodes = (x + (nx + 1) * (y + (ny + 1) * z))[:, None] + np.array(
        [(a & 1) + (nx + 1) * ((a >> 1 & 1) + (ny + 1) * (a >> 2)) for a in range(8)])
    c = [np.asarray(u[i][nodes], L) @ SIGN.astype(L) for i in range(3)]
    g = [np.zeros_like(c[0]) for _ in range(3)]
    for m, w in ((0, L(1) / 16), (1, L(1) / 48), (2, L(1) / 48), (4, L(1) / 48), (3, L(1) / 144), (5, L(1) / 144), (6, L(1) / 144)):
        D = [[c[i][:, m | 1 << j] if not m >> j & 1 else 0 * c[0][:, 0] for j in range(3)] for i in range(3)]
        tr = D[0][0] + D[1][1] + D[2][2]
        for i in range(3):
            for j in range(3):
                if not m >> j & 1:
                    g[i][:, m | 1 << j] += w * (L(mu) * (D[i][j] + D[j][i]) + (L(lam) * tr if i == j else 0))
    out, scale = np.zeros((3, wl.nv), L), np.zeros(wl.nv)
    stiff = max(abs(lam) / 48, mu / 48, abs(lam + 4 * mu) / 144)
    mode = np.max([np.abs(q[:, 1:]).max(1) for q in c], axis=0).astype(float)
    np.add.at(scale, nodes, (rhop[on] * mode * stiff)[:, None])
    for i in range(3):
        np.add.at(out[i], nodes, (g[i] @ SIGN.T.astype(L)) * np.asarray(rhop[on], L)[:, None])
        out[i] *= (vmask >> i & 1) & (vmask >> 3 & 1)
    return out, scale


def _fx_product(p, wl, vm, u):
    """-(f - K u) with a load far below K u's last bit."""
    f = np.zeros((3, wl.nv))
    f[2, np.flatnonzero(vm >> 2 & 1)[-1]] = 1e-140
    p.put("f", f)
    p.put("u", u)
    p.solve(mode=capi.SOLVE_PCG64, max_iter=0, check=False)
    return -p.get("r").reshape(3, -1)


# An element's force is within 111 units (see test_fx_host), a vertex's sum of eight within 24 more of the largest;
# a unit is 2^-57 of mode times constant, each up to twice its value: 4 x 135 x 2^-57 < 34 x 2^-53 of the scale.
def check_every_vertex():
    for nu in (-0.9, 0.0, 0.4999):
        for spread in (1.0, 1e9):  # how much further the vertices of the void alone move
            wl = workloads.cantilever(37, 21, 13, lattice=(9, 6, 5))
            p = setup_gpu(wl, nu=nu)
            solid = np.zeros((13, 21, 37), bool)
            solid[:, 4:17, 10:30] = True
            p.put("rho", np.where(solid, 1.0, 1e-3).ravel())
            p.update_operators()
            vm = p.get("vmask")
            u = random_masked_u(wl.nv, vm, 3).reshape(3, -1) * 1e-6
            touched = np.zeros((14, 22, 38), bool)
            for k in range(8):
                touched[(k >> 2):13 + (k >> 2), (k >> 1 & 1):21 + (k >> 1 & 1), (k & 1):37 + (k & 1)] |= solid
            u = np.where(touched.ravel(), u, spread * u)
            y = _fx_product(p, wl, vm, u)
            exact, scale = _exact(wl, p.get("rhop"), vm, u, nu)
            p.close()
            err = np.abs((y - exact).astype(float)).max(0)
            assert (err <= 34 * 2.0 ** -53 * scale + 2.0 ** -53 * np.abs(y).max(0)).all(), (nu, spread)


def test_every_vertex_within_its_elements_rounding():
    """In a process of its own: a device holds one material at a time, and other tests' handles may be alive."""
    subprocess.run([sys.executable, "-c", "from tests import test_gpu_fine_fx_forms as t; t.check_every_vertex()"],
                   cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), check=True, timeout=300)


@pytest.mark.parametrize("nrhs", [1, 2, 5])
def test_right_hand_sides_have_their_own_residuals(nrhs):
    """A solve of no steps reports each right-hand side's residual: FP64 sums of at most 1e5 squares."""
    wl = workloads.cantilever(37, 21, 13, lattice=(9, 6, 5))
    p = setup_gpu(wl)
    p.set_operator_precision(2)
    p.update_operators()
    p.multi_reserve(5)
    vm = p.get("vmask")
    U = np.stack([random_masked_u(wl.nv, vm, 3 + k) * 10.0 ** -k for k in range(nrhs)])
    F = np.stack([random_masked_u(wl.nv, vm, 50 + k) * 1e6 for k in range(nrhs)])
    _, _, rr = p.solve_multi(F, U, max_iter=0, check=False)
    for k in range(nrhs):
        r = F[k].reshape(3, -1) - _exact(wl, p.get("rhop"), vm, U[k].reshape(3, -1), 0.4)[0]
        assert abs(rr[k] / float(np.sqrt((r ** 2).sum() / (F[k] ** 2).sum())) - 1) < 1e-12


@pytest.mark.parametrize("degree", [1, 3])
@pytest.mark.parametrize("size, wl", [((33, 9, 13), "box"), ((62, 31, 29), "box"), ((80, 40, 40), "void")])
def test_chebyshev_step_as_in_native_fp64(size, wl, degree):
    """One step of PCG64, whose preconditioner is Chebyshev smoothing with fixed-point products, against native FP64.
    Roundings of 2^-52 through some ten products, amplified by the coarse solve's condition of 1e5: 1e-10."""
    nx, ny, nz = size
    w = workloads.large_ellipsoids(nx, ny, nz) if wl == "void" else workloads.cantilever(
        nx, ny, nz, lattice=tuple(max(4, n // 4 + 1) for n in size))
    coeff = random_coeff(int(np.prod([q + w.order for q in w.partition])), seed=9, lo=0.2)
    found = []
    for arithmetic in (0, 1):
        p = setup_gpu(w, coeff)
        p.set_fine_arithmetic(arithmetic)
        p.update_operators()
        p.solve(mode=capi.SOLVE_PCG64, smoother=capi.SMOOTH_CHEBYSHEV, pre=2, post=2, cheb_degree=degree, max_iter=1,
                rtol=1e-14, check=False)
        found.append((p.get("u"), p.get("r")))
        p.close()
    assert np.linalg.norm(found[0][0]) > 0
    assert rel(found[1][0], found[0][0]) < 1e-10
    assert rel(found[1][1], found[0][1]) < 1e-10


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e306])
def test_not_finite_is_reported(value):
    wl = workloads.cantilever(33, 9, 13, lattice=(9, 4, 4))
    p = setup_gpu(wl)
    p.update_operators()
    u = np.zeros(3 * wl.nv)
    u[wl.nv // 2] = value
    p.put("u", u)
    with pytest.raises(capi.TopoError) as e:
        p.solve(mode=capi.SOLVE_PCG64)
    assert e.value.code == capi.TOPO_E_NONFINITE


@pytest.mark.parametrize("size", [(48, 24, 24), (61, 37, 29), (112, 96, 80)])
def test_one_mixed_step_as_in_fp64(size):
    """One outer step with one FP32 V-cycle against the same in FP64 (the FP32 restriction's forms: eight lanes a coarse
    vertex on the first two boxes, rows on the third).  FP32 roundings of 6e-8 through ten products and the coarse
    solve: 1e-4; a misplaced weight is of the order of the correction itself."""
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(max(4, n // 4 + 1) for n in size))
    coeff = random_coeff(int(np.prod([q + wl.order for q in wl.partition])), seed=9, lo=0.2)
    found = []
    for mode, precision in ((capi.SOLVE_PCG64, 1), (capi.SOLVE_MIXED, 2)):
        p = setup_gpu(wl, coeff)
        p.set_operator_precision(precision)
        p.update_operators()
        p.solve(mode=mode, smoother=capi.SMOOTH_CHEBYSHEV, pre=1, post=1, max_iter=1, inner_max=1, rtol=1e-14, check=False)
        found.append(p.get("u"))
        p.close()
    assert rel(found[1], found[0]) < 1e-4
