"""The fixed-point fine operator of the CG solvers: the residual f - K u that a
solve of no iterations leaves, against K u in extended precision.  Ragged tiles,
z blocks of every remainder, void planes, smooth and rough fields, densities
over the whole SIMP range.  Its error has to stay within that of FP64."""
import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, random_masked_u

pytestmark = pytest.mark.gpu


def _apply_exact(wl, rhop, vmask, u):
    """K u in long double: per element the modal form's sums over nodes, dense."""
    L = np.longdouble
    nx, ny, nz = wl.nx, wl.ny, wl.nz
    vx, vy = nx + 1, ny + 1
    lam, mu = 1e6 * 0.4 / ((1 + 0.4) * (1 - 2 * 0.4)), 1e6 / (2 * (1 + 0.4))
    H = np.array([[np.prod([(1 if a >> k & 1 else -1) if S >> k & 1 else 1 for k in range(3)]) for S in range(8)]
                  for a in range(8)])
    on = np.flatnonzero(rhop)
    z, y, x = on // (nx * ny), on // nx % ny, on % nx
    nodes = (x + vx * (y + vy * z))[:, None] + np.array([(a & 1) + vx * ((a >> 1 & 1) + vy * (a >> 2)) for a in range(8)])
    c = [np.asarray(u[i][nodes], L) @ H.astype(L) for i in range(3)]
    g = [np.zeros_like(c[0]) for _ in range(3)]
    for fset, w in (((0,), L(1) / 16), ((1, 2, 4), L(1) / 48), ((3, 5, 6), L(1) / 144)):
        for m in fset:  # gradient restricted to function m: d_j u_i ~ c_i[m | j], j not in m
            D = [[(c[i][:, m | 1 << j] if not m >> j & 1 else 0 * c[0][:, 0]) for j in range(3)] for i in range(3)]
            tr = D[0][0] + D[1][1] + D[2][2]
            for i in range(3):
                for j in range(3):
                    if not m >> j & 1:
                        s = L(mu) * (D[i][j] + D[j][i]) + (L(lam) * tr if i == j else 0)
                        g[i][:, m | 1 << j] += w * s
    out = np.zeros((3, wl.nv), L)
    for i in range(3):
        f = (g[i] @ H.T.astype(L)) * np.asarray(rhop[on], L)[:, None]
        np.add.at(out[i], nodes, f)
        out[i] *= (vmask >> i & 1) & (vmask >> 3 & 1)
    return out


@pytest.mark.parametrize("field", ["rough", "smooth", "offset"])
@pytest.mark.parametrize("size, tz, masked", [((16, 8, 8), 4, False), ((33, 9, 5), 1, False), ((31, 7, 6), 16, False),
                                              ((37, 21, 13), 4, True), ((62, 15, 9), 3, False), ((5, 4, 30), 7, False)])
def test_residual_within_fp64_error(size, tz, masked, field):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(max(4, s // 4 + 1) for s in size))
    if masked:
        wl.eactive = workloads.perforated(nx, ny, nz, holes=4, radius=(1.5, 2.2), seed=5)
    p = setup_gpu(wl)
    rng = np.random.default_rng(8)
    rho = 10.0 ** rng.uniform(-3, 0, p.ne) * (p.get("eactive") != 0)
    p.put("rho", rho)
    p.update_operators()
    p.set_tiles(tz, tz)
    vm = p.get("vmask")
    u = random_masked_u(wl.nv, vm, 3).reshape(3, -1) * 1e-6
    if field != "rough":
        z, y, x = np.meshgrid(*(np.arange(n + 1.0) for n in (nz, ny, nx)), indexing="ij")
        free = np.stack([(vm >> c & 1) & (vm >> 3 & 1) for c in range(3)])
        lin = np.stack([1e-6 * (0.3 * x + 0.1 * y), 1e-6 * (0.2 * z - 0.1 * x), -2e-6 * x * x / nx]).reshape(3, -1)
        u = (1e-3 * u + lin + (1e-2 if field == "offset" else 0.0)) * free
    f = np.zeros((3, wl.nv))
    f[2, np.flatnonzero(vm >> 2 & 1)[-1]] = 1e-140  # a load, so that the solve runs (its square is not 0), below the last bit of K u
    p.put("f", f)
    p.put("u", u)
    p.solve(mode=capi.SOLVE_PCG64, max_iter=0, check=False)
    r = -p.get("r").reshape(3, -1)
    exact = _apply_exact(wl, p.get("rhop"), vm, u)
    native = p.apply_fine(u, 0).reshape(3, -1)
    norm = float(np.sqrt((exact ** 2).sum()))
    e_fx = float(np.sqrt(((r - exact) ** 2).sum())) / norm
    e_64 = float(np.sqrt(((native - exact) ** 2).sum())) / norm
    print(size, tz, field, "fixed point %.2e FP64 %.2e" % (e_fx, e_64))
    # one rounding of the result to FP64 is up to 1.1e-16; the rest is the operator's
    assert e_fx <= max(1.2e-16, e_64)
    assert np.array_equal(p.get("u").reshape(3, -1), u)


def test_not_a_number_is_reported():
    wl = workloads.cantilever(16, 8, 8, lattice=(7, 5, 5))
    p = setup_gpu(wl)
    p.update_operators()
    u = np.zeros(3 * wl.nv)
    u[wl.nv // 2] = np.nan
    p.put("u", u)
    with pytest.raises(capi.TopoError) as e:
        p.solve(mode=capi.SOLVE_PCG64)
    assert e.value.code == capi.TOPO_E_NONFINITE
