"""Prolongation by a factor of 4 on rows of one to several units of 32 vertices, dealt to one, two and three warps, against
the oracle (each value rounded a few times: 1e-14); and its time against the restriction's, which moves the same vectors
one way."""
import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, setup_oracle, rel, random_masked_u

pytestmark = pytest.mark.gpu


def _box(nx, ny, nz):
    return workloads.cantilever(nx, ny, nz, lattice=tuple(max(4, n // 4 + 1) for n in (nx, ny, nz)))


@pytest.mark.parametrize("size", [(30, 9, 11), (31, 8, 8), (32, 8, 9), (63, 9, 8), (64, 8, 10), (97, 9, 9), (127, 8, 9),
                                  (160, 9, 8), (191, 8, 8), (224, 9, 9), (289, 8, 8)])
def test_rows_of_every_deal(oracle_mod, size):
    wl = _box(*size)
    g, o = setup_gpu(wl), setup_oracle(wl)
    uc = np.random.default_rng(7).standard_normal(g.size("u", 1))
    u = random_masked_u(wl.nv, o.get("vmask"), 9)
    for p in (g, o):
        p.update_operators()
        p.put("u", u)
        p.put("u", uc, 1)
        p.prolong(0)
    assert rel(g.get("u"), o.get("u")) < 1e-14


def test_fp64_prolongation_takes_less_than_the_restriction():
    """192x96x96: 55 against 90 us with a thread per four vertices, 43 against 74 now; 74 against 74 with whole pieces of 96
    from a row's start, the last of them with one vertex."""
    p = setup_gpu(_box(192, 96, 96))
    p.set_operator_precision(1)
    p.update_operators()
    us = []
    for call in (lambda: p.prolong(0), lambda: p.restrict(1)):
        t = []
        for _ in range(9):
            p.sync()
            p.timer_start()
            for _ in range(20):
                call()
            t.append(p.timer_stop() / 20 * 1e3)
        us.append(float(np.median(t)))
    p.close()
    assert us[0] < 0.8 * us[1], us
