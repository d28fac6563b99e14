"""Spline evaluation by chunks of element rows at the sizes where its tables change: more than 48 KB of shared
memory, a partition finer than the elements (the chunk's rows use more basis rows than the table holds), an x
partition finer than the elements, and rows above 1,024 elements, which go to the two-pass form.  Densities against
the oracle; double-float products of up to 64 terms whose weights add up to 1: 64 x 2^-46 of the largest coefficient."""
import threading

import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu, setup_oracle, random_coeff

pytestmark = pytest.mark.gpu


def _workload(size, partition, order):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(p + order for p in partition), order=order)
    assert wl.partition == tuple(partition)
    return wl


@pytest.mark.parametrize("size, partition, order", [
    ((64, 8, 8), (1500, 3, 3), 4),    # 60 KB, one row a chunk
    ((64, 8, 8), (4800, 3, 3), 4),    # 192 KB
    ((64, 8, 8), (5200, 3, 3), 4),    # more than a CTA may take: two passes
    ((40, 48, 48), (900, 12, 12), 3),  # 52 KB, three rows a chunk
    ((8, 40, 40), (3, 100, 100), 4),  # more basis rows than the table holds
    ((8, 104, 96), (3, 250, 30), 2),
    ((1024, 4, 4), (30, 3, 3), 3),    # the longest row of one CTA
    ((1025, 4, 4), (30, 3, 3), 3),
])
def test_densities_match_oracle(oracle_mod, size, partition, order):
    wl = _workload(size, partition, order)
    coeff = random_coeff(int(np.prod([p + order for p in partition])), seed=11, lo=-0.2, hi=1.2)
    g, o = setup_gpu(wl, coeff), setup_oracle(wl, coeff)
    a, b = g.get("rho"), o.get("rho")
    assert np.max(np.abs(a - b)) < 64 * 2.0 ** -46 * 1.2
    # the trial volumes of an OC update decide its bracket: the same trials and threshold
    csens = -np.random.default_rng(3).uniform(0.5, 2.0, coeff.size)
    for p in (g, o):
        p.put("csens", csens)
    (tg, lg), (to, lo) = g.oc_update(0.5), o.oc_update(0.5)
    assert tg == to and abs(lg - lo) <= 1e-12 * abs(lo)
    assert np.max(np.abs(g.get("rho") - o.get("rho"))) < 64 * 2.0 ** -46 * 1.2
    g.close()


def test_threads_with_different_tables():
    """Two designs whose tables need different amounts of shared memory, a host thread each: neither takes the other's
    launches away."""
    errors = []

    def work(nx_partition):
        try:
            wl = _workload((64, 8, 8), (nx_partition, 3, 3), 4)
            p = setup_gpu(wl)
            first = p.get("rho")
            for _ in range(4000):
                p.coeff_to_density()
            if not np.array_equal(first, p.get("rho")):
                errors.append("densities changed")
            p.close()
        except capi.TopoError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(n,)) for n in (1300, 2300, 1800, 4000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
