"""Spline evaluation by chunks of element rows with tables of more than 48 KB of shared memory."""
import threading

import numpy as np
import pytest

from topoptspline3d_gb300 import capi, workloads
from tests.helpers import setup_gpu

pytestmark = pytest.mark.gpu


def _workload(size, partition, order):
    nx, ny, nz = size
    wl = workloads.cantilever(nx, ny, nz, lattice=tuple(p + order for p in partition), order=order)
    assert wl.partition == tuple(partition)
    return wl


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
