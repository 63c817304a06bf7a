"""Carried GFM coefficients resolved from a list longer than one pass of the
kernel's grid (77,824 threads): along a solid west wall of 300 x 300 cells
every W face is listed, as are none in a box without solid.  Bit for bit
against the oracle."""
import numpy as np
import pytest

from simcoflow3d_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solid", [("xslab", 0.2), None])
def test_carried_coefficients(gpu_lib, solid):
    from simcoflow3d_gb300.projection import Projection
    w = W.build_workload("wall", 10, 300, 300, solid=solid, liquid=W._surface(0.5, 0.02, None),
                         rho_l=1000.0, rho_g=1.2)
    p = Projection.for_workload(w, rel_tol=1e-3, stale_init=0.75)
    got, _, _ = p.poisson_solve(w)
    p.close()
    assert np.array_equal(got, O.pocoef(w, stale_init=0.75), equal_nan=True)
