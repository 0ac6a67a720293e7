"""The third-form kernels (csrc/form3.cuh) against the CPU oracle at every
compiled order, on small ragged boxes with randomly rotated element frames.

Bounds: those of test_gpu_parity.py (round-off of a few steps in FP64, where
the observed distance is about 1e-15 of the state's scale).
"""
import numpy as np
import pytest

import oracle
from cases import rotated_box
from oracle import ics

pytestmark = pytest.mark.gpu

ORDERS = [(1, 3)] + [(p, q) for p in range(2, 8) for q in (p + 1, p + 2)]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("inttype", [14, 4, 3])
@pytest.mark.parametrize("p,q", ORDERS)
def test_navier_stokes_3d_every_order(p, q, inttype):
    """Flux and update kernels: right-hand side on GLL values and two steps
    of each integrator."""
    import dgm_b200
    n = (3, 2, 2) if p < 6 else (2, 1, 2)
    m = rotated_box(3, n, 0.0, 2 * np.pi, p, q, seed=p)
    P = oracle.Problem(m, oracle.NS3D, flux="roe", vis=0.02)
    D = dgm_b200.Domain(m, dgm_b200.NS3D, flux="roe", inttype=inttype, vis=0.02)
    x, y, z = P.coords()
    f = ics.taylor_green(x, y, z, Ma=0.3)
    U0 = P.project(f)
    F_o, F_g = P.rhs(U0), D.time_derivative(U0)
    scale = np.sqrt((F_o ** 2).sum()) + np.sqrt((U0 ** 2).sum())
    assert np.sqrt(((F_g - F_o) ** 2).sum()) / scale < 1e-12
    P.set_state(U0)
    D.set_state(f)
    dt = 0.02 / (p + 1) ** 2
    assert P.advance(inttype, dt, 2) == 0
    D.advance(dt, 2)
    assert rel(D.state(), P.state()) < 1e-12
    D.close()
