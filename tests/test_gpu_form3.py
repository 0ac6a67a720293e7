"""The 3-D and 2-D tiles (csrc/form3.cuh, stage2.cuh, stage2d.cuh) against the
CPU oracle at every compiled order, on small ragged boxes with randomly rotated
element frames.

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
    """Flux and update kernels of every tile: right-hand side on GLL values
    and two steps of each integrator."""
    import dgm_b200
    n = (3, 2, 2) if p < 6 else (2, 1, 2)
    m = rotated_box(3, n, 0.0, 2 * np.pi, p, q, seed=p)
    P = oracle.Problem(m, oracle.NS3D, flux="roe", vis=0.02)
    D = dgm_b200.Domain(m, dgm_b200.NS3D, flux="roe", inttype=inttype, vis=0.02)
    x, y, z = P.coords()
    f = ics.taylor_green(x, y, z, Ma=0.3)
    U0 = P.project(f)
    F_o = P.rhs(U0)
    scale = np.sqrt((F_o ** 2).sum()) + np.sqrt((U0 ** 2).sum())
    P.set_state(U0)
    dt = 0.02 / (p + 1) ** 2
    assert P.advance(inttype, dt, 2) == 0
    for k in range(D.variant_count()):
        D.set_variant(k)
        assert np.sqrt(((D.time_derivative(U0) - F_o) ** 2).sum()) / scale < 1e-12
        D.set_state(f)
        D.advance(dt, 2)
        assert rel(D.state(), P.state()) < 1e-12
    D.close()


@pytest.mark.parametrize("inttype", [14, 4, 3])
@pytest.mark.parametrize("flux", ["laxfriedrichs", "roe"])
@pytest.mark.parametrize("p,q", ORDERS)
def test_euler_3d_every_order(p, q, flux, inttype):
    """Every tile (third form; at q = p+2 up to p = 5 the second form too, whose
    TVD3 and RK4 stages run the third) and its right-hand side on GLL values."""
    import dgm_b200
    n = (3, 2, 2) if p < 6 else (2, 1, 2)
    m = rotated_box(3, n, 0.0, 2 * np.pi, p, q, seed=p)
    P = oracle.Problem(m, oracle.EULER3D, flux=flux)
    D = dgm_b200.Domain(m, dgm_b200.EULER3D, flux=flux, inttype=inttype)
    x, y, z = P.coords()
    f = ics.taylor_green(x, y, z, Ma=0.3)
    U0 = P.project(f)   # at q = p+1 projecting twice is not projecting once
    F_o = P.rhs(U0)
    scale = np.sqrt((F_o ** 2).sum()) + np.sqrt((U0 ** 2).sum())
    P.set_state(U0)
    dt = 0.02 / (p + 1) ** 2
    assert P.advance(inttype, dt, 2) == 0
    for k in range(D.variant_count()):
        D.set_variant(k)
        assert np.sqrt(((D.time_derivative(U0) - F_o) ** 2).sum()) / scale < 1e-12
        D.set_state(f)
        D.advance(dt, 2)
        assert rel(D.state(), P.state()) < 1e-12
    D.close()


ORDERS_2D = [(p, q) for p in range(1, 9) for q in (p + 1, p + 2)]


@pytest.mark.parametrize("phys", ["euler2d", "ns2d", "shallow"])
@pytest.mark.parametrize("inttype", [14, 4, 3])
@pytest.mark.parametrize("p,q", ORDERS_2D)
def test_2d_every_order(p, q, inttype, phys):
    """Every 2-D tile on a ragged, randomly rotated mesh (more elements than
    one CTA holds, not a multiple of it), and the right-hand side on GLL
    values (one launch, traces interpolated in it)."""
    import dgm_b200
    code = {"euler2d": 1, "ns2d": 2, "shallow": 30}[phys]
    m = rotated_box(2, (7, 5), -5.0, 5.0, p, q, seed=p)
    flux, vis = ("laxfriedrichs", 0.0) if phys == "shallow" else ("roe", 0.02 if phys == "ns2d" else 0.0)
    P = oracle.Problem(m, code, flux=flux, vis=vis)
    if phys == "shallow":
        P.set_sw_balance(False)
    x, y, _ = P.coords()
    f = ics.gaussian_bump(x, y, w=2.0) if phys == "shallow" else ics.isentropic_vortex(x, y, beta=2.0, period=(10.0, 10.0))
    U0 = P.project(f)
    dt = 0.01 / (p + 1) ** 2
    F_o = P.rhs(U0)
    P.set_state(U0)
    assert P.advance(inttype, dt, 2) == 0
    D = dgm_b200.Domain(m, code, flux=flux, inttype=inttype, vis=vis, sw_balance=False)
    scale = np.sqrt((F_o ** 2).sum()) + np.sqrt((U0 ** 2).sum())
    for k in range(D.variant_count()):
        D.set_variant(k)
        assert np.sqrt(((D.time_derivative(U0) - F_o) ** 2).sum()) / scale < 1e-12
        D.set_state(f)
        D.advance(dt, 2)
        assert rel(D.state(), P.state()) < 1e-12
    D.close()


@pytest.mark.parametrize("phys,p", [("euler2d", 1), ("euler2d", 4), ("euler2d", 8), ("shallow", 3), ("shallow", 8),
                                    ("euler3d", 1), ("euler3d", 4), ("euler3d", 7)])
def test_mixed_form_every_tile(phys, p):
    """The FP32 form of the same tiles: 1e-6 of the FP64 oracle, the bar of
    the mixed form's other tests."""
    import dgm_b200
    code, dim = {"euler2d": (1, 2), "shallow": (30, 2), "euler3d": (8, 3)}[phys]
    n = (7, 5) if dim == 2 else (3, 2, 2)
    lo, hi = (-5.0, 5.0) if dim == 2 else (0.0, 2 * np.pi)
    m = rotated_box(dim, n, lo, hi, p, 0, seed=p)
    flux = "laxfriedrichs" if phys == "shallow" else "roe"
    P = oracle.Problem(m, code, flux=flux)
    if phys == "shallow":
        P.set_sw_balance(False)
    x, y, z = P.coords()
    f = (ics.gaussian_bump(x, y, w=2.0) if phys == "shallow" else
         ics.isentropic_vortex(x, y, beta=2.0, period=(10.0, 10.0)) if dim == 2 else ics.taylor_green(x, y, z, Ma=0.3))
    U0 = P.project(f)
    dt = 0.01 / (p + 1) ** 2
    P.set_state(U0)
    assert P.advance(14, dt, 2) == 0
    D = dgm_b200.Domain(m, code, flux=flux, precision=dgm_b200.MIXED, sw_balance=False)
    for k in range(D.variant_count()):
        D.set_variant(k)
        D.set_state(f)
        D.advance(dt, 2)
        assert rel(D.state(), P.state()) < 1e-6
    D.close()
