"""The FP32 viscous form of Navier-Stokes (precision = MIXED) at every compiled
order and tile: its distance from the FP64 handle of the same mesh, and what
the tuner times for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [(2, p, q) for p in range(1, 9) for q in (p + 1, p + 2)] + [(3, 1, 3)] + \
         [(3, p, q) for p in range(2, 8) for q in (p + 1, p + 2)]


def flow(x, y, z, dim, V):
    """A Taylor-Green flow carried along at the speed V."""
    u = [np.sin(x) * np.cos(y) * np.cos(z) + V, -np.cos(x) * np.sin(y) * np.cos(z) - V, 0.0 * x + 0.5 * V][:dim]
    r, P = 1 + 0.1 * np.sin(x), 8.0 + (np.cos(2 * x) + np.cos(2 * y)) / 4
    return np.stack([r] + [r * a for a in u] + [2.5 * P + 0.5 * r * sum(a * a for a in u)])


@pytest.mark.parametrize("dim,p,q", ORDERS)
def test_viscous_part_at_any_speed(dim, p, q):
    """Distance of the momentum equations' viscous part from FP64, whatever the
    flow's mean speed: the gradient does not see it.  A second derivative
    amplifies a rounding of 2^-24 by about (p+1)^4; twice that (observed: 0.4
    of the bound at most).  Velocities rounded at full size miss it."""
    import dgm_b200
    from dgm_b200 import meshgen, requests
    n = 12 if dim == 2 else (5 if p < 5 else 3)
    m = meshgen.box(dim, (n,) * dim, 0.0, 2 * np.pi, p, q)
    c = requests.coordinates(m)
    code = dgm_b200.NS2D if dim == 2 else dgm_b200.NS3D
    for V in (0.0, 4.0, 32.0):
        U = flow(*c, dim, V)
        D = dgm_b200.Domain(m, code, flux="roe", vis=0.02, precision=dgm_b200.MIXED)
        R = dgm_b200.Domain(m, code, flux="roe", vis=0.02)
        E = dgm_b200.Domain(m, code, flux="roe", vis=0.0)
        F, I = R.time_derivative(U), E.time_derivative(U)
        for k in range(D.variant_count()):
            D.set_variant(k)
            G = D.time_derivative(U)
            for f in (1, 2):
                d = np.linalg.norm(G[f] - F[f]) / np.linalg.norm(F[f] - I[f])
                assert d < 2.0 ** -23 * (p + 1) ** 4, (V, k, f, d)
        for h in (D, R, E):
            h.close()


def test_taylor_green_24():
    """Ten LSRK14 steps of the 24^3, p = 7 Taylor-Green vortex: per-field
    distance from FP64 no larger than when the states were rounded less their
    means (1.2e-9, 7.7e-8, 8.3e-8, 2.4e-5, 1.6e-9; observed here 2.7e-10, 2.2e-8,
    2.0e-8, 6.4e-6, 3.7e-10)."""
    import dgm_b200
    from dgm_b200 import meshgen, requests
    m = meshgen.box(3, (24,) * 3, 0.0, 2 * np.pi, 7, 9)
    U = requests.taylor_green(*requests.coordinates(m), Ma=0.1)
    S = []
    for precision in (dgm_b200.FP64, dgm_b200.MIXED):
        D = dgm_b200.Domain(m, dgm_b200.NS3D, flux="roe", vis=1.0 / 1600, precision=precision)
        D.set_state(U)
        D.advance(7.9333e-4, 10)
        S.append(D.state())
        D.close()
    for k, bound in enumerate((1.19e-9, 7.7e-8, 8.3e-8, 2.4e-5, 1.62e-9)):
        assert np.linalg.norm(S[1][k] - S[0][k]) / np.linalg.norm(S[0][k]) < bound, k
