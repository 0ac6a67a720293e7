"""dgmx_time_derivative_device in place (F_dev == U_dev) against separate
buffers, on meshes of several waves of CTAs, where a tile that starts late
would read what its neighbours have stored.

Both evaluate the same sums, in another order for the traces in 2-D: the
bound is that of the right-hand side against the oracle (test_gpu_form3.py).
"""
import numpy as np
import pytest

from cases import rotated_box
from oracle import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phys,n,p", [
    ("euler2d", (150, 140), 2), ("euler2d", (90, 70), 5), ("shallow", (150, 140), 3), ("shallow", (60, 60), 8),
    ("ns2d", (90, 70), 4), ("euler3d", (14, 13, 12), 2), ("euler3d", (11, 10, 9), 5), ("ns3d", (11, 10, 9), 3)])
def test_in_place(phys, n, p):
    import torch

    import dgm_b200
    from dgm_b200 import requests
    code, dim = {"euler2d": (1, 2), "ns2d": (2, 2), "shallow": (30, 2), "euler3d": (8, 3), "ns3d": (9, 3)}[phys]
    lo, hi = (-5.0, 5.0) if dim == 2 else (0.0, 2 * np.pi)
    m = rotated_box(dim, n, lo, hi, p, 0, seed=p)
    D = dgm_b200.Domain(m, code, vis=0.01 if phys.startswith("ns") else 0.0, sw_balance=False)
    x, y, z = requests.coordinates(m)
    f = (ics.gaussian_bump(x, y, w=2.0) if phys == "shallow" else
         ics.isentropic_vortex(x, y, beta=2.0, period=(10.0, 10.0)) if dim == 2 else ics.taylor_green(x, y, z, Ma=0.3))
    U = torch.as_tensor(np.ascontiguousarray(f), device="cuda").reshape(D.nf, -1)
    F = torch.empty_like(U)
    D.time_derivative_device(U.data_ptr(), F.data_ptr())
    D.sync()
    scale = F.norm() + U.norm()
    for _ in range(3):
        V = U.clone()
        torch.cuda.synchronize()
        D.time_derivative_device(V.data_ptr(), V.data_ptr())
        D.sync()
        assert float((V - F).norm() / scale) < 1e-12
    D.close()
