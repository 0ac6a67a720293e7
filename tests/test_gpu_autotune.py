"""What dgmx_autotune times for Navier-Stokes: all kernels of a stage in the
handle's own form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tuned(precision, tensor=False):
    import dgm_b200
    from dgm_b200 import meshgen, requests
    m = meshgen.box(3, (10, 10, 10), 0.0, 2 * np.pi, 5)
    D = dgm_b200.Domain(m, dgm_b200.NS3D, vis=1e-2, precision=precision)
    D.set_state(requests.taylor_green(*requests.coordinates(m), Ma=0.3))
    if tensor:
        D.set_tensor_contractions(True)
    n0 = D.launch_count()
    rows, pick = D.autotune(reps=10)
    launches = (D.launch_count() - n0) / (len(rows) * 12)   # 2 + 10 stages per tile
    D.advance(1e-4, 1)
    D.close()
    return rows[:, 3], pick, launches


def test_navier_stokes_forms():
    """The FP32 viscous form's flux kernel is at least half of a stage (with it
    left out the tuner read half of FP64's times); the 3xTF32 form has three
    kernels, the same ones for every tile."""
    import dgm_b200
    us, pick, launches = tuned(dgm_b200.FP64)
    us32, pick32, launches32 = tuned(dgm_b200.MIXED)
    _, _, launches_tc = tuned(dgm_b200.MIXED, True)
    assert (launches, launches32, launches_tc) == (2, 2, 3)
    assert pick == np.argmin(us) and pick32 == np.argmin(us32)
    assert us32.min() > 0.6 * us.min()
