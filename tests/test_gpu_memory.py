"""What a solver leaves of the device's memory."""
import ctypes as C

import numpy as np
import pytest

from helpers import Case

pytestmark = pytest.mark.gpu


def _free():
    rt = C.CDLL("libcudart.so.13")
    a, b = C.c_size_t(), C.c_size_t()
    assert rt.cudaMemGetInfo(C.byref(a), C.byref(b)) == 0
    return a.value


@pytest.mark.parametrize("opt", ["OPT_OPT1", "OPT_GENERAL"])
def test_velocity_factors_leave_room_for_the_callers_next_allocation(opt):
    """With little more left than the solver's own buffers, the velocity factors
    (48 bytes a DOF at p = 1, as much as those) are left out, a further allocation
    of their size succeeds, and the steps have the same bits."""
    import sdg
    c = Case(64, 64, 65, 1)
    f = [a[: c.nown].copy() for a in (c.q, c.u, c.v, c.w)]
    make = lambda: sdg.Solver(64, 64, 65, 1, c.D, c.Lift, opt=getattr(sdg, opt))
    s = make()  # loads the kernels
    s.upload(*f)
    s.step(c.dt, 2)
    s.tendency()
    want = s.download()
    s.close()
    factors = 48 * c.nown
    own = 56 * c.nown + (16 << 20)
    ballast = sdg.DeviceArray(n=_free() - own - 3 * factors, dtype=np.uint8)
    s = make()
    more = sdg.DeviceArray(n=5 * factors // 2, dtype=np.uint8)
    s.upload(*f)
    s.step(c.dt, 2)
    assert np.array_equal(s.download(), want)
    more.free()
    s.tendency()
    s.close()
    ballast.free()
