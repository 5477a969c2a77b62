"""Device calls whose outputs lie over their inputs, as a caller short of memory
makes them.  The expected values are the oracle's or long double's on the inputs
as they were; the tolerance is 1e-12 relative L2."""
import itertools

import numpy as np
import pytest

import oracle as O
from helpers import Case, TOL_TEND, rel_l2

pytestmark = pytest.mark.gpu


def _along(a, M, axis, N):
    """sum_l M(i, l) a(.., l, ..) over elements of N^3 values, M given (out, in)."""
    a = a.reshape(-1, N, N, N).astype(np.longdouble)
    return np.moveaxis(np.tensordot(a, M.astype(np.longdouble), axes=([3 - axis], [1])), -1,
                       3 - axis).reshape(-1).astype(float)


@pytest.mark.parametrize("p,nelem", [(2, 600), (3, 2400), (7, 301), (8, 207), (11, 40), (15, 40)])
@pytest.mark.parametrize("order", list(itertools.permutations(range(3))))
def test_divlike_outputs_over_its_inputs(p, nelem, order):
    """Output direction d over input direction order[d], on both sides of the
    element counts that choose the kernel."""
    import sdg
    N = p + 1
    r = np.random.RandomState(p)
    D, Dt = r.randn(N * N), r.randn(N * N)
    f = [r.randn(nelem * N ** 3) for _ in range(3)]
    d = [sdg.DeviceArray(x) for x in f]
    m, mt = sdg.DeviceArray(D), sdg.DeviceArray(Dt)
    out = [d[k] for k in order]
    for opt in (sdg.OPT_OPT1, sdg.OPT_GENERAL):
        for x, y in zip(d, f):
            x.upload(y)
        assert sdg.lib.sdg_tensorprod_divlike_dirXYZ_dev(
            out[0].ptr, out[1].ptr, out[2].ptr, m.ptr, mt.ptr, d[0].ptr, d[1].ptr, d[2].ptr, N,
            nelem, opt, None) == 0
        for axis in range(3):
            M = D.reshape(N, N).T if axis == 0 else Dt.reshape(N, N)
            assert rel_l2(out[axis].numpy(), _along(f[axis], M, axis, N)) <= TOL_TEND


@pytest.mark.parametrize("p,nelem", [(3, 2400), (8, 207), (15, 40)])
@pytest.mark.parametrize("over", [0, 1, 2])
def test_gradlike_and_a_direction_over_the_field(p, nelem, over):
    import sdg
    N = p + 1
    r = np.random.RandomState(p)
    D, Dt, f = r.randn(N * N), r.randn(N * N), r.randn(nelem * N ** 3)
    want = [_along(f, D.reshape(N, N).T if k == 0 else Dt.reshape(N, N), k, N) for k in range(3)]
    m, mt = sdg.DeviceArray(D), sdg.DeviceArray(Dt)
    d = [sdg.DeviceArray(f) for _ in range(3)]
    assert sdg.lib.sdg_tensorprod_gradlike_dirXYZ_dev(d[0].ptr, d[1].ptr, d[2].ptr, m.ptr, mt.ptr,
                                                      d[over].ptr, N, nelem, None) == 0
    for k in range(3):
        assert rel_l2(d[k].numpy(), want[k]) <= TOL_TEND
    x = sdg.DeviceArray(f)
    M = m if over == 0 else mt
    assert sdg.lib.sdg_element_matvec_dir_dev(over + 1, x.ptr, M.ptr, x.ptr, N, nelem, None) == 0
    assert rel_l2(x.numpy(), want[over]) <= TOL_TEND
