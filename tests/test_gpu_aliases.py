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


@pytest.mark.parametrize("opt", ["OPT_EVENODD", "OPT_OPT1"])
@pytest.mark.parametrize("p,dims", [(3, (4, 5, 3)), (3, (15, 14, 13)), (7, (8, 7, 8)),
                                    (13, (3, 5, 4))])
@pytest.mark.parametrize("over", ["q", "u", "v", "w", "Escale"])
def test_tendency_over_one_of_its_fields(opt, p, dims, over):
    """dqdt in place of a field (or of Escale's x part), on both sides of the
    small-mesh rule; an EVENODD call still reports operators without the
    symmetries."""
    import sdg
    c = Case(*dims, p)
    m = c.mesh
    want = c.oracle_tend(O.OPT1)
    A = sdg.DeviceArray
    f = {"q": A(c.q), "u": A(c.u), "v": A(c.v), "w": A(c.w), "Escale": A(m.Escale)}
    D, Dt, L, M, P, n, S = [A(a) for a in (c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn,
                                           m.Fscale)]
    flux, err = A(n=m.NfpTot * m.Ne), A(np.zeros(1, dtype=np.int32))

    def call(D):
        return sdg.lib.sdg_advect3d_eq_cal_tend_dev(
            f[over].ptr, f["q"].ptr, f["u"].ptr, f["v"].ptr, f["w"].ptr, D.ptr, Dt.ptr, L.ptr,
            M.ptr, P.ptr, n.ptr, f["Escale"].ptr, S.ptr, m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA,
            getattr(sdg, opt), flux.ptr, err.ptr, None)

    assert call(D) == 0
    assert rel_l2(f[over].numpy()[: c.nown], want) <= TOL_TEND
    assert err.numpy()[0] == 0
    bad = c.D.copy()
    bad[1] *= 1.5
    assert call(A(bad)) == 0
    assert err.numpy()[0] == (2 if opt == "OPT_EVENODD" else 0)
