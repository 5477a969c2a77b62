"""Exact zeros in the fixed-point forms: where FP64 sums are zero, so are they."""
import numpy as np
import pytest

import oracle as O
from helpers import Case, TOL_TEND, rel_l2

pytestmark = pytest.mark.gpu

both = pytest.mark.parametrize("opt", ["OPT_EVENODD", "OPT_OPT1"])
ORDERS = pytest.mark.parametrize("p,dims", [(1, (5, 4, 3)), (3, (4, 3, 3)), (7, (3, 3, 4)),
                                            (8, (3, 3, 3)), (12, (3, 3, 3))])


def _solver(c, opt, f):
    import sdg
    s = sdg.Solver(c.NeX, c.NeY, c.NeZ, c.p, c.D, c.Lift, opt=getattr(sdg, opt))
    s.upload(*f)
    return s


def _spare_fields(c):
    """A tracer in one element that leaves it in x alone: every x line beside it has
    a face flux, y and z lines have none there."""
    q, u, v, w = [a[: c.nown].copy() for a in (c.q, c.u, c.v, c.w)]
    e = np.arange(c.nown) // c.mesh.Np
    q = np.where(e == 0, q + 0.5, 0.0)
    return e, [q, np.abs(u) + 0.1, np.zeros_like(v), np.zeros_like(w)]


@both
@ORDERS
def test_rows_whose_terms_are_zero_give_zero(opt, p, dims):
    """Operators whose middle rows do not see the faces: beside a front those nodes'
    sums have zero terms only, of either sign, and are zero."""
    c = Case(*dims, p)
    if p < 2:
        pytest.skip("no rows between the ends")
    e, f = _spare_fields(c)
    f[1] = -f[1]  # zeros times a negative velocity are negative zeros
    N = p + 1
    L = c.Lift.reshape(6, N, N, N).copy()
    for face, axis in ((0, 1), (1, 2), (2, 1), (3, 2), (4, 0), (5, 0)):
        mid = [slice(None)] * 3
        mid[axis] = slice(1, N - 1)
        L[(face,) + tuple(mid)] = 0.0
    c.Lift = L.reshape(-1)
    m = c.mesh
    full = []
    for a in f:
        x = np.zeros(m.Np * m.NeA)
        x[: c.nown] = a
        m.update_halo(x)
        full.append(x)
    want = O.cal_tend(m, *full, c.D, c.Dt, c.Lift, O.OPT1)[: c.nown]
    got = _solver(c, opt, f).tendency()
    assert rel_l2(got, want) <= TOL_TEND
    assert np.count_nonzero(want[e != 0]) > 0
    assert np.all(got[want == 0.0] == 0.0)


@both
@ORDERS
@pytest.mark.parametrize("exp", [0, -690])
def test_lines_of_zeros_beside_others(opt, p, dims, exp):
    """A velocity without one of its components, and a tracer of one element, in a
    box whose axes' scale factors lie 2^40 apart, with the tracer also near the
    least magnitude the fixed-point lines take."""
    import sdg
    c = Case(*dims, p)
    L = (1.0, 2.0 ** -40, 1.0)
    m = O.Mesh(*dims, p, c.x1D, L=L)
    e = np.arange(c.nown) // m.Np
    q, u, v, w = [a[: c.nown].copy() for a in (c.q, c.u, c.v, c.w)]
    q = np.ldexp(q + 0.25, exp)
    for f in ([q, u, 0.0 * v, w], [q, u, 0.0 * v, 0.0 * w], [q * (e == 1), u, v * 2.0 ** -40, w]):
        full = []
        for a in f:
            x = np.zeros(m.Np * m.NeA)
            x[: c.nown] = a
            m.update_halo(x)
            full.append(x)
        want = O.cal_tend(m, *full, c.D, c.Dt, c.Lift, O.OPT1)[: c.nown]
        s = sdg.Solver(*dims, p, c.D, c.Lift, opt=getattr(sdg, opt), L=L)
        s.upload(*f)
        assert rel_l2(np.ldexp(s.tendency(), -exp), np.ldexp(want, -exp)) <= TOL_TEND
        sdg.dg_optr_kernel_setup(opt[4:])
        got = np.zeros(m.Np * m.NeA)
        sdg.advect3d_eq_cal_tend(got, *full, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn,
                                 m.Escale, m.Fscale, m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA)
        assert rel_l2(np.ldexp(got[: c.nown], -exp), np.ldexp(want, -exp)) <= TOL_TEND
