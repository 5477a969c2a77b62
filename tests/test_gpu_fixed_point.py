"""The fixed-point FP64 stage where its line scales and its FP64 lines matter:
regions of zeros, magnitudes at the ends of the exponent range, infinities and
NaN, steep fields, anisotropic boxes.  The expected values are the oracle's;
the tolerance is the FP64 form's 1e-12 relative L2 per tendency."""
import numpy as np
import pytest

import oracle as O
from helpers import Case, TOL_TEND, rel_l2

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 6, 7, 8, 12, 15]
both = pytest.mark.parametrize("opt", ["OPT_EVENODD", "OPT_OPT1"])


def _tendencies(c, q, u, v, w, opt):
    """(GPU tendency, oracle tendency) of the owned elements."""
    import sdg
    m = c.mesh
    full = []
    for a in (q, u, v, w):
        f = np.zeros(m.Np * m.NeA)
        f[: c.nown] = a
        m.update_halo(f)
        full.append(f)
    want = O.cal_tend(m, *full, c.D, c.Dt, c.Lift, O.OPT1)[: c.nown]
    s = sdg.Solver(c.NeX, c.NeY, c.NeZ, c.p, c.D, c.Lift, opt=getattr(sdg, opt),
                   precision=sdg.PREC_FP64)
    s.upload(q, u, v, w)
    return s.tendency(), want


def _fields(c):
    return [a[: c.nown].copy() for a in (c.q, c.u, c.v, c.w)]


@both
@pytest.mark.parametrize("p", ORDERS)
@pytest.mark.parametrize("exp", [-1030, -990, -600, 0, 500, 690])
def test_magnitudes_across_the_exponent_range(opt, p, exp):
    c = Case(3, 2, 2, p)
    q, u, v, w = _fields(c)
    q = np.ldexp(q + 0.25, exp)
    got, want = _tendencies(c, q, u, v, w, opt)
    # below 2^-1022 the line sums are subnormal: their absolute spacing counts
    if exp < -1000:
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want)) + 4096 * 5e-324
    else:
        k = -exp
        assert rel_l2(np.ldexp(got, k), np.ldexp(want, k)) <= TOL_TEND


@both
@pytest.mark.parametrize("p", ORDERS)
def test_zero_regions_stay_zero_and_neighbours_agree(opt, p):
    c = Case(4, 3, 2, p)
    q, u, v, w = _fields(c)
    e = np.arange(c.nown) // c.mesh.Np
    q[e != 5] = 0.0
    u[e == 0] = 0.0
    got, want = _tendencies(c, q, u, v, w, opt)
    assert rel_l2(got, want) <= TOL_TEND
    far = np.isin(e, [23, 21])  # share no face with element 5
    assert np.all(got[far] == 0.0) and np.all(want[far] == 0.0)


@both
@pytest.mark.parametrize("p", ORDERS)
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_reach_the_nodes_they_reach_in_the_oracle(opt, p, bad):
    c = Case(3, 3, 2, p)
    q, u, v, w = _fields(c)
    n = 4 * c.mesh.Np + c.mesh.Np // 2  # an inner node of element 4
    q[n] = bad
    w[n] = 0.75
    got, want = _tendencies(c, q, u, v, w, opt)
    fine = np.isfinite(want)
    assert 0 < np.count_nonzero(~fine) < want.size
    if p % 2 == 0 and opt == "OPT_EVENODD":
        # n is the middle of its three lines, and D(mid,mid) = 0: the even-odd
        # rows leave that term out where the oracle forms 0 * inf
        assert not fine[n]
        got[n], want[n], fine[n] = 0.0, 0.0, True
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_l2(got[fine], want[fine]) <= TOL_TEND


@both
@pytest.mark.parametrize("p", ORDERS)
def test_steep_fields_and_uneven_axes(opt, p):
    import sdg
    c = Case(5, 1, 2, p)
    q, u, v, w = _fields(c)
    r = np.random.RandomState(p)
    q = np.exp(-40.0 * r.rand(q.size))
    u *= np.exp(20.0 * (r.rand(q.size) - 0.5))
    v *= 1e-9
    got, want = _tendencies(c, q, u, v, w, opt)
    assert rel_l2(got, want) <= TOL_TEND
    # a box whose scale factors the coefficients cannot hold: lines in FP64
    tiny = 2.0 ** -220
    a = sdg.Solver(3, 2, 2, p, c.D, c.Lift, opt=getattr(sdg, opt), L=(tiny, tiny, tiny))
    b = sdg.Solver(3, 2, 2, p, c.D, c.Lift, opt=getattr(sdg, opt))
    c = Case(3, 2, 2, p)
    for s in (a, b):
        s.upload(*_fields(c))
    assert rel_l2(a.tendency() * tiny, b.tendency()) <= TOL_TEND
