"""Calls at the edges of the fixed-point forms' ranges: face fluxes and scale
factors whose exponents lie far apart, on the reference's arrays.  The expected
values are the oracle's; the tolerance is the FP64 form's 1e-12 relative L2 per
tendency."""
import copy

import numpy as np
import pytest

import oracle as O
from helpers import Case, TOL_TEND, rel_l2

pytestmark = pytest.mark.gpu

both = pytest.mark.parametrize("opt", ["OPT_EVENODD", "OPT_OPT1"])


def _cal_tend(c, m, q, opt, D=None, Lift=None):
    """(GPU tendency, oracle tendency) of state q on mesh m."""
    import sdg
    D = c.D if D is None else D
    Dt = np.ascontiguousarray(D.reshape(m.Nq, m.Nq).T).reshape(-1)
    Lift = c.Lift if Lift is None else Lift
    want = O.cal_tend(m, q, c.u, c.v, c.w, D, Dt, Lift, O.OPT1)[: c.nown]
    sdg.dg_optr_kernel_setup(opt[4:])
    got = np.zeros(m.Np * m.NeA)
    sdg.advect3d_eq_cal_tend(got, q, c.u, c.v, c.w, D, Dt, Lift, m.VMapM, m.VMapP, m.normal_fn,
                             m.Escale, m.Fscale, m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA)
    return got[: c.nown], want


def _loop(c, m, q, dt, nstep, opt):
    """(GPU state, oracle state) after nstep steps of the loop on mesh m."""
    import sdg
    got = sdg.advect3d_eq_step(q, c.u, c.v, c.w, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn,
                               m.Escale, m.Fscale, m.halo_src_map, m.Nq, m.Np, m.NfpTot, m.Ne,
                               m.NeA, m.NhaloNode, dt, nstep, getattr(sdg, opt))[: c.nown]
    want = q.copy()
    O.run(m, want, c.u, c.v, c.w, c.D, c.Dt, c.Lift, dt, nstep, O.OPT1)
    return got, want[: c.nown]


def _agree(got, want):
    fine = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_l2(got[fine], want[fine]) <= TOL_TEND


# element counts on the fixed-point side of the small-mesh rule
MESHES = pytest.mark.parametrize("p,dims", [(3, (15, 14, 13)), (7, (8, 7, 8)), (8, (7, 7, 6)),
                                            (13, (3, 5, 4))])


@both
@MESHES
@pytest.mark.parametrize("length", [1.0, 30.0, 1e4])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_neighbours_reach_elements_of_any_size(opt, p, dims, length, bad):
    """A face value that is not finite reaches the element beyond the face
    whatever the elements' size: with Escale = 2 / h far above one, near and far
    below a half."""
    c = Case(*dims, p)
    m = O.Mesh(*dims, p, c.x1D, L=(length,) * 3)
    q = c.q.copy()
    q[m.Np * (m.Ne // 2)] = bad  # a corner: on the -x, -y and -z face
    m.update_halo(q)
    with np.errstate(all="ignore"):
        got, want = _cal_tend(c, m, q, opt)
        beyond = [i for i in range(m.Ne) if i != m.Ne // 2
                  and not np.isfinite(want[i * m.Np:(i + 1) * m.Np]).all()]
        assert len(beyond) == 3
        _agree(got, want)
        _agree(*_loop(c, m, q, 0.5 * c.dt * length, 1, opt))


@both
@MESHES
def test_huge_face_fluxes_over_small_scale_factors(opt, p, dims):
    """Face fluxes of 2^1011 beside Escale of 2^-16: their ratio passes the
    largest double, every result is finite."""
    c = Case(*dims, p)
    m = copy.copy(c.mesh)
    m.Escale = m.Escale * 2.0 ** -20
    q = c.q.copy()
    q[m.Np * (m.Ne // 2 + 1) - 1] = 2.0 ** 1008  # flows out through three faces
    m.update_halo(q)
    got, want = _cal_tend(c, m, q, opt)
    assert np.isfinite(want).all() and np.abs(want).max() > 2.0 ** 1005
    k = 2.0 ** -900
    _agree(got * k, want * k)


@both
@MESHES
def test_scales_that_lie_apart_only_together(opt, p, dims):
    """State, Escale and operators whose exponents each lie within the fixed-point
    range and add up past a double's: the largest results near 2^-1005, those of
    the tracer's tail subnormal."""
    c = Case(*dims, p)
    m = copy.copy(c.mesh)
    m.Escale, m.Fscale = m.Escale * 2.0 ** -148, m.Fscale * 2.0 ** -148
    q = c.q * 2.0 ** -685
    D, Lift = c.D * 2.0 ** -180, c.Lift * 2.0 ** -180
    got, want = _cal_tend(c, m, q, opt, D, Lift)
    assert 0.0 < np.abs(want).max() < 2.0 ** -995
    assert np.count_nonzero(np.abs(want) < 2.0 ** -1022) > 0
    _agree(np.ldexp(got, 1000), np.ldexp(want, 1000))


@both
@pytest.mark.parametrize("p,dims", [(1, (9, 8, 7)), (2, (6, 7, 5)), (3, (15, 14, 13)),
                                    (7, (8, 7, 8)), (8, (7, 7, 6)), (13, (3, 5, 4)),
                                    (15, (3, 4, 3))])
@pytest.mark.parametrize("kind", ["mild", "wide", "edges", "nonfinite"])
def test_escale_per_node(opt, p, dims, kind):
    """Escale that varies over an element's nodes: mildly, over 60 powers of two,
    with zeros, negative values and exponents past the folded ones, and with an
    infinity and a NaN; beside elements of one Escale and elements of zeros.  A
    result's error is held against its own terms where they differ in size: the
    sums' bound on the element times its Escale, 1e-12 of it."""
    c = Case(*dims, p)
    m = copy.copy(c.mesh)
    r = np.random.RandomState(p)
    es = m.Escale.reshape(3, m.Ne, m.Np).copy()
    curved = np.arange(m.Ne) % 3 == 1
    f = 0.5 + r.rand(3, m.Ne, m.Np)
    if kind == "wide":
        f = np.ldexp(f, r.randint(-30, 31, f.shape))
    if kind == "edges":
        f[:, :, 0], f[:, :, 1], f[:, :, 2], f[:, :, 3] = 0.0, -1.0, 2.0 ** 160, 2.0 ** -160
    if kind == "nonfinite":
        f[1, 1, 0], f[2, 4, 5] = np.inf, np.nan
    es[:, curved] *= f[:, curved]
    m.Escale = es.reshape(-1)
    q = c.q.copy()
    q[: c.nown].reshape(m.Ne, m.Np)[np.arange(m.Ne) % 5 == 0] = 0.0
    m.update_halo(q)
    with np.errstate(all="ignore"):
        got, want = _cal_tend(c, m, q, opt)
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fine)
        N = p + 1
        rows = np.abs(c.D.reshape(N, N)).sum(axis=0).max() + 2 * np.abs(c.Lift).max()
        vel = max(np.abs(a).max() for a in (c.u, c.v, c.w))
        size = rows * vel * np.abs(c.q).max() * (np.abs(es).sum(axis=0) + 3 * m.Fscale.max())
    assert np.all(np.abs(got - want)[fine] <= 1e-12 * size.reshape(-1)[fine])
    if kind in ("mild", "wide"):
        _agree(*_loop(c, m, q, 0.25 * c.dt / f.max(), 1, opt))
