"""Tendencies node by node where a node's value exceeds all others of its lines by
far: its own derivative does not see it (D has a zero there) and is formed of the
small values.  Bounds: FP64 sums to 3 (N + 2) + 20 roundings of 2^-53 of their terms'
magnitudes (three lines; the face fluxes, the lift and the sum of the three); in
fixed point in addition (1.5 N + 4) 2^-59 of a row's magnitudes times the largest
value, three times.  The expected values are the oracle's, which has the first
error as well."""
import numpy as np
import pytest

import oracle as O
from helpers import Case

pytestmark = pytest.mark.gpu


def _terms(c, f):
    """Sum of the magnitudes of a node's terms."""
    m, N = c.mesh, c.p + 1
    q, u, v, w = [np.abs(x) for x in f]
    D = np.abs(c.D.reshape(N, N).T)
    es = m.Escale.reshape(3, m.Ne, N, N, N)
    own = m.Np * m.Ne
    out = 0.0
    for d, vel in enumerate((u, v, w)):
        F = (q * vel)[:own].reshape(m.Ne, N, N, N)
        out = out + es[d] * np.moveaxis(np.tensordot(F, D, axes=([3 - d], [1])), -1, 3 - d)
    M, P = m.VMapM - 1, m.VMapP - 1
    n = np.abs(m.normal_fn.reshape(3, -1))
    vM, vP = [u[i] * n[0] + v[i] * n[1] + w[i] * n[2] for i in (M, P)]
    alpha = 0.5 * (vM + vP)
    g = 0.5 * m.Fscale * (q[P] * vP + q[M] * vM + alpha * (q[P] + q[M]))
    g = g.reshape(m.Ne, 6, N, N)
    L = np.abs(c.Lift.reshape(6, N, N, N))
    for face in range(6):
        # Lift(i,j,k,face) times the flux of the face node beside (i,j,k)
        side = {0: g[:, 0][:, :, None, :], 2: g[:, 2][:, :, None, :], 1: g[:, 1][..., None],
                3: g[:, 3][..., None], 4: g[:, 4][:, None], 5: g[:, 5][:, None]}[face]
        out = out + L[face] * side
    return out.reshape(-1)


def _spiked(c, at):
    """1e-12 and one node of every second element at `at` (i, j, k) of order one."""
    m, N = c.mesh, c.p + 1
    r = np.random.RandomState(c.p)
    q = 1e-12 * (0.5 + r.rand(c.nown))
    e = np.arange(0, m.Ne, 2)
    node = e * m.Np + at[0] + N * at[1] + N * N * at[2]
    q[node] = 0.5 + r.rand(e.size)
    f = []
    for a in (q, c.u[: c.nown], c.v[: c.nown], c.w[: c.nown]):
        x = np.zeros(m.Np * m.NeA)
        x[: c.nown] = a
        m.update_halo(x)
        f.append(x)
    return f, node


def _check(c, f, spikes, got, D):
    m, N = c.mesh, c.p + 1
    Dt = np.ascontiguousarray(D.reshape(N, N).T).reshape(-1)
    want = O.cal_tend(m, *f, D, Dt, c.Lift, O.OPT1)[: c.nown]
    terms = _terms(c, f)
    top = max(np.abs(f[0]).max() * np.abs(x).max() for x in f[1:])
    rows = np.abs(c.D.reshape(N, N)).sum(axis=0).max() + 2 * np.abs(c.Lift).max()
    bound = 2 * (3 * (N + 2) + 20) * 2.0 ** -53 * terms
    loose = 3 * (1.5 * N + 4) * 2.0 ** -59 * rows * m.Escale.max() * 2 * top
    away = np.full(c.nown, loose)
    away[spikes] = 0.0
    assert np.all(terms[spikes] < 1e-6 * terms.max())
    assert np.all(np.abs(got - want) <= bound + away)


def _tendencies(c, f, opt):
    import sdg
    m = c.mesh
    s = sdg.Solver(c.NeX, c.NeY, c.NeZ, c.p, c.D, c.Lift, opt=getattr(sdg, opt))
    s.upload(*[x[: c.nown] for x in f])
    yield s.tendency()
    sdg.dg_optr_kernel_setup(opt[4:])
    got = np.zeros(m.Np * m.NeA)
    sdg.advect3d_eq_cal_tend(got, *f, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn, m.Escale,
                             m.Fscale, m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA)
    yield got[: c.nown]


@pytest.mark.parametrize("p,dims", [(2, (20, 18, 17)), (3, (15, 14, 13)), (7, (8, 7, 8)),
                                    (8, (7, 7, 6)), (13, (3, 5, 4))])
@pytest.mark.parametrize("opt", ["OPT_OPT1", "OPT_GENERAL"])
def test_a_spike_inside_an_element(p, dims, opt):
    c = Case(*dims, p)
    f, spikes = _spiked(c, (1, p // 2, p - 1))
    for got in _tendencies(c, f, opt):
        _check(c, f, spikes, got, c.D)


@pytest.mark.parametrize("p,dims", [(2, (20, 18, 17)), (4, (10, 9, 9)), (8, (7, 7, 6)),
                                    (12, (4, 4, 5))])
def test_a_spike_in_the_middle_with_evenodd_pairs(p, dims):
    """The pairs' D is the given one's antisymmetric part, whose middle entry is zero
    where the given one's may be some 1e-16."""
    c = Case(*dims, p)
    f, spikes = _spiked(c, (p // 2, p // 2, p // 2))
    D = 0.5 * (c.D - c.D[::-1])
    for got in _tendencies(c, f, "OPT_EVENODD"):
        _check(c, f, spikes, got, D)


@pytest.mark.parametrize("p,dims", [(3, (15, 14, 13)), (7, (8, 7, 8)), (13, (3, 5, 4))])
@pytest.mark.parametrize("kind", ["lumped", "sparse"])
def test_operators_with_zeros(p, dims, kind):
    """A lift that only the face's own nodes see, under a jump of 1e12; a derivative
    matrix with zeros: each node against its own terms."""
    c = Case(*dims, p)
    m, N = c.mesh, p + 1
    if kind == "lumped":
        L = c.Lift.reshape(6, N, N, N).copy()
        for face, axis, at in ((0, 1, 0), (1, 2, N - 1), (2, 1, N - 1), (3, 2, 0), (4, 0, 0),
                               (5, 0, N - 1)):
            x = np.moveaxis(L[face], axis, 0)
            x[np.arange(N) != at] = 0.0
        c.Lift = L.reshape(-1)
    else:
        D = c.D.reshape(N, N).copy()
        D[np.abs(np.subtract.outer(np.arange(N), np.arange(N))) > 1] = 0.0
        c.D, c.Dt = D.reshape(-1), np.ascontiguousarray(D.T).reshape(-1)
    r = np.random.RandomState(p)
    e = np.arange(c.nown) // m.Np
    q = np.where(e % 2 == 0, 1.0, 1e-12) * (0.5 + r.rand(c.nown))
    f = []
    for a in (q, c.u[: c.nown], c.v[: c.nown], c.w[: c.nown]):
        x = np.zeros(m.Np * m.NeA)
        x[: c.nown] = a
        m.update_halo(x)
        f.append(x)
    want = O.cal_tend(m, *f, c.D, c.Dt, c.Lift, O.OPT1)[: c.nown]
    terms = _terms(c, f)
    # a dense row holds its line's largest value to 2^-10 of the row's magnitudes
    extra = 3 * (1.5 * N + 4) * 2.0 ** -59 * 2.0 ** 10 * 16
    for got in _tendencies(c, f, "OPT_OPT1"):
        assert np.all(np.abs(got - want) <= (2 * (3 * (N + 2) + 20) * 2.0 ** -53 + extra) * terms)
