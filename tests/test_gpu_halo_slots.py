"""The time loop on the reference's arrays where the caller keeps some halo slots:
a boundary condition in slots that halo_src_map does not cover.  The expected
values are the oracle's; the tolerance is 1e-12 relative L2."""
import copy

import numpy as np
import pytest

import oracle as O
from helpers import Case, TOL_TEND, rel_l2

pytestmark = pytest.mark.gpu


def _step(c, m, q, nstep, opt):
    import sdg
    return sdg.advect3d_eq_step(q, c.u, c.v, c.w, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn,
                                m.Escale, m.Fscale, m.halo_src_map, m.Nq, m.Np, m.NfpTot, m.Ne,
                                m.NeA, m.NhaloNode, c.dt, nstep, opt)


def _open_mesh(c, kind):
    """The periodic mesh with the -x boundary faces reading slots of their own
    ("some"), or with every halo slot the caller's ("all")."""
    m = copy.copy(c.mesh)
    q = c.q.copy()
    own, ids = m.Np * m.Ne, np.arange(m.Np * m.NeA)
    r = np.random.RandomState(c.p)
    if kind == "all":
        m.NhaloNode = 0
        q[own:] = r.rand(ids.size - own)
        return m, q
    free = ids[own + m.NhaloNode:]
    assert free.size >= m.Nfp * m.NeY * m.NeZ
    q[free] = 1.0 + r.rand(free.size)
    P = m.VMapP.reshape(m.Ne, 6, m.Nfp).copy()
    at = 0
    for e in range(0, m.Ne, m.NeX):  # elements at x = 0, face -x
        P[e, 3] = free[at: at + m.Nfp] + 1
        at += m.Nfp
    m.VMapP = P.reshape(-1)
    return m, q


@pytest.mark.parametrize("p,dims", [(1, (5, 4, 3)), (3, (4, 3, 2)), (7, (3, 2, 4)), (12, (2, 2, 3))])
@pytest.mark.parametrize("opt", ["OPT_OPT1", "OPT_GENERAL"])
@pytest.mark.parametrize("kind", ["some", "all"])
def test_halo_slots_the_caller_keeps(p, dims, opt, kind):
    import sdg
    c = Case(*dims, p)
    m, q = _open_mesh(c, kind)
    got = _step(c, m, q, 2, getattr(sdg, opt))
    want = q.copy()
    O.run(m, want, c.u, c.v, c.w, c.D, c.Dt, c.Lift, c.dt, 2, getattr(O, opt[4:]))
    assert rel_l2(want[: c.nown], c.oracle_run(2)) > 1e-4  # the boundary counts
    assert rel_l2(got[: c.nown], want[: c.nown]) <= TOL_TEND
    kept = slice(m.Np * m.Ne + m.NhaloNode, None)
    assert np.array_equal(got[kept], q[kept])


def test_the_evenodd_loop_still_refuses_them():
    import sdg
    c = Case(4, 3, 2, 3)
    m, q = _open_mesh(c, "some")
    with pytest.raises(sdg.SdgError) as e:
        _step(c, m, q, 1, sdg.OPT_EVENODD)
    assert e.value.status == sdg.ERR_MESH
