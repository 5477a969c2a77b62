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


def _mesh_arrays(c, scale_of_element=None):
    m = c.mesh
    es = m.Escale.copy().reshape(3, m.Ne, m.Np)
    if scale_of_element is not None:
        es *= scale_of_element.reshape(3, m.Ne, -1)
    return es.reshape(-1)


@both
@pytest.mark.parametrize("p,dims", [(1, (9, 8, 7)), (2, (6, 7, 5)), (5, (10, 9, 9)),
                                    (7, (8, 7, 8)), (8, (7, 7, 6)), (13, (3, 5, 4)),
                                    (15, (3, 4, 3))])
@pytest.mark.parametrize("kind", ["affine", "own", "curved", "bad"])
def test_tendency_and_loop_on_reference_arrays(opt, p, dims, kind):
    """cal_tend and the time loop with one Escale for the mesh, one an element,
    one a node in every third element, and a non-finite state, on meshes on
    both sides of the small-mesh rule, against the oracle on the same arrays."""
    import copy

    import sdg
    c = Case(*dims, p)
    m = copy.copy(c.mesh)
    r = np.random.RandomState(p)
    if kind == "own":
        m.Escale = _mesh_arrays(c, 0.5 + r.rand(3, m.Ne, 1))
    elif kind == "curved":
        f = 0.5 + r.rand(3, m.Ne, m.Np)
        f[:, np.arange(m.Ne) % 3 != 0, :] = 1.0
        m.Escale = _mesh_arrays(c, f)
    q = c.q.copy()
    if kind == "bad":
        q[m.Np * (m.Ne // 2)] = np.inf
        m.update_halo(q)
    want = O.cal_tend(m, q, c.u, c.v, c.w, c.D, c.Dt, c.Lift, O.OPT1)[: c.nown]
    sdg.dg_optr_kernel_setup(opt[4:])
    got = np.zeros(m.Np * m.NeA)
    sdg.advect3d_eq_cal_tend(got, q, c.u, c.v, c.w, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP,
                             m.normal_fn, m.Escale, m.Fscale, m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA)
    got = got[: c.nown]
    fine = np.isfinite(want)
    assert np.array_equal(np.isfinite(got), fine)
    assert rel_l2(got[fine], want[fine]) <= TOL_TEND
    if kind == "bad":
        return
    args = (m.VMapM, m.VMapP, m.normal_fn, m.Escale, m.Fscale, m.halo_src_map, m.Nq, m.Np,
            m.NfpTot, m.Ne, m.NeA, m.NhaloNode)
    a = sdg.advect3d_eq_step(q, c.u, c.v, c.w, c.D, c.Dt, c.Lift, *args, 0.5 * c.dt, 2,
                             getattr(sdg, opt))
    qq = q.copy()
    O.run(m, qq, c.u, c.v, c.w, c.D, c.Dt, c.Lift, 0.5 * c.dt, 2, O.OPT1)
    assert rel_l2(a[: c.nown], qq[: c.nown]) <= TOL_TEND


@both
@pytest.mark.parametrize("p", [1, 6, 11, 14])
def test_loop_with_the_least_scratch(opt, p):
    """Scratch without room for the operator tables (all that was asked for
    before there were any) still runs, to the same result."""
    import sdg
    c = Case(3, 2, 2, p)
    m = c.mesh
    A = sdg.DeviceArray
    need = int(sdg.lib.sdg_advect3d_eq_step_scratch_bytes(m.Nq, m.Ne))
    N, H, HR = m.Nq, m.Nq // 2, (m.Nq + 1) // 2
    te = H * H + HR * H + (N & 1) * H + HR + H
    up = lambda n: (n + 255) // 256 * 256
    least = (2 * up(8 * m.Np * m.Ne) + up(16 * m.NfpTot * m.Ne) + up(8 * m.NfpTot * m.Ne)
             + up(24 * te) + up(32 * m.Ne))
    assert least < need
    arrs = [A(a) for a in (c.u, c.v, c.w, c.D, c.Dt, c.Lift, m.VMapM, m.VMapP, m.normal_fn,
                           m.Escale, m.Fscale, m.halo_src_map)]
    out = []
    for size, want in ((need, 0), (least, 0), (least - 1, sdg.ERR_INVALID_ARG)):
        q, scratch, err = A(c.q), A(n=size, dtype=np.uint8), A(np.zeros(1, dtype=np.int32))
        st = sdg.lib.sdg_advect3d_eq_step_dev(
            q.ptr, *[a.ptr for a in arrs], m.Nq, m.Np, m.NfpTot, m.Ne, m.NeA, m.NhaloNode, c.dt,
            2, getattr(sdg, opt), scratch.ptr, size, err.ptr, None)
        assert st == want
        if st == 0:
            assert err.numpy()[0] == 0
            out.append(q.numpy()[: c.nown])
    assert rel_l2(out[1], out[0]) <= TOL_TEND


@pytest.mark.parametrize("p,nelem", [(1, 20011), (2, 5600), (3, 2400), (6, 441), (7, 301), (8, 207),
                                     (10, 113), (11, 1), (12, 5), (15, 3), (15, 40)])
def test_contractions_in_fixed_point(p, nelem):
    """divlike, gradlike and the single directions on both sides of the element
    counts that choose the kernel: unsymmetric matrices, steep fields, zero
    lines, and lines with infinities, NaN and extreme magnitudes."""
    import sdg
    N = p + 1
    r = np.random.RandomState(p)
    D, Dt = r.randn(N * N), r.randn(N * N)
    D[0] = 0.0
    f = [np.exp(-20 * r.rand(nelem * N ** 3)) * r.randn(nelem * N ** 3) for _ in range(3)]
    f[0][: N ** 3] = 0.0
    f[1][5] = np.inf
    f[2][N ** 3 - 1] = np.nan
    f[0][-1] = 1e300
    f[1][-2] = 1e-300

    def along(a, axis):
        a = a.reshape(nelem, N, N, N).astype(np.longdouble)
        M = (D if axis == 0 else Dt).reshape(N, N).astype(np.longdouble)
        M = M.T if axis == 0 else M  # (out, in)
        return np.moveaxis(np.tensordot(a, M, axes=([3 - axis], [1])), -1, 3 - axis).reshape(-1)

    def check(got, want):
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fine)
        # each line against its own size: 1e-12 of the sum of its terms' magnitudes
        assert rel_l2(got[fine & (np.abs(want) < 1e200)],
                      want[fine & (np.abs(want) < 1e200)].astype(float)) <= TOL_TEND
        big = fine & (np.abs(want) >= 1e200)
        if big.any():
            assert rel_l2(got[big] * 2.0 ** -700, (want[big] * np.longdouble(2) ** -700).astype(float)) \
                <= TOL_TEND

    with np.errstate(all="ignore"):
        sdg.dg_optr_kernel_setup("OPT1")
        for axis, got in enumerate(sdg.tensorprod_divlike_dirXYZ(D, Dt, *f, N)):
            check(got, along(f[axis], axis))
        for axis, got in enumerate(sdg.tensorprod_gradlike_dirXYZ(D, Dt, f[0], N)):
            check(got, along(f[0], axis))
        for axis in range(3):
            got = sdg.element_matvec_dir(axis + 1, D if axis == 0 else Dt, f[axis], N)
            check(got, along(f[axis], axis))
    # the first element's zero z lines (the last holds the 1e300 when it is alone)
    zero = sdg.tensorprod_gradlike_dirXYZ(D, Dt, f[0], N)[2][: N * N - 1]
    assert np.all(zero == 0.0)


@both
@pytest.mark.parametrize("p,dims", [(1, (5, 4, 3)), (1, (20, 19, 17)), (2, (7, 3, 2)),
                                    (3, (16, 19, 10)), (3, (1, 1, 1)), (5, (4, 5, 3)),
                                    (7, (8, 5, 19)), (7, (2, 1, 3)), (8, (5, 4, 4)),
                                    (11, (3, 2, 4)), (12, (3, 3, 2)), (15, (2, 3, 2))])
@pytest.mark.parametrize("nstep", [1, 5, 1100])
def test_steps_in_one_launch_equal_a_launch_a_stage(opt, p, dims, nstep):
    """Whole step calls of small boxes (one resident grid) against the same box as
    one z-slab, whose stages are launches of their own: the same bits, also over
    calls that follow one another and with a non-finite state in a corner."""
    import sdg
    c = Case(*dims, p)
    q, u, v, w = _fields(c)
    q[-1] = np.inf if nstep == 5 else q[-1]
    a = sdg.Solver(*dims, p, c.D, c.Lift, opt=getattr(sdg, opt))
    b = sdg.Slabs(*dims, p, c.D, c.Lift, 1, opt=getattr(sdg, opt))
    for s in (a, b):
        s.upload(q, u, v, w)
        s.step(c.dt, nstep)
        s.step(0.5 * c.dt, 2)
    assert np.array_equal(a.download(), b.download(), equal_nan=True)


@pytest.mark.parametrize("p", [1, 2, 4, 7, 8, 10, 15])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 3), (13, 5, 7)])
def test_fp32_line_stage_within_its_rounding_bound(p, dims):
    """Tendency of the FP32 form node by node against the oracle's, at one element,
    at blocks that are not full and at uneven boxes: a line result is a chain of
    at most N + 4 roundings (coefficient, product, pair, multiply-adds, faces),
    each at most 2^-24 of the terms' magnitudes; three lines add up."""
    import sdg
    c = Case(*dims, p)
    q, u, v, w = _fields(c)
    m, N = c.mesh, p + 1
    _, want = _tendencies(c, q, u, v, w, "OPT_EVENODD")
    s = sdg.Solver(*dims, p, c.D, c.Lift, opt=sdg.OPT_EVENODD, precision=sdg.PREC_FP32)
    s.upload(q, u, v, w)
    rows = np.abs(np.asarray(c.D).reshape(N, N)).sum(axis=0).max()  # of a row, by symmetry
    rows = max(rows, np.abs(np.asarray(c.D).reshape(N, N)).sum(axis=1).max())
    lift = np.abs(np.asarray(c.Lift)).max()
    Es, Fs = np.abs(m.Escale).max(), np.abs(m.Fscale).max()
    qm, um = np.abs(q).max(), max(np.abs(a).max() for a in (u, v, w))
    bound = 3 * qm * um * (Es * rows + 2 * Fs * lift * 2) * (N + 4) * 2.0 ** -24
    assert np.max(np.abs(s.tendency() - want)) <= bound


@pytest.mark.parametrize("threads,epb", [(32, 1), (96, 5), (128, 2), (512, 8)])
def test_batched_line_stage_equals_the_single_box_bit_for_bit(threads, epb):
    """Every order of the batch at block sizes below and above one element's
    lines, items of part of a block's lines and of several rounds: the members'
    bits are the single-box solver's."""
    import sdg
    import workloads as W
    orders = list(range(1, 12))
    tab = {p: W.reference_operators(p) for p in orders}
    dims = [(3 + p % 3, 2 + p % 2, 3) for p in orders]
    dt = [1e-3 / (2 * p + 1) for p in orders]
    ens = sdg.Ensemble(dims, orders, dt, tab)
    for p in orders:
        ens.set_epb(p, 1)
        ens.set_threads(threads, p=p)
        ens.set_epb(p, min(epb, 8 if p < 9 else 4))
    states = []
    for i, p in enumerate(orders):
        c = Case(*dims[i], p)
        f = _fields(c)
        states.append((c, f))
        ens.upload(i, *f)
    ens.step(3)
    for i, (c, f) in enumerate(states):
        s = sdg.Solver(*dims[i], orders[i], *tab[orders[i]][1::2], opt=sdg.OPT_EVENODD,
                       precision=sdg.PREC_FP32)
        s.upload(*f)
        s.step(dt[i], 3)
        assert np.array_equal(ens.download(i), s.download()), orders[i]


@pytest.mark.parametrize("offset", [0, 1, 4099])
def test_download_into_fresh_and_offset_memory(offset):
    """A download that maps its destination first: fresh memory, any alignment,
    nothing outside the destination."""
    import sdg
    c = Case(9, 8, 7, 3)
    f = _fields(c)
    s = sdg.Solver(9, 8, 7, 3, c.D, c.Lift)
    s.upload(*f)
    whole = np.empty(c.nown + offset + 8192)
    whole[:offset] = 7.0
    whole[offset + c.nown:] = 7.0
    s.download(out=whole[offset: offset + c.nown])
    assert np.array_equal(whole[offset: offset + c.nown], f[0])
    assert np.all(whole[:offset] == 7.0) and np.all(whole[offset + c.nown:] == 7.0)


@pytest.mark.parametrize("stage", [1, 2, 3])
@pytest.mark.parametrize("n,offset", [(1, 0), (2, 0), (1001, 0), (1000, 1), (4097, 1)])
def test_rk_stage_at_odd_sizes_and_alignments(stage, n, offset):
    """The 8- and 16-byte forms against numpy: five roundings there and three here,
    each of at most the terms' size, weigh no more than 7 units of it."""
    import sdg
    r = np.random.RandomState(n + stage)
    q, q0, t = [r.randn(n + offset + 1) for _ in range(3)]
    dq, d0, dt = [sdg.DeviceArray(x) for x in (q, q0, t)]
    assert sdg.lib.sdg_rk_stage_dev(dq.ptr + 8 * offset, d0.ptr + 8 * offset,
                                    dt.ptr + 8 * offset, n, 1, stage, 0.37, None) == 0
    got = dq.numpy()
    a, b = [(0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)][stage - 1]
    m = slice(offset, offset + n)
    want = a * q0[m] + b * (q[m] + 0.37 * t[m])
    size = np.abs(q0[m]) + np.abs(q[m]) + np.abs(t[m])
    assert np.all(np.abs(got[m] - want) <= 7 * 2.0 ** -53 * size)
    assert np.array_equal(got[:offset], q[:offset]) and got[offset + n] == q[offset + n]
