"""The element contractions output by output.  In FP64 a sum is off by (N + 2) units
of 2^-53 of the sum of its terms' magnitudes at most; in fixed point by 2^-59 of its
row's magnitudes times its line's largest value, 1.5 N + 3 times at most: a value is
off by one unit of 2^-59 of twice the largest (2), a coefficient by one of 2^-60 of
twice the row (N), the dropped low limbs N / 2, the last shift 1; and by half a unit
of the result."""
import numpy as np
import pytest

from helpers import operators

pytestmark = pytest.mark.gpu

# sizes on the fixed-point side of the kernel choice
SIZES = [(1, 20011), (2, 5600), (3, 2400), (7, 301), (8, 207), (11, 90), (12, 5), (15, 40)]


def _lines(a, axis, N):
    """(line, node) view of an element array along an axis."""
    return np.moveaxis(a.reshape(-1, N, N, N), 3 - axis, -1).reshape(-1, N)


def _calls(N, D, Dt, f):
    """(axis, result, input) of every entry point."""
    import sdg
    out = []
    for opt in ("OPT1", "GENERAL"):
        sdg.dg_optr_kernel_setup(opt)
        out += [(k, x, f[k]) for k, x in enumerate(sdg.tensorprod_divlike_dirXYZ(D, Dt, *f, N))]
    out += [(k, x, f[0]) for k, x in enumerate(sdg.tensorprod_gradlike_dirXYZ(D, Dt, f[0], N))]
    out += [(k, sdg.element_matvec_dir(k + 1, D if k == 0 else Dt, f[k], N), f[k])
            for k in range(3)]
    return out


def _steep(r, n, N):
    """Magnitudes over sixty powers of two beside one another."""
    return np.exp2(-60 * r.rand(n * N ** 3)) * r.choice([-1.0, 1.0], n * N ** 3)


@pytest.mark.parametrize("p,n", SIZES)
def test_the_identity_returns_its_input(p, n):
    N = p + 1
    r = np.random.RandomState(p)
    f = [_steep(r, n, N) for _ in range(3)]
    eye = np.eye(N).reshape(-1)
    for axis, got, x in _calls(N, eye, eye, f):
        assert np.array_equal(got, x)


def _exact(M, x, axis, N):
    a = _lines(x, axis, N).astype(np.longdouble)
    return a @ M.T.astype(np.longdouble), np.abs(a) @ np.abs(M.T).astype(np.longdouble)


@pytest.mark.parametrize("p,n", SIZES)
@pytest.mark.parametrize("kind", ["triangular", "graded", "small"])
def test_matrices_with_small_entries_have_fp64_sums(p, n, kind):
    """Each output against the sum of its own terms."""
    N = p + 1
    r = np.random.RandomState(p)
    M = 0.5 + r.rand(N, N)
    if kind == "triangular":
        M = np.tril(M)
    elif kind == "graded":
        M *= np.exp2(-12.0 * np.abs(np.subtract.outer(np.arange(N), np.arange(N))))
    else:
        M[0, N - 1] = 2.0 ** -30
    f = [_steep(r, n, N) for _ in range(3)]
    D, Dt = np.ascontiguousarray(M.T).reshape(-1), M.reshape(-1)
    for axis, got, x in _calls(N, D, Dt, f):
        want, terms = _exact(M, x, axis, N)
        assert np.all(np.abs(_lines(got, axis, N) - want) <= (N + 2) * 2.0 ** -53 * terms)


@pytest.mark.parametrize("p,n", SIZES)
@pytest.mark.parametrize("field", ["steep", "spike", "smooth"])
def test_derivative_against_its_lines(p, n, field):
    """The order's own D1D: each output within the fixed-point bound of its own line,
    and where it is its line's largest value's, all others less than a 128th of
    that, within the FP64 bound of its own terms."""
    N = p + 1
    r = np.random.RandomState(p)
    _, D, Dt, _ = operators(p)
    M = np.asarray(D).reshape(N, N).T
    if field == "steep":
        f = [_steep(r, n, N) for _ in range(3)]
    elif field == "spike":
        f = [1e-12 * r.randn(n * N ** 3) for _ in range(3)]
        for x in f:
            x.reshape(-1, N ** 3)[np.arange(n), r.randint(0, N ** 3, n)] = r.randn(n)
    else:
        f = [np.sin(np.arange(n * N ** 3) / (3.0 + k)) for k in range(3)]
    rows = np.abs(M).sum(axis=1)
    for axis, got, x in _calls(N, D, Dt, f):
        want, terms = _exact(M, x, axis, N)
        a = np.abs(_lines(x, axis, N))
        top = a.max(axis=1, keepdims=True)
        err = np.abs(_lines(got, axis, N) - want)
        fixed = (1.5 * N + 3) * 2.0 ** -59 * rows * top + 2.0 ** -53 * np.abs(want)
        double = (N + 2) * 2.0 ** -53 * terms
        # with zeros on the diagonal the output of a largest value 64 times the next
        # may be formed either way, above 128 times in FP64
        ratio = top[:, 0] / np.maximum(np.sort(a, axis=1)[:, -2], 5e-324)
        i = a.argmax(axis=1)
        line = np.arange(i.size)
        zeros = np.any(np.abs(np.diag(M)) < rows * 2.0 ** -10)
        either = zeros & (ratio >= 64)
        lone = zeros & (ratio > 128)
        fixed[line[either], i[either]] = np.maximum(fixed, double)[line[either], i[either]]
        fixed[line[lone], i[lone]] = double[line[lone], i[lone]]
        assert np.all(err <= fixed)
        if field == "spike" and p > 1:
            assert np.count_nonzero(lone) > 0
