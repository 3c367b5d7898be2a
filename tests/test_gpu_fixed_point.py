"""GPU: the fixed-point FP64 passes (csrc/fft_fx.cu, csrc/fft_fxc.cu).

Reference: pocketfft in long double (80 bits or more) on the same doubles.
Tolerance: a result is rounded once to 53 bits (rel-L2 at most 2^-53 =
1.1e-16) after integer stages whose noise stays below that up to 4096 points,
so 4 x 2^-53 = 4.4e-16 bounds a single pass; through r2c and c2r two passes.
"""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 4.5e-16
# one line short of and past the plans' edges: the smallest lengths, primes in
# registers (7, 11, 13) and as direct sums (17, 127, 251), compile-time plans
# with idle threads in a stage (96, 243, 384), radix-16 plans (1024 and up),
# the longest fixed-point lengths (2047, 2048, 4096) and FP64's next (2049)
LENGTHS = [2, 3, 5, 7, 8, 11, 13, 15, 16, 17, 30, 33, 96, 121, 126, 127, 169, 210, 243, 251, 256, 384, 400, 512,
           1000, 1024, 2047, 2048, 2049, 4096]


def rel(x, ref):
    d = x.astype(ref.dtype) - ref
    return float(np.sqrt((np.abs(d) ** 2).sum() / (np.abs(ref) ** 2).sum()))


def engine(n, lines, axis, real):
    """An engine whose only pass runs over `lines` lines of n points: along x
    (contiguous) or y / z (strided), c2c or the format's real axis."""
    import gbfft
    if real:
        shape = (n, lines, 1) if axis == 0 else (lines, 1, n)
        return gbfft.Engine(1 if axis == 0 else 3, *shape, skip=(axis != 0, True, axis == 0), prec=gbfft.PREC_DOUBLE)
    shape = (n, lines, 1) if axis == 0 else (lines, n, 1)
    return gbfft.Engine(1, *shape, skip=(axis != 0, axis == 0, True), prec=gbfft.PREC_DOUBLE)


def to_device(a, axis, real):
    """Lines (rows of `a`) as the engine's array."""
    b = a[None] if axis == 0 else (a.T[:, None, :] if real else a.T[None])
    return torch.from_numpy(np.ascontiguousarray(b)).cuda()


def to_lines(t, axis, real):
    b = t.cpu().numpy()
    return b[0] if axis == 0 else (b[:, 0, :].T if real else b[0].T)


def inputs(kind, shape, rng):
    a = rng.standard_normal(shape)
    n = shape[-1]
    if kind == "peak":
        a *= 1e-3
        a[..., n // 3] += 1e6
    if kind == "decay":
        a *= np.exp(-30 * np.arange(n) / n)
    return a


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", LENGTHS)
def test_lengths_against_long_double(n, axis):
    rng = np.random.default_rng(n)
    for kind in ("noise", "peak", "decay"):
        lines = 13
        c = inputs(kind, (lines, n), rng) + 1j * rng.standard_normal((lines, n))
        e = engine(n, lines, axis, False)
        x = to_device(c, axis, False)
        y = torch.empty_like(x)
        e.c2c(x, y, -1)
        assert rel(to_lines(y, axis, False), scipy_fft.fft(c.astype(np.clongdouble), axis=1)) <= TOL, kind
        e.c2c(x, y, 1)
        assert rel(to_lines(y, axis, False), scipy_fft.ifft(c.astype(np.clongdouble), axis=1) * n) <= TOL, kind
        r = inputs(kind, (lines, n), rng)
        e = engine(n, lines, axis, True)
        x = to_device(r, axis, True)
        s, b = e.empty_spectral(), torch.empty_like(x)
        e.r2c(x, s)
        spec = to_lines(s, axis, True)
        assert rel(spec, scipy_fft.rfft(r.astype(np.longdouble), axis=1)) <= TOL, kind
        e.c2r(s, b)
        assert rel(to_lines(b, axis, True), scipy_fft.irfft(spec.astype(np.clongdouble), n=n, axis=1) * n) <= TOL, kind


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [12, 30, 64, 243])
def test_every_line_has_its_own_scale(n, axis):
    """Neighbouring lines 2^-900 .. 2^900 apart (fixed point), beyond that
    (FP64) and all zero: each is as accurate as alone, zeros stay zeros."""
    rng = np.random.default_rng(n)
    exps = np.array([0, -900, 900, 40, -40, 1010, -1030, -1060])
    a = rng.standard_normal((exps.size, n)) + 1j * rng.standard_normal((exps.size, n))
    a = np.ldexp(a.real, exps[:, None]) + 1j * np.ldexp(a.imag, exps[:, None])
    a[3] = 0
    for rows in (a, a[:5]):  # with and without lines that take the tile to FP64
        e = engine(n, len(rows), axis, False)
        x = to_device(rows, axis, False)
        y = torch.empty_like(x)
        e.c2c(x, y, -1)
        got = to_lines(y, axis, False)
        ref = scipy_fft.fft(rows.astype(np.clongdouble), axis=1)
        for i, k in enumerate(exps[: len(rows)]):
            if i == 3:
                assert not got[i].any()
            elif k > -1030:
                scale = np.longdouble(2) ** int(-k)
                assert rel((got[i].real * scale) + 1j * (got[i].imag * scale), ref[i] * scale) <= 5e-15, k
            else:  # subnormal inputs: an absolute error of a few spacings a stage
                assert np.abs(got[i] - ref[i]).max() <= 64 * 2.0 ** -1074 * n, k


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [12, 30, 64, 243])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_stay_in_their_line(n, axis, bad):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((9, n)) + 1j * rng.standard_normal((9, n))
    ref = scipy_fft.fft(a, axis=1)
    a[4, n // 2] = bad
    e = engine(n, 9, axis, False)
    x = to_device(a, axis, False)
    y = torch.empty_like(x)
    e.c2c(x, y, 1)
    e.c2c(x, y, -1)
    got = to_lines(y, axis, False)
    keep = np.arange(9) != 4
    assert not np.isfinite(got[4]).any()
    assert rel(got[keep], ref[keep]) <= 5e-15


def test_scaling_by_a_power_of_two_is_exact():
    rng = np.random.default_rng(5)
    a = rng.standard_normal((6, 360)) + 1j * rng.standard_normal((6, 360))
    out = []
    for k in (0, 70, -300):
        e = engine(360, 6, 1, False)
        x = to_device(a * 2.0 ** k, 1, False)
        y = torch.empty_like(x)
        e.c2c(x, y, -1)
        out.append(y * 2.0 ** -k)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


# ---- real-to-real passes ---------------------------------------------------
def r2r_matrix(kind, n):
    """FFTW's definition of kind 1..8 at n points, in long double."""
    j, k = np.arange(n, dtype=np.int64)[None], np.arange(n, dtype=np.int64)[:, None]
    num, den = {1: (j * k, n - 1), 2: ((2 * j + 1) * k, 2 * n), 3: (j * (2 * k + 1), 2 * n),
                4: ((2 * j + 1) * (2 * k + 1), 4 * n), 5: ((j + 1) * (k + 1), n + 1), 6: ((2 * j + 1) * (k + 1), 2 * n),
                7: ((j + 1) * (2 * k + 1), 2 * n), 8: ((2 * j + 1) * (2 * k + 1), 4 * n)}[kind]
    pi = np.longdouble("3.14159265358979323846264338327950288")
    a = pi * (num % (2 * den)).astype(np.longdouble) / np.longdouble(den)
    m = 2 * (np.cos(a) if kind <= 4 else np.sin(a))
    if kind in (1, 3):
        m[:, 0] /= 2
    if kind in (1, 7):
        m[:, -1] /= 2
    return m


def r2r(lines, kind, axis, pad=0):
    """`lines` (rows) through a pass of `kind` along x or y; the window starts
    `pad` points in."""
    import gbfft
    a = np.pad(lines, ((0, 0), (pad, pad)), constant_values=7.0)
    x = torch.from_numpy(np.ascontiguousarray(a[None] if axis == 0 else a.T[None])).cuda()
    y = torch.empty_like(x)
    cfg = [kind if axis == 0 else 2, kind if axis == 1 else 2, 2]
    first, gone = [1, 1, 1], [0, 0, 0]
    first[axis], gone[axis] = pad + 1, 2 * pad
    d = gbfft.Dtt(1, x.shape[2], x.shape[1], 1, cfg + first + gone + first, skip=(axis != 0, axis != 1, True))
    d.r2r(x, y, -1)
    got = y.cpu().numpy()[0]
    got = got if axis == 0 else got.T
    assert (got[:, :pad] == 7).all() and (got[:, got.shape[1] - pad:] == 7).all()
    return got[:, pad:got.shape[1] - pad]


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kind", range(1, 9))
@pytest.mark.parametrize("n", [2, 3, 4, 5, 9, 16, 17, 32, 33, 96, 127, 129, 255, 256, 400, 512])
def test_r2r_lengths_against_long_double(n, kind, axis):
    rng = np.random.default_rng(n + kind)
    m = r2r_matrix(kind, n)
    for lines, pad in ((7, 0), (8, 2)):  # an odd and an even number of real lines
        a = rng.standard_normal((lines, n))
        assert rel(r2r(a, kind, axis, pad), a.astype(np.longdouble) @ m.T) <= TOL


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kind", range(1, 9))
@pytest.mark.parametrize("n", [12, 16, 17])
def test_r2r_lines_are_independent(n, kind, axis):
    """The two real lines of a pair share a complex transform: their scales
    and their non-finite values stay apart."""
    rng = np.random.default_rng(n + kind)
    m = r2r_matrix(kind, n)
    a = rng.standard_normal((8, n)) * 2.0 ** np.array([0, -200, 0, 300, -300, 0, 0, 50])[:, None]
    a[5] = 0
    got, ref = r2r(a, kind, axis), a.astype(np.longdouble) @ m.T
    for i in range(8):
        assert not got[i].any() if i == 5 else rel(got[i], ref[i]) <= 2 * TOL, i
    a[2, n // 2] = np.nan
    a[7, 0] = np.inf
    got = r2r(a, kind, axis)
    for i in range(8):
        if i in (2, 7):
            assert not np.isfinite(got[i]).all()
        elif i != 5:
            assert rel(got[i], ref[i]) <= 5e-15, i
