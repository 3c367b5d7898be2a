"""GPU: FP64 passes where fixed point ends: lines that go to FP64, lines whose
sums reach the bound that the scale is chosen by, and the longest r2r windows.

Reference: pocketfft in long double; tolerances as in test_gpu_fixed_point.py."""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_fixed_point import TOL, engine, r2r, rel, to_device, to_lines  # noqa: E402

# a compile-time plan, the smooth-length kernel (even and odd), the general kernel
KERNELS = [64, 30, 243, 66, 38]


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", KERNELS)
@pytest.mark.parametrize("lines", [9, 40 * 1024 + 1])  # one pair a CTA, and full CTAs; the last line has no neighbour
def test_real_lines_out_of_range(n, axis, lines):
    """r2c and c2r: NaN, infinities, huge and subnormal lines; the others of
    their CTA run in FP64 too and are right."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((lines, n))
    at = {2: np.nan, 5: np.inf}
    if lines > 9:
        at.update({20001: -np.inf, 30000: np.nan})
    for i, v in at.items():
        a[i, n // 2] = v
    a[0:2] *= 2.0 ** 1010
    a[-1] *= 2.0 ** -1040
    e = engine(n, lines, axis, True)
    x = to_device(a, axis, True)
    s, b = e.empty_spectral(), torch.empty_like(x)
    e.r2c(x, s)
    got = to_lines(s, axis, True)
    bad = [i for p in at for i in (p - p % 2, p - p % 2 + 1)]  # a pair shares its transform
    keep = np.setdiff1d(np.arange(2, lines - 1), bad)
    assert not np.isfinite(got[list(at)]).all(axis=1).any()
    assert rel(got[keep], scipy_fft.rfft(a[keep], axis=1)) <= 5e-15
    assert rel(got[:2] * 2.0 ** -1010, scipy_fft.rfft(a[:2] * 2.0 ** -1010, axis=1)) <= 5e-15
    assert np.abs(got[-1] - scipy_fft.rfft(a[-1])).max() <= 64 * 2.0 ** -1074 * n
    # back from the spectra of the lines that are finite, one NaN and one infinity put in
    a[list(at)] = 0
    a[:2] *= 2.0 ** -1010
    spec = scipy_fft.rfft(a, axis=1)
    spec[4, 1] = np.nan
    spec[7, 0] = np.inf
    e.c2r(to_device(spec, axis, True), b)
    back = to_lines(b, axis, True)
    keep = np.setdiff1d(np.arange(lines - 1), [4, 5, 6, 7])
    assert not np.isfinite(back[[4, 7]]).all(axis=1).any()
    assert rel(back[keep], a[keep] * n) <= 5e-15


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", KERNELS)
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_lines_of_full_tiles(n, axis, bad):
    lines = 20 * 1024 + 3
    rng = np.random.default_rng(n)
    a = rng.standard_normal((lines, n)) + 1j * rng.standard_normal((lines, n))
    ref = scipy_fft.fft(a, axis=1)
    rows = [0, 7, 10001, lines - 1]
    a[rows, n - 1] = bad
    e = engine(n, lines, axis, False)
    x = to_device(a, axis, False)
    y = torch.empty_like(x)
    e.c2c(x, y, -1)
    got = to_lines(y, axis, False)
    keep = np.setdiff1d(np.arange(lines), rows)
    assert not np.isfinite(got[rows]).all(axis=1).any()
    assert rel(got[keep], ref[keep]) <= 5e-15


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [2, 3, 8, 15, 17, 30, 64, 127, 243, 251, 400, 512, 1000, 1024, 1969, 2008, 2047, 2048, 4096])
def test_flat_lines_reach_the_bound(n, axis):
    """Constant lines and single modes at full mantissa, whose output is the sum
    of the line's moduli: no stage overflows."""
    rng = np.random.default_rng(n)
    j, k = np.arange(n), rng.integers(0, n, (8, 1))
    mode = np.exp(2j * np.pi * (k * j % n) / n) * (1 + rng.random((8, 1))) * np.exp(2j * np.pi * rng.random((8, 1)))
    sign = np.where(j % 2 == 0, 1.0, -1.0) * (1 + rng.random((8, 1)))
    same = np.broadcast_to(1 + rng.random((8, 1)), (8, n)) * (1 - 1j)
    for a in (mode, sign + 0j, same, np.abs(mode.real) + 1j * np.abs(mode.imag)):
        e = engine(n, 8, axis, False)
        x = to_device(a, axis, False)
        y = torch.empty_like(x)
        for isign, f in ((-1, scipy_fft.fft), (1, lambda v, axis: scipy_fft.ifft(v, axis=axis) * n)):
            e.c2c(x, y, isign)
            assert rel(to_lines(y, axis, False), f(a.astype(np.clongdouble), axis=1)) <= TOL
        r = np.ascontiguousarray(a.real)
        e = engine(n, 8, axis, True)
        x = to_device(r, axis, True)
        s, b = e.empty_spectral(), torch.empty_like(x)
        e.r2c(x, s)
        spec = to_lines(s, axis, True)
        assert rel(spec, scipy_fft.rfft(r.astype(np.longdouble), axis=1)) <= TOL
        # a spectrum of one modulus, its outputs' sum in one point
        flat = np.exp(-2j * np.pi * (k * j[None, :n // 2 + 1] % n) / n) * (1 + rng.random((8, 1)))
        e.c2r(to_device(flat, axis, True), b)
        ref = flat.astype(np.clongdouble)
        ref[:, 0] = ref[:, 0].real
        if n % 2 == 0:
            ref[:, -1] = ref[:, -1].real
        assert rel(to_lines(b, axis, True), scipy_fft.irfft(ref, n=n, axis=1) * n) <= TOL


# windows up to the longest whose extension is accepted: radix-16 plans of 1024
# and 2048 points (DCT-I and DST-I: 1025 and 1023 points), direct sums of 89 and
# of 2039
LONG = [(1, 1025), (5, 1023), (2, 2047), (3, 1024), (6, 1023), (7, 2047), (4, 1025), (8, 2046), (2, 2039), (3, 2039)]


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kind,n", LONG)
def test_r2r_long_windows(kind, n, axis):
    rng = np.random.default_rng(n + kind)
    f, t = (scipy_fft.dct, kind) if kind <= 4 else (scipy_fft.dst, kind - 4)
    noise = rng.standard_normal((5, n))
    peak = 1e-3 * noise
    peak[:, n // 3] += 1e6
    for a in (noise, peak, np.broadcast_to(1 + rng.random((5, 1)), (5, n))):
        got = r2r(a, kind, axis)
        # a direct sum over 2039 points of two lines: 9 bits of headroom, so its
        # unit is 2^-52 of the largest sum, rounded on the way in and in the sum
        assert rel(got, f(a.astype(np.longdouble), type=t, axis=1)) <= (4 * 2.0 ** -52 if n == 2039 else TOL)
