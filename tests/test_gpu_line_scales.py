"""GPU: the scales of FP64 lines in fixed point (csrc/fft_fx.cuh): what a line
keeps next to lines, points and bins of another size.

Reference: pocketfft in long double.  Tolerance of a pass: TOL of
test_gpu_fixed_point.py, a line on its own."""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_fixed_point import TOL, engine, r2r, rel, to_device, to_lines  # noqa: E402

# a compile-time plan, the smooth-length kernel, the general kernel (factors 11
# and 19), a plan with idle threads in a stage
KERNELS = [64, 30, 112, 66, 38, 243]


def real_passes(rows, axis):
    """(spectra, lines back) of rows through r2c, then of the exact spectra,
    rounded, through c2r; and the exact results of both."""
    lines, n = rows.shape
    e = engine(n, lines, axis, True)
    x = to_device(rows, axis, True)
    s, b = e.empty_spectral(), torch.empty_like(x)
    e.r2c(x, s)
    exact = scipy_fft.rfft(rows.astype(np.longdouble), axis=1)
    spec = exact.astype(np.complex128)
    e.c2r(to_device(spec, axis, True), b)
    return (to_lines(s, axis, True), exact), (to_lines(b, axis, True),
                                              scipy_fft.irfft(spec.astype(np.clongdouble), n=n, axis=1) * n)


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", KERNELS)
def test_real_neighbours_have_their_own_scales(n, axis):
    """r2c and c2r carry two real lines in one complex line: a line 2^60 .. 2^300
    smaller than its neighbour is as accurate as alone, a zero one stays zero."""
    rng = np.random.default_rng(n)
    exps = np.array([0, -60, 300, 0, 0, 40, -200, 0, 0])  # 9 lines: the last without a neighbour
    a = np.ldexp(rng.standard_normal((exps.size, n)), exps[:, None])
    a[3], a[4] = 300.0, 0
    for got, ref in real_passes(a, axis):
        for i in range(exps.size):
            assert not got[i].any() if i == 4 else rel(got[i], ref[i]) <= TOL, i


def spread(kind, shape, rng):
    """Lines (complex) of few digits near a value whose part of the sums FP64
    cancels exactly."""
    g = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    if kind == "fp32 mean":
        return (101325 + 100 * g).astype(np.complex64).astype(np.complex128)
    if kind == "integers":
        return 2.0 ** 20 + rng.integers(-8, 9, shape) + 1j * rng.integers(-8, 9, shape)
    if kind == "negative":
        return -1 - 1j + np.rint(g * 2.0 ** 20) * 2.0 ** -40
    if kind == "one component":
        return 1e6 + 1j * g.imag
    # every second line a constant one, the others noise
    return np.where(np.arange(shape[0])[:, None] % 2 == 0, 300.0 + 0j, g * 1e-3)


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", KERNELS + [2, 17, 512, 1024, 4096])
def test_a_mean_leaves_the_rest_its_digits(n, axis):
    """c2c both ways and r2c of lines near a constant of few digits: the other
    bins, whose exact values are taken on the line less that constant, are as
    accurate as those of a line without it; bin 0 is within two roundings."""
    rng = np.random.default_rng(n)
    for kind in ("fp32 mean", "integers", "negative", "one component", "neighbours"):
        a = spread(kind, (7, n), rng)
        for real in (False, True):
            rows = np.ascontiguousarray(a.real) if real else a
            mean = rows[:, :1] * (np.abs(rows[:, :1]) > 0.5)
            rest = rows.astype(np.clongdouble) - mean
            e = engine(n, 7, axis, real)
            x = to_device(rows, axis, real)
            for sign in (-1,) if real else (-1, 1):
                y = e.empty_spectral() if real else torch.empty_like(x)
                e.r2c(x, y) if real else e.c2c(x, y, sign)
                got = to_lines(y, axis, real)
                ref = scipy_fft.fft(rest, axis=1) if sign < 0 else scipy_fft.ifft(rest, axis=1) * n
                ref = ref[:, :got.shape[1]]
                dc, of = rows.astype(np.clongdouble).sum(axis=1), mean[:, 0].real != 0
                assert (np.abs(got[of, 0] - dc[of]) <= 2.0 ** -51 * np.abs(dc[of])).all(), (kind, real)
                for i in range(7):
                    err = np.sqrt((np.abs(got[i, 1:] - ref[i, 1:]) ** 2).sum())
                    assert err <= TOL * np.sqrt((np.abs(ref[i]) ** 2).sum()), (kind, real, i)


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("n", [9, 33, 64, 129, 257])
def test_r2r_of_a_mean_leaves_the_rest_its_digits(n, kind, axis):
    rng = np.random.default_rng(n)
    rows = np.rint(101325 * 64 + 6400 * rng.standard_normal((5, n))) / 64
    rows[2] = 300.0
    got = r2r(rows, kind, axis)
    rest = scipy_fft.dct(rows.astype(np.longdouble) - rows[:, :1], type=kind, axis=1)
    dc = scipy_fft.dct(rows.astype(np.longdouble), type=kind, axis=1)[:, 0]
    assert (np.abs(got[:, 0] - dc) <= 2.0 ** -51 * np.abs(dc)).all()
    for i in range(5):
        err = np.sqrt((np.abs(got[i, 1:] - rest[i, 1:]) ** 2).sum())
        assert err <= TOL * np.sqrt((np.abs(rest[i]) ** 2).sum()), i


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [12, 30, 38, 512, 840, 960, 1296, 1331, 1536, 4096])
def test_bin_0_costs_the_others_no_digits(n, axis):
    """c2r of fields of one sign, whose bin 0 is far above the others: at most
    the FP64 kernels' error (1.9e-16 to 2.6e-16 on these)."""
    rng = np.random.default_rng(n)
    a = 1e-3 * rng.standard_normal((9, n))
    a[:, rng.choice(n, n // 4 if n < 1024 else 256, replace=False)] += 1e6 * (1 + rng.random())
    a[4] = 0
    a[5] = 300.0  # nothing but bin 0
    got, ref = real_passes(a, axis)[1]
    for i in range(9):
        assert not got[i].any() if i == 4 else rel(got[i], ref[i]) <= 2.2e-16, i


# rel-L2 of the FP64 kernels, c2r of the spectrum of one peak
FP64_PEAK = {23 * 89: 3.1e-16, 41 * 43: 3.1e-16, 29 * 67: 3.6e-16, 11 * 179: 4.3e-16}


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", FP64_PEAK)
def test_direct_sums_keep_fp64_accuracy(n, axis):
    """c2r of a flat spectrum through direct-sum stages."""
    rng = np.random.default_rng(n)
    a = 1e-3 * rng.standard_normal((9, n))
    a[:, n // 3] += 1e6 * (1 + rng.random())
    got, ref = real_passes(a, axis)[1]
    for i in range(9):
        assert rel(got[i], ref[i]) <= FP64_PEAK[n], i


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("n", KERNELS)
def test_small_fields_scale_exactly(n, real):
    """Down to 2^-930 a line is transformed as its multiple by a power of two."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((6, n)) + (0 if real else 1j * rng.standard_normal((6, n)))
    out = []
    for k in (0, -930):
        e = engine(n, 6, 0, real)
        x = to_device(a * 2.0 ** k, 0, real)
        y = e.empty_spectral() if real else torch.empty_like(x)
        e.r2c(x, y) if real else e.c2c(x, y, -1)
        if real:
            e.c2r(y, x)
            out.append(x * 2.0 ** -k)
        out.append(y * 2.0 ** -k)
    assert all(torch.equal(u, v) for u, v in zip(out[:len(out) // 2], out[len(out) // 2:]))


# rel-L2 of the FP64 kernels, c2r of the spectrum of noise
FP64_NOISE = {7 * 11 * 13: 2.3e-16, 7 * 17 * 17: 2.8e-16}


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", FP64_NOISE)
def test_large_radices_keep_fp64_accuracy(n, axis):
    rng = np.random.default_rng(n)
    got, ref = real_passes(rng.standard_normal((9, n)), axis)[1]
    assert rel(got, ref) <= FP64_NOISE[n]
