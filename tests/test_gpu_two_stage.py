"""GPU: the compile-time two-stage FP32 passes (csrc/fft_mixed.cuh).

Reference: pocketfft in long double on the same floats.  Tolerance: two stages
of composite butterflies round a value at most about ten times, 10 x 2^-24 =
6e-7.  Lengths: for every second radix the smallest and the largest first one.
"""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 6e-7
LENGTHS = [12, 15, 25, 18, 36, 35, 49, 40, 56, 45, 81, 40, 100, 44, 121, 48, 144, 65, 169, 70, 196, 75, 225, 96, 240, 108, 324, 140,
           400, 147, 441, 176, 484, 192, 576, 225, 625, 234, 676, 243, 729, 280, 784, 300, 900, 352, 960]


def rel(x, ref):
    d = x.astype(ref.dtype) - ref
    return float(np.sqrt((np.abs(d) ** 2).sum() / (np.abs(ref) ** 2).sum()))


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("lines", [1, 7, 64])
@pytest.mark.parametrize("n", sorted(set(LENGTHS)))
def test_lengths_against_long_double(n, lines, axis):
    import gbfft
    rng = np.random.default_rng(n + lines)
    c = (rng.standard_normal((lines, n)) + 1j * rng.standard_normal((lines, n))).astype(np.complex64)
    shape = (n, lines, 1) if axis == 0 else (lines, n, 1)
    e = gbfft.Engine(1, *shape, skip=(axis != 0, axis == 0, True), prec=gbfft.PREC_SINGLE)
    x = torch.from_numpy(np.ascontiguousarray(c[None] if axis == 0 else c.T[None])).cuda()
    y = torch.empty_like(x)
    lines_of = (lambda t: t.cpu().numpy()[0]) if axis == 0 else (lambda t: t.cpu().numpy()[0].T)
    e.c2c(x, y, -1)
    assert rel(lines_of(y), scipy_fft.fft(c.astype(np.clongdouble), axis=1)) <= TOL
    e.c2c(x, x, 1)
    assert rel(lines_of(x), scipy_fft.ifft(c.astype(np.clongdouble), axis=1) * n) <= TOL
    r = rng.standard_normal((lines, n)).astype(np.float32)
    shape = (n, lines, 1) if axis == 0 else (lines, 1, n)
    e = gbfft.Engine(1 if axis == 0 else 3, *shape, skip=(axis != 0, True, axis == 0), prec=gbfft.PREC_SINGLE)
    x = torch.from_numpy(np.ascontiguousarray(r[None] if axis == 0 else r.T[:, None, :])).cuda()
    lines_of = (lambda t: t.cpu().numpy()[0]) if axis == 0 else (lambda t: t.cpu().numpy()[:, 0, :].T)
    s, b = e.empty_spectral(), torch.empty_like(x)
    e.r2c(x, s)
    spec = lines_of(s)
    assert rel(spec, scipy_fft.rfft(r.astype(np.longdouble), axis=1)) <= TOL
    e.c2r(s, b)
    assert rel(lines_of(b), scipy_fft.irfft(spec.astype(np.clongdouble), n=n, axis=1) * n) <= TOL
