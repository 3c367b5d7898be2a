"""GPU: the smooth-length runtime kernel in FP32 (csrc/fft_rt.cuh; its FP64
form is covered by test_gpu_fixed_point.py).

Reference: pocketfft in long double on the same floats.  Tolerance: a pass of
two to four stages rounds a value at most about ten times, 10 x 2^-24 = 6e-7.
"""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 6e-7
# two stages of every radix (4 = 2 2 ... 240 = 16 15), prime radices, three and
# four stages, threads idle in a stage, the most threads a line (4095)
LENGTHS = [4, 6, 9, 10, 15, 18, 20, 22, 26, 28, 33, 42, 49, 60, 63, 80, 99, 110, 121, 126, 143, 168, 169, 180, 182, 195,
           208, 225, 240, 250, 330, 405, 500, 729, 1001, 1155, 2197, 4095]


def rel(x, ref):
    d = x.astype(ref.dtype) - ref
    return float(np.sqrt((np.abs(d) ** 2).sum() / (np.abs(ref) ** 2).sum()))


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("lines", [1, 5, 40])
@pytest.mark.parametrize("n", LENGTHS)
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
    # the real axis: x (contiguous lines) or z (strided; an odd and an even
    # number of lines, with and without the paired accesses)
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
