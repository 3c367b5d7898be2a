"""GPU: the scales of FP64 lines in fixed point (csrc/fft_fx.cuh): what a line
keeps next to lines, points and bins of another size.

Reference: pocketfft in long double.  Tolerance of a pass: TOL of
test_gpu_fixed_point.py, a line on its own."""
import numpy as np
import pytest

scipy_fft = pytest.importorskip("scipy.fft")
torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_fixed_point import TOL, engine, rel, to_device, to_lines  # noqa: E402

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
