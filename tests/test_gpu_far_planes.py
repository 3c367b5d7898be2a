"""GPU: the kernel of an axis does not depend on how far apart the rows of
another axis lie: lines of a grid whose plane holds more than 2^28 points
transform bit for bit as on a small grid."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, LINES, FEW = 960, 280000, 1024  # (960 + 8) x 280000 > 2^28


@pytest.mark.parametrize("prec", [4, 8])
def test_x_lines_of_a_large_plane(prec):
    import gbfft
    dt = torch.complex64 if prec == 4 else torch.complex128
    g = torch.Generator(device="cuda").manual_seed(prec)
    x = torch.randn((1, LINES, N), dtype=dt, device="cuda", generator=g)
    few = x[:, -FEW:].contiguous()
    y = torch.empty_like(few)
    gbfft.Engine(1, N, FEW, 1, skip=(False, True, True), prec=prec).c2c(few, y, -1)
    gbfft.Engine(1, N, LINES, 1, inplace=True, skip=(False, True, True), prec=prec).c2c(x, x, -1)
    assert torch.equal(x[:, -FEW:], y)
