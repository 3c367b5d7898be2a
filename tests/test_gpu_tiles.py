"""GPU: gbfft_engine_set_tile records the tiles that the passes run."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# axis length, precision; a tile its kernel holds; one that only another kernel
# of the length would hold; one beyond every limit (64 lines at most are asked)
TILES = [(270, 4, 8, 32, None), (400, 4, 8, 24, 64), (64, 8, 16, None, 64), (512, 8, 4, 8, 64), (1024, 4, 8, None, 64),
         (48, 4, 16, None, 64), (225, 4, 16, None, 32)]


@pytest.mark.parametrize("n,prec,held,other,refused", TILES)
def test_tiles_in_use_are_reported(n, prec, held, other, refused):
    import gbfft
    e = gbfft.Engine(1, 64, n, 64, prec=prec)
    e.set_tile("c2c_y", held)
    assert e.tuning()["tiles"]["c2c_y"] == held
    if other:
        e.set_tile("c2c_y", other)  # accepted, and the built-in tile runs
        assert e.tuning()["tiles"]["c2c_y"] == 0
    if refused:
        with pytest.raises(gbfft.GbfftError):
            e.set_tile("c2c_y", refused)
    e.close()
