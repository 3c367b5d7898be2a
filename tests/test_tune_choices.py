"""CPU: the autotuner times only choices that change what runs."""
import pytest

import gbfft
import tune


@pytest.mark.parametrize("n", [16, 64, 256, 270, 400, 512, 1024])
def test_double_precision_has_one_plan_and_no_clusters(n):
    assert tune.plan_choices(8, n) == [None]
    assert tune.launch_choices(8, "c2c_y", n, 16) == [(0, 0)]
    assert len(tune.plan_choices(4, n)) > 1


def test_cluster_forms_are_the_power_of_two_kernels():
    assert tune.launch_choices(4, "c2c_y", 512, 16) == tune.LAUNCHES
    for kind, n, points in (("xy_fused", 512, 16), ("c2c_y", 270, 30), ("c2c_y", 225, 0)):
        assert tune.launch_choices(4, kind, n, points) == [(0, 0)]


class Tiles:
    """An engine whose kernel holds up to 8 lines and refuses more than 16."""

    def __init__(self):
        self.tiles = {"c2c_y": 0}

    def set_tile(self, kind, lines):
        if lines > 16:
            raise gbfft.GbfftError(1, "tile exceeds the kernel's thread limit")
        self.tiles[kind] = lines if lines <= 8 else 0

    def tuning(self):
        return {"tiles": self.tiles}


def test_only_tiles_in_use_are_timed():
    eng = Tiles()
    assert [L for L in [0] + tune.TILES if tune.take_tile(eng, "c2c_y", L)] == [0, 1, 2, 4, 8]
