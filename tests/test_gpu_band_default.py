"""The default between band visits and tile launches is the faster of the two, or near it."""
import pytest

pytestmark = pytest.mark.gpu


# The larger of the two measured times over the smaller is given; a default on the wrong side
# is that much off, so a tenth tells them apart with room for the runs' few per cent.
@pytest.mark.parametrize("n,ncases,isolve", [
    (128, 128, 1),    # bands 1.22
    (96, 128, 1),     # bands 1.25
    (64, 56, 1),      # bands 1.40
    (128, 16, 1),     # tiles 1.24
    (64, 60, 2),      # bands 1.29
    (128, 64, 2),     # tiles 1.34
    (96, 32, 2),      # tiles 1.29
])
def test_default_is_the_faster(n, ncases, isolve):
    from mgfvm import Solver, configs
    with Solver([configs.small(n, 1, isolve=isolve, amuf=1.0 / (20.0 + k % 7)) for k in range(ncases)]) as s:
        def time():
            best = 1e30
            for _ in range(5):
                s.cycle(10)
                best = min(best, s.last_elapsed_ms)
            return best
        s.cycle(10)
        default = time()
        s.set_tuning(band_visit=[1] * 16)
        tiles = time()
        s.set_tuning(band_visit=[2] * 16)
        bands = time()
        assert default < 1.1 * min(tiles, bands), (default, tiles, bands)
