"""The codes that an engine reports can be given back to it, at every side and
whatever was set or tuned before: the same codes are reported again, and the
results are the same bits.  The sides whose default is a cluster per individual
have a code of their own for it, which goes with no other."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64, 128, 256, 384, 512, 768, 1024, 2048, 100])
def test_codes_go_back(n):
    I, _, _ = synthetic.polygon_pattern(seed=1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=1)
    dens, S = synthetic.start_population(n, 2, n * 0.25, seed=5)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))

    def run():
        e.upload(0, dens, S)
        e.raar(0, 2, 2, 0.87, 0.0)
        return e.download(0, 2)[0].view(np.uint32)

    want, default = run(), e.tiles()
    e.set_tiles(*default)
    assert e.tiles() == default and np.array_equal(run(), want)
    if n != 100:
        e.upload(0, dens, S)
        e.autotune(0, 2, 2)
        tuned = e.tiles()
        e.set_tiles(0, 0)
        e.set_tiles(*tuned)
        assert e.tiles() == tuned and np.array_equal(run(), want)
    if n in (32, 64, 128):
        assert default == (900, 900)
        e.set_tiles(16, 8)
        assert e.tiles() == (16, 8) and np.array_equal(run(), want)
        for bad in ((900, 8), (16, 900), (901, 0)):
            with pytest.raises(_lib.EngineError):
                e.set_tiles(*bad)
        assert e.tiles() == (16, 8)
        for code in ((900, 0), (0, 900), (900, 900)):
            e.set_tiles(16, 8)
            e.set_tiles(*code)
            assert e.tiles() == (900, 900) and np.array_equal(run(), want)
