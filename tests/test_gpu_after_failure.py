"""A call that the runtime refuses (an allocation of terabytes) returns an error
and leaves the next calls alone: the same results as before."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 100, 512])
def test_refused_allocation(n):
    I, _, _ = synthetic.polygon_pattern(seed=1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=2)
    dens, S = synthetic.start_population(n, 3, n * 0.25, seed=5)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))

    def run():
        e.upload(0, dens, S)
        e.raar(0, 3, 2, 0.9, 0.0)
        e.sw(0, 3, 2.0, 0.1)
        m = e.evaluate(0, 3)
        d, s = e.download(0, 3)
        return d.view(np.uint32), s, [k["error"] for k in m]

    want = run()
    for _ in range(2):
        with pytest.raises(_lib.EngineError) as err:
            e.reserve(2 ** 31 - 1)
        assert err.value.code == 3  # SPE_ERR_NOMEM
        got = run()
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and got[2] == want[2]
    assert e.capacity == 3
