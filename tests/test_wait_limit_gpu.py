"""Waits of the resident sweep and quench launches that run out: limited to one poll,
each form returns with the status word set, the calls that wait report it, and after
a new state and control block the lattice follows its chain again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    ((32, 32, 32), "periodic"),   # neighbours' words, a site of each colour per thread
    ((33, 31, 17), "open"),
    ((56, 54, 56), "periodic"),   # sweeps by the grid barrier, a quench of 896 threads per SM
    ((64, 60, 64), "open"),       # a unit per thread
    ((96, 96, 96), "periodic"),   # several units per thread
]


def _lattice(shape, boundary):
    from chllmodel_b200.lattice import Lattice

    lat = Lattice(*shape, boundary=boundary)
    lat.init_random(5)
    lat.set_control(0.1, step=1)
    return lat


@pytest.mark.parametrize("shape,boundary", SHAPES)
@pytest.mark.parametrize("what", ["sweep", "quench"])
def test_waits_that_run_out(shape, boundary, what):
    from chllmodel_b200 import _lib
    from chllmodel_b200.lattice import coupling

    cp = coupling(0.5, 0.8, 0.1)

    def go(lat, n):
        lat.sweep(cp, n, seed=3) if what == "sweep" else lat.quench(cp, 0.05, n)

    lat = _lattice(shape, boundary)
    lat.set_kernel("resident")
    go(lat, 3)
    lat.sync()
    lat.set_wait_limit(1)
    go(lat, 200)
    for call in (lat.sync, lambda: lat.observe(cp), lat.download_f4, lat.control,
                 lambda: lat.energy_sums(cp)):
        with pytest.raises(_lib.ChllError, match="status word") as e:
            call()
        assert e.value.code == _lib.CHLL_EDEVICE
    go(lat, 2)  # does nothing
    with pytest.raises(_lib.ChllError, match="status word"):
        lat.sync()
    lat.set_wait_limit(1 << 22)
    lat.init_random(5)
    lat.set_control(0.1, step=1)
    alone = _lattice(shape, boundary)
    alone.set_kernel("resident")
    for n in (1, 2, 7):
        go(lat, n)
        go(alone, n)
        assert np.array_equal(lat.download_f4(), alone.download_f4())
        assert lat.control() == alone.control()
    lat.close()
    alone.close()


def test_one_cta_waits_for_nobody():
    from chllmodel_b200 import _lib
    from chllmodel_b200.lattice import coupling

    lat = _lattice((8, 8, 6), "periodic")
    lat.set_wait_limit(1)
    lat.sweep(coupling(0.5, 0.8), 100)
    lat.quench(coupling(0.5, 0.8), 0.05, 20)
    lat.sync()
    assert lat.control()["step"] == 101
    with pytest.raises(_lib.ChllError, match="polls"):
        lat.set_wait_limit(0)
    lat.close()
