"""A batch goes on through changes of its launch shape: a run, other shapes with
larger CTA maps, then the first shape's run again, equal to the lattice alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("between", ["info", "autotune"])
def test_same_run_after_a_larger_shape(between):
    from chllmodel_b200.batched import Batch, replica
    from chllmodel_b200.lattice import Lattice, coupling

    with Batch([replica(32, kT=0.6, K=0.8, seed=r, replica=r) for r in range(16)]) as b:
        b.init_random()
        b.set_tuning(512)
        b.run(4, 2)
        if between == "info":
            b.set_tuning(128)
            assert b.info()["grid"] > 148
        else:
            b.autotune(trial_sweeps=2)
        b.set_tuning(512, 0, 0)
        b.run(4, 2)
        m = b.moments()
        after = b.download_f4(15)
    assert np.all(m[:, 15] == 0) and np.all(m[:, 12] == 9)
    lat = Lattice(32, 32, 32, boundary="periodic")
    lat.init_random(15, 15)
    lat.set_control(0.1, step=1)
    lat.sweep(coupling(0.6, 0.8), 8, seed=15, replica=15)
    assert np.array_equal(after, lat.download_f4())
    lat.close()


def test_tuned_with_waits_that_run_out():
    """Trials limited to one poll per wait give up: the tuner reports it, and with the
    default limit the batch goes on as if they had not been."""
    from chllmodel_b200 import _lib
    from chllmodel_b200.batched import Batch, replica
    from chllmodel_b200.lattice import Lattice, coupling

    with Batch([replica(64, kT=0.6, K=0.8, seed=r, replica=r) for r in range(2)]) as b:
        b.init_random()
        b.run(2, 1)
        b.set_wait_limit(1)
        with pytest.raises(_lib.ChllError, match="timed out"):
            b.autotune(trial_sweeps=20)
        b.set_wait_limit(1 << 24)
        b.run(3, 0)
        m = b.moments()
        after = b.download_f4(1)
    assert np.all(m[:, 15] == 0) and np.all(m[:, 12] == 6) and np.all(m[:, 0] == 2)
    lat = Lattice(64, 64, 64, boundary="periodic")
    lat.init_random(1, 1)
    lat.set_control(0.1, step=1)
    lat.sweep(coupling(0.6, 0.8), 5, seed=1, replica=1)
    assert np.array_equal(after, lat.download_f4())
    lat.close()
