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
