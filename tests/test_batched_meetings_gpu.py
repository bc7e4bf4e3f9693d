"""The batch's meetings: groups of one and of many CTAs, paired and single, in
one wave and several, with and without measurements, run after run -- every
replica equal to the same lattice swept alone, control values included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,paired,wave_bytes", [
    (None, False, 0), (128, True, 0), (256, False, 0), (512, True, 0), (128, False, 1 << 20),
    (256, True, 3 << 20),
])
def test_replicas_follow_their_lattices(threads, paired, wave_bytes):
    from chllmodel_b200.batched import Batch, replica
    from chllmodel_b200.lattice import Lattice, coupling
    from chllmodel_b200.observables import B_D, B_FACCEPT, B_NMEAS, B_PACCEPT, B_STEP

    specs = [replica(8, kT=0.5, K=0.9, g=0.1, seed=3, replica=0),
             replica(40, 36, 44, kT=0.7, K=0.5, seed=4, replica=1),
             replica(30, 18, 10, kT=0.3, K=1.0, seed=5, replica=2, boundary="open"),
             replica(64, kT=1.1, K=1.0, g=0.3, seed=(7 << 33) + 1, replica=3),
             replica(5, 3, 7, kT=0.4, K=0.2, seed=6, replica=4, boundary="open")]
    runs = ((7, 3), (1, 1), (5, 0), (6, 3))  # sweeps, measured every
    with Batch(specs) as b:
        if threads:
            b.set_tuning(threads, 0, wave_bytes, paired, False)
        b.init_random()
        for n, every in runs:
            b.run(n, every)
        m = b.moments()
        states = [b.download_f4(r) for r in range(len(specs))]
    for r, sp in enumerate(specs):
        lat = Lattice(sp["ni"], sp["nj"], sp["nk"], boundary=sp["boundary"])
        lat.set_kernel("fused")
        lat.init_random(sp["seed"], sp["replica"])
        lat.set_control(sp["d"], step=1)
        cp = coupling(sp["kT"], sp["K"], sp["g"], sp["eps"])
        rows = []
        for n, every in runs:
            for i in range(n):
                lat.sweep(cp, 1, seed=sp["seed"], replica=sp["replica"])
                if every and (i + 1) % every == 0:
                    rows.append(lat.observe(cp))
        assert np.array_equal(states[r], lat.download_f4())
        ctl = lat.control()
        assert m[r, B_NMEAS] == len(rows)
        assert (m[r, B_D], m[r, B_STEP]) == (ctl["d"], ctl["step"])
        assert (m[r, B_PACCEPT], m[r, B_FACCEPT]) == (ctl["paccept"], ctl["faccept"])
        e = np.array([row[5] for row in rows]) / lat.nsites
        # FP64 sums of the same terms in another order
        assert m[r, 1] == pytest.approx(e.sum(), rel=1e-11, abs=1e-11)
        lat.close()


@pytest.mark.parametrize("threads", [128, 512])
def test_more_replicas_than_ctas(threads):
    """A batch of more replicas than the grid has CTAs fills wave after wave."""
    from chllmodel_b200.batched import Batch, replica
    from chllmodel_b200.lattice import Lattice, coupling

    specs = [replica(4, 4, 2 + 2 * (i % 3), kT=0.5, K=0.7, seed=i, replica=i) for i in range(700)]
    with Batch(specs) as b:
        b.set_tuning(threads)
        b.init_random()
        b.run(5, 5)
        grid = b.info()["grid"]
        assert b.tuning()["waves"] == -(-len(specs) // grid)
        m = b.moments()
        assert np.all(m[:, 12] == 6) and np.all(m[:, 15] == 0)
        for r in (0, 299, 699):
            sp = specs[r]
            lat = Lattice(sp["ni"], sp["nj"], sp["nk"], boundary="periodic")
            lat.init_random(sp["seed"], sp["replica"])
            lat.set_control(0.1, step=1)
            lat.sweep(coupling(0.5, 0.7), 5, seed=sp["seed"], replica=sp["replica"])
            assert np.array_equal(b.download_f4(r), lat.download_f4())
            lat.close()


@pytest.mark.parametrize("size,count", [(48, 10), (48, 11), (8, 148), (20, 149)])
def test_tuned_batches_keep_their_state(size, count):
    """Either side of the sizes whose lower occupancies are tried: the tuner
    leaves states and control values as they were, and the run follows its lattice."""
    from chllmodel_b200.batched import Batch, replica
    from chllmodel_b200.lattice import Lattice, coupling

    with Batch([replica(size, kT=0.6, K=0.8, seed=r, replica=r) for r in range(count)]) as b:
        b.init_random()
        before = b.download_f4(count - 1)
        tuned = b.autotune(trial_sweeps=2, cache=False)
        assert np.array_equal(before, b.download_f4(count - 1))
        assert tuned["ctas_per_sm"] >= 1
        b.run(3, 0)
        after = b.download_f4(count - 1)
    lat = Lattice(size, size, size, boundary="periodic")
    lat.init_random(count - 1, count - 1)
    lat.set_control(0.1, step=1)
    lat.sweep(coupling(0.6, 0.8), 3, seed=count - 1, replica=count - 1)
    assert np.array_equal(after, lat.download_f4())
    lat.close()
