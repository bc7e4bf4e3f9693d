"""Small lattices' sweeps, which wait for neighbours' sites instead of the grid:
the fused passes' chain bit for bit at the edges of their range, over launches
with and without adaptation, new sites in between, and chiralities of any size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,boundary", [
    ((8, 8, 8), "open"), ((8, 13, 5), "open"),                # 256 slots per colour, and 260
    ((8, 34, 2), "periodic"), ((4, 2, 66), "periodic"),       # rows of one block, double bonds
    ((1, 23, 17), "open"), ((2, 700, 1), "open"),             # padding on either side, one plane
    ((2, 16, 18), "periodic"), ((6, 6, 4), "periodic"),       # padded rows that wrap,
    ((30, 18, 10), "periodic"), ((62, 74, 30), "periodic"),   # in one block and in many
    ((64, 74, 30), "periodic"), ((64, 37, 60), "open"),       # 71,040 slots: 148 x 480
    ((64, 74, 32), "periodic"), ((61, 38, 60), "open"),       # beyond
    ((62, 74, 32), "periodic"), ((62, 76, 32), "periodic"),
])
def test_flow_equals_fused(shape, boundary):
    from chllmodel_b200.lattice import Lattice, coupling

    cp = coupling(0.3, 0.9, 0.2)
    out = []
    for other in ("fused", "auto"):
        rng = np.random.default_rng(7)
        lat = Lattice(*shape, boundary=boundary)
        lat.set_kernel(other)
        res = []
        for adapt_until, chunks in ((400, (1, 300, 2)), (0, (1, 6, 2)), (9, (3, 5, 4, 1))):
            f = rng.normal(size=(lat.nsites, 4)).astype(np.float32)
            f[:, :3] /= np.linalg.norm(f[:, :3], axis=1, keepdims=True)
            lat.upload_f4(f)  # chirality: any value, not only a sign
            lat.set_control(0.15, step=1, adapt_until=adapt_until)
            for n in chunks:
                lat.sweep(cp, n, seed=8, replica=1)
            lat.set_kernel("fused")
            lat.sweep(cp, 2, seed=8, replica=1)
            lat.set_kernel(other)
            lat.sweep(cp, 3, seed=8, replica=1)
            res.append((lat.download_f4(), lat.control()))
        out.append(res)
        lat.close()
    for (state, control), (got, got_control) in zip(*out):
        assert np.array_equal(state, got)
        assert control == got_control


@pytest.mark.parametrize("shape,boundary", [((12, 10, 9), "open"), ((30, 18, 10), "periodic"),
                                            ((64, 74, 32), "periodic")])  # a unit per thread
def test_sweeps_and_quench_take_turns(shape, boundary):
    """Both count on one sweep number; a lattice that sweeps by single passes in
    between, and one that is new for every turn, go the same way."""
    from chllmodel_b200.lattice import Lattice, coupling

    cp = coupling(0.3, 0.9, 0.2)
    turns = ((5, 3), (1, 2), (4, 1), (2, 8))
    ends = []
    for mode in ("auto", "fused", "new"):
        lat = Lattice(*shape, boundary=boundary)
        lat.set_kernel("fused" if mode == "fused" else "auto")
        lat.init_random(4)
        for i, (sweeps, steps) in enumerate(turns):
            if mode == "new" and i:
                state, lat = lat.download_f4(), Lattice(*shape, boundary=boundary)
                lat.upload_f4(state)
            lat.set_control(0.1, step=1, adapt_until=3)
            lat.sweep(cp, sweeps, seed=6)
            lat.quench(cp, 0.05, steps)
        ends.append(lat.download_f4())
    assert np.array_equal(ends[0], ends[1])
    assert np.array_equal(ends[0], ends[2])
