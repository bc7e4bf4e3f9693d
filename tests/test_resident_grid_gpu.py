"""The resident launch's shapes: one CTA, one unit per thread and more, padded
rows, one-site lattices -- each the fused passes' chain bit for bit, also after
single passes that leave counts open."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,boundary", [
    ((1, 1, 1), "open"), ((3, 2, 1), "open"), ((2, 2, 2), "periodic"),
    ((8, 8, 8), "periodic"),                                    # one CTA
    ((16, 16, 4), "periodic"), ((16, 16, 5), "open"),           # 256 units, and the next plane
    ((33, 31, 17), "open"), ((30, 18, 10), "open"),             # padded rows, a unit each
    ((30, 18, 10), "periodic"),                                 # padded rows, unit loop
    ((64, 74, 64), "periodic"), ((64, 74, 64), "open"),         # 75,776 units: 148 x 512
    ((64, 76, 64), "periodic"), ((64, 76, 64), "open"),         # more units than threads
    ((67, 75, 65), "open"), ((128, 64, 66), "periodic"),
])
def test_resident_equals_fused(shape, boundary):
    from chllmodel_b200.lattice import FUSED_A0, FUSED_B, Lattice, coupling

    cp = coupling(0.5, 0.7, 0.1)
    out = []
    for kind in ("fused", "resident", "auto"):
        lat = Lattice(*shape, boundary=boundary)
        lat.set_kernel(kind)
        lat.init_random(11)
        lat.set_control(0.1, step=1, adapt_until=12)
        for n in (1, 2, 7):
            lat.sweep(cp, n, seed=(5 << 32) + 3, replica=2)
        lat.half_sweep(cp, FUSED_A0, seed=4)
        lat.half_sweep(cp, FUSED_B, seed=4)
        for n in (1, 5):
            lat.sweep(cp, n, seed=4)
        out.append((lat.download_f4(), lat.control()))
        lat.close()
    for state, control in out[1:]:
        assert np.array_equal(out[0][0], state)
        assert out[0][1] == control
