"""Shell correlations at the edges of the kernel's strips and chunks, against
the numpy oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(shape, boundary, seed):
    from chllmodel_b200.lattice import Lattice, coupling

    lat = Lattice(*shape, boundary=boundary)
    lat.init_random(seed)
    lat.sweep(coupling(0.6, 1.0, 0.2), 3, seed=seed)
    return lat


@pytest.mark.parametrize("shape,shells,wrap", [
    ((1, 1, 1), 1, False), ((5, 1, 4), 3, False), ((7, 8, 2), 4, False), ((6, 9, 5), 6, False),
    ((31, 17, 9), 9, False), ((4, 24, 4), 20, False), ((64, 40, 8), 3, False),
    ((2, 2, 2), 3, True), ((8, 6, 4), 9, True), ((12, 10, 16), 5, True), ((34, 20, 6), 12, True),
    ((4, 6, 4), 64, False),
])
def test_shells(shape, shells, wrap):
    from chllmodel_b200.analysis import shell_correlations
    from oracle import analysis as oa

    lat = _lattice(shape, "periodic" if wrap else "open", 5)
    gn, gs, c = shell_correlations(lat, shells, wrap=wrap)
    again = shell_correlations(lat, shells, wrap=wrap)
    nx, ny, nz, s = lat.download_f64()
    lat.close()
    wn, ws, wc = oa.shell_corr(nx, ny, nz, s, shells, wrap=wrap)
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip((gn, gs, c), again))
    np.testing.assert_array_equal(c, wc)
    has = wc > 0
    # a dot product in FP32 (3 roundings) squared, at most 128 such terms in FP32:
    # relative error below (2 * 3 + 1 + 128) 2^-24 = 8e-6, in practice random
    np.testing.assert_allclose(gn[has], wn[has], rtol=2e-6, atol=1e-7)
    np.testing.assert_allclose(gs[has], ws[has], rtol=0, atol=1e-13)
    assert np.isnan(gn[~has]).all()
