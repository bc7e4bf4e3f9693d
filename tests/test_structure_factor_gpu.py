"""The structure factor at the edges of its kernels' runs and bins, against the
numpy oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(shape, boundary, seed):
    from chllmodel_b200.lattice import Lattice, coupling

    lat = Lattice(*shape, boundary=boundary)
    lat.init_random(seed)
    lat.sweep(coupling(0.6, 1.0, 0.2), 3, seed=seed)
    return lat


@pytest.mark.parametrize("shape", [(1, 1, 1), (6, 5, 4), (33, 3, 70), (7, 64, 9), (130, 40, 24)])
@pytest.mark.parametrize("plane", [(1, 1, 1), (0, 0, 1), (1, 0, 0), (0, 1, 0), (1, -1, 2), (0, 2, -3),
                                   (-3, 1, 0), (0, 0, 0)])
def test_structure_factor(shape, plane):
    from chllmodel_b200.analysis import projection, structure_factor
    from oracle import analysis as oa

    lat = _lattice(shape, "open", 9)
    s = lat.download_f64()[3]
    m, hist = projection(lat, plane)
    sf, kvs = structure_factor(lat, 23, 0.0, 3.0, plane)
    none, _ = structure_factor(lat, 0, 0.0, 3.0, plane)
    lat.close()
    i, j, k = np.meshgrid(*(np.arange(1, n + 1) for n in shape), indexing="ij")
    at = plane[0] * i + plane[1] * j + plane[2] * k
    assert np.array_equal(hist, [s[at == v].sum() for v in m])
    want, wk = oa.structure_factor(s, 23, 0.0, 3.0, plane)
    assert np.array_equal(kvs, wk) and none.shape == (0,)
    np.testing.assert_allclose(sf, want, rtol=1e-9, atol=1e-13)
