"""The measurement row against FP64 numpy: padded rows, odd and single edges,
both boundaries, more columns than threads and several planes per task."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# FP64 arithmetic on the FP32 state: a few roundings per term, sums of N terms of
# order 1 in a fixed tree; 1e-12 of the number of terms is far above either.
RTOL = 1e-12


def _row64(f4, shape, eps, K, g, periodic):
    ni, nj, nk = shape
    a = f4.astype(np.float64).reshape(nk, nj, ni, 4)
    n, s = a[..., :3], a[..., 3]
    E = ref = -g * s.sum()
    for axis, dim in enumerate((2, 1, 0)):
        b, t = np.roll(n, -1, dim), np.roll(s, -1, dim)
        p, q = (axis + 1) % 3, (axis + 2) % 3
        X = n[..., p] * b[..., q] - n[..., q] * b[..., p]
        d = b.copy()
        if axis == 1:
            d[..., 0] = np.roll(b[..., 0], -1, 2)
        for which, other in ((0, b), (1, d)):
            c = (n * other).sum(-1)
            e = eps * (1 - c * c) - K * c * X * 0.5 * (s + t)
            open_end = not periodic if which == 0 else axis == 2
            if open_end:
                e = np.take(e, range(e.shape[dim] - 1), dim)
            if which == 0:
                E += e.sum()
            else:
                ref += e.sum()
    q = [(n[..., i] * n[..., j]).sum() for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    return E, ref, s.sum(), q


@pytest.mark.parametrize("shape,periodic", [
    ((1, 1, 1), False), ((4, 1, 1), False), ((3, 5, 1), False), ((2, 2, 2), True),
    ((6, 4, 2), True), ((5, 3, 7), False), ((8, 7, 3), False), ((33, 9, 6), False),
    ((34, 10, 8), True), ((64, 32, 6), True), ((150, 125, 101), False), ((128, 128, 40), True),
    ((700, 640, 2), True), ((701, 641, 3), False),
])
def test_row_matches_fp64(shape, periodic):
    from chllmodel_b200 import _lib
    from chllmodel_b200.lattice import Lattice, coupling

    N = shape[0] * shape[1] * shape[2]
    lat = Lattice(*shape, boundary="periodic" if periodic else "open")
    lat.init_random(17)
    lat.set_control(0.1, step=8)
    cp = coupling(0.3, 0.9, 0.4, 1.2)
    rows = [lat.observe(cp), lat.observe(cp)]
    lat.reserve_rows(2)
    lat.measure(cp, 1)
    queued = lat.read_rows(1, 1)[0]
    E, ref, S, q = _row64(lat.download_f4(), shape, 1.2, 0.9, 0.4, periodic)
    lat.close()
    assert np.array_equal(rows[0], rows[1])
    assert rows[0][_lib.ROW_STEP] == 7 and queued[_lib.ROW_STEP] == -1
    assert np.array_equal(np.delete(rows[0], _lib.ROW_STEP), np.delete(queued, _lib.ROW_STEP))
    row = rows[0]
    assert abs(row[_lib.ROW_ENERGY] - E) <= RTOL * 8 * N
    assert abs(row[_lib.ROW_ETOT_SUM] - ref) <= RTOL * 8 * N
    assert row[_lib.ROW_SUM_S] == S
    np.testing.assert_allclose(row[_lib.ROW_QXX:_lib.ROW_QXX + 6], q, rtol=0, atol=RTOL * N)
