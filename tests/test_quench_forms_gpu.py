"""The quench's forms: one site or unit per thread, the unit loop and a launch per pass
follow the same steps, and each step is the FP64 one to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tiled(shape, copies, steps):
    from chllmodel_b200.lattice import Lattice, coupling

    base = Lattice(*shape, boundary="periodic")
    base.init_random(5)
    f4 = base.download_f4()
    base.close()
    lat = Lattice(shape[0], shape[1], shape[2] * copies, boundary="periodic")
    lat.upload_f4(np.tile(f4, (copies, 1)))
    cp = coupling(0.0, 0.9, 0.4, 1.1)
    for n in steps:
        lat.quench(cp, 0.05, n)
    out = lat.download_f4()
    sums = lat.energy_sums(cp)
    _, both = lat.energy_grad(cp)
    assert np.array_equal(sums, both)
    lat.close()
    return out.reshape(copies, -1, 4)


@pytest.mark.parametrize("shape,copies", [((64, 64, 32), (1, 2, 4, 18)),   # 32,768 .. 589,824 units
                                          ((64, 74, 32), (1, 2)),  # 75,776 and 151,552 slots
                                          ((62, 74, 28), (1, 2)),  # padded: 66,304, 132,608
                                          ((30, 18, 10), (1, 3, 30, 440))])  # padded rows
def test_forms_agree(shape, copies):
    """A lattice repeated along z stays a repetition: every copy equals the
    smallest lattice's run, whatever form its size takes."""
    runs = [_tiled(shape, c, (1, 2, 9)) for c in copies]
    for run in runs:
        for copy in run:
            assert np.array_equal(copy, runs[0][0])


@pytest.mark.parametrize("shape,periodic", [((1, 1, 1), False), ((4, 4, 1), False), ((33, 5, 3), False),
                                            ((8, 8, 8), True), ((6, 4, 2), True),
                                            ((65, 61, 20), False)])
def test_steps_match_fp64(shape, periodic):
    from chllmodel_b200.lattice import Lattice, coupling

    ni, nj, nk = shape
    eps, K, h, eta, steps = 1.1, 0.9, 0.4, 0.05, 3
    lat = Lattice(*shape, boundary="periodic" if periodic else "open")
    lat.init_random(3)
    f4 = lat.download_f4()
    lat.quench(coupling(0.0, K, h, eps), eta, steps)
    got = lat.download_f4()
    lat.close()
    a = f4.astype(np.float64).reshape(nk, nj, ni, 4)
    n, s = a[..., :3].copy(), a[..., 3]
    k, j, i = np.meshgrid(*(np.arange(v) for v in (nk, nj, ni)), indexing="ij")
    for _ in range(steps):
        for colour in (0, 1):
            g = np.zeros_like(n)
            for axis, (dim, pos) in enumerate(((2, i), (1, j), (0, k))):
                p, q = (axis + 1) % 3, (axis + 2) % 3
                for shift, sigma in ((-1, -1.0), (1, 1.0)):
                    b = np.roll(n, shift, dim)
                    w = sigma * K * 0.5 * (s + np.roll(s, shift, dim))
                    c = (n * b).sum(-1)
                    X = n[..., p] * b[..., q] - n[..., q] * b[..., p]
                    t = (-2 * eps * c + w * X)[..., None] * b
                    t[..., p] += w * c * b[..., q]
                    t[..., q] -= w * c * b[..., p]
                    if not periodic:
                        t[pos == (n.shape[dim] - 1 if shift < 0 else 0)] = 0
                    g += t
            tang = g - ((g * n).sum(-1) / (n * n).sum(-1))[..., None] * n
            m = n - eta * tang
            m /= np.linalg.norm(m, axis=-1, keepdims=True)
            n[(i + j + k) % 2 == colour] = m[(i + j + k) % 2 == colour]
    # a step rounds a handful of FP32 operations of order 1 (eta of the gradient's
    # dozens): below 20 * 2^-24 per step, hardly amplified in three
    np.testing.assert_allclose(got[:, :3].reshape(nk, nj, ni, 3), n, rtol=0, atol=8e-6)
    assert np.array_equal(got[:, 3], f4[:, 3])
