"""The adjoint of natural-order arrays against a plain FP64 torch energy and
its automatic derivative: row and warp ends, single planes and rows, more
columns than threads."""
import pytest

pytestmark = pytest.mark.gpu

# Six bond terms of FP32 products per site, each a few roundings of magnitude
# |K| + 2 |eps| <= 4: absolute error below 6 * 8 * 4 * 2^-24 = 1.2e-5; FP64
# sums of at most 5e5 terms of order 1: far below 1e-11 relative to sum |terms|.
GRAD_ATOL, SUM_RTOL = 1.2e-5, 1e-11


def _energy64(n, s, eps, K, h, shape, periodic):
    import torch

    ni, nj, nk = shape
    n, s = n.view(nk, nj, ni, 3), s.view(nk, nj, ni)
    E = -h * s.sum()
    for axis, dim in enumerate((2, 1, 0)):
        L = n.shape[dim]
        b, t = torch.roll(n, -1, dim), torch.roll(s, -1, dim)
        a, u = n, s
        if not periodic:
            a, b, u, t = (v.narrow(dim, 0, L - 1) for v in (a, b, u, t))
        p, q = (axis + 1) % 3, (axis + 2) % 3
        c = (a * b).sum(-1)
        X = a[..., p] * b[..., q] - a[..., q] * b[..., p]
        E = E + (eps * (1 - c * c) - K * c * X * 0.5 * (u + t)).sum()
    return E


@pytest.mark.parametrize("shape,boundary", [
    ((1, 1, 1), "open"), ((1, 5, 3), "open"), ((2, 2, 2), "periodic"), ((32, 1, 1), "open"),
    ((33, 3, 2), "open"), ((31, 2, 9), "open"), ((64, 2, 4), "periodic"), ((30, 18, 10), "periodic"),
    ((250, 41, 7), "open"), ((400, 400, 3), "open"), ((16, 8, 130), "periodic"),
])
def test_natural_adjoint(shape, boundary):
    import torch

    from chllmodel_b200.autograd import coupling_sensitivities, lattice_energy, tangent_gradient

    N = shape[0] * shape[1] * shape[2]
    gen = torch.Generator(device="cuda").manual_seed(N)
    n = torch.randn((N, 3), generator=gen, device="cuda")
    n = (n / n.norm(dim=1, keepdim=True)).requires_grad_(True)
    s = torch.where(torch.rand(N, generator=gen, device="cuda") < 0.5, -1.0, 1.0)
    c = [torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in (1.2, 0.9, 0.3)]
    E = lattice_energy(n, s, *c, shape, boundary)
    got = torch.autograd.grad(E, [n] + c)
    n64 = n.detach().double().requires_grad_(True)
    want_E = _energy64(n64, s.double(), *c, shape, boundary == "periodic")
    want = torch.autograd.grad(want_E, [n64] + c)
    size = 5.0 * N  # bounds the sum of the terms' magnitudes
    assert abs(float(E) - float(want_E)) <= SUM_RTOL * size
    assert float((got[0] - want[0]).abs().max()) <= GRAD_ATOL
    for g, w in zip(got[1:], want[1:]):
        assert g.device == w.device and abs(float(g) - float(w)) <= SUM_RTOL * size
    t = tangent_gradient(n, s, 1.2, 0.9, 0.3, shape, boundary)
    m = n64.detach()
    wt = want[0] - (want[0] * m).sum(1, keepdim=True) * m / (m * m).sum(1, keepdim=True)
    assert t.shape == (N, 3) and float((t - wt).abs().max()) <= 3 * GRAD_ATOL
    sens = coupling_sensitivities(n.detach().cpu(), s.cpu(), 1.2, 0.9, 0.3, shape, boundary)
    assert abs(sens["E"] - float(want_E)) <= SUM_RTOL * size
    assert abs(sens["dE_dK"] - float(want[2])) <= SUM_RTOL * size


def test_natural_adjoint_refuses_what_a_lattice_refuses():
    import torch

    from chllmodel_b200._lib import ChllError
    from chllmodel_b200.autograd import lattice_energy, tangent_gradient

    n, s = torch.ones((27, 3), device="cuda"), torch.ones(27, device="cuda")
    with pytest.raises(ChllError, match="even"):
        lattice_energy(n, s, 1.0, 1.0, 0.0, (3, 3, 3), "periodic")
    with pytest.raises(ValueError):
        lattice_energy(n, s, 1.0, 1.0, 0.0, (3, 3, 4), "open")
    with pytest.raises(ValueError):
        tangent_gradient(n, s, 1.0, 1.0, 0.0, (3, 3, 4), "open")
