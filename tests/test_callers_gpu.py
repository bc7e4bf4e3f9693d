"""Callers other than one lattice on its own stream: lattices that sweep, measure and
quench at once from threads, and the natural-order adjoint of tensors of other types
and strides, on another stream, with couplings on the device."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 32), "periodic"), ((48, 48, 48), "open"), ((64, 64, 64), "periodic"),
          ((96, 96, 96), "periodic"), ((33, 31, 17), "open"), ((8, 8, 8), "periodic")]


@pytest.mark.parametrize("own_stream", [True, False])
def test_lattices_at_once_follow_their_chains(own_stream):
    import torch

    from chllmodel_b200.lattice import Lattice, coupling

    cp = coupling(0.5, 0.8, 0.1)

    def chain(i, out):
        shape, boundary = SHAPES[i]
        lat = Lattice(*shape, boundary=boundary)
        stream = torch.cuda.Stream()
        if not own_stream:
            lat.set_stream(stream.cuda_stream)
        lat.init_random(7, i)
        lat.set_control(0.1, step=1)
        rows = []
        for n in (50, 13, 77):
            lat.sweep(cp, n, seed=3, replica=i)
            rows.append(lat.observe(cp))
        lat.quench(cp, 0.05, 40)
        out[i] = (lat.download_f4(), np.array(rows), lat.energy_sums(cp), lat.control())
        lat.close()

    alone, together = {}, {}
    for i in range(len(SHAPES)):
        chain(i, alone)
    for _ in range(2):
        threads = [threading.Thread(target=chain, args=(i, together)) for i in range(len(SHAPES))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in range(len(SHAPES)):
            for a, b in zip(alone[i][:3], together[i][:3]):
                assert np.array_equal(a, b)
            assert alone[i][3] == together[i][3]


def _energy(n, s, eps, K, h, shape, periodic):
    """The lattice energy in torch, FP64."""
    import torch

    ni, nj, nk = shape
    n, s = n.reshape(nk, nj, ni, 3), s.reshape(nk, nj, ni)
    total = -h * s.sum()
    for dim, axis in ((2, 0), (1, 1), (0, 2)):
        m, t = torch.roll(n, -1, dim), torch.roll(s, -1, dim)
        c = (n * m).sum(-1)
        e = eps * (1 - c * c) - K * c * torch.cross(n, m, dim=-1)[..., axis] * 0.5 * (s + t)
        total = total + (e if periodic else e.narrow(dim, 0, e.shape[dim] - 1)).sum()
    return total


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("couplings", ["cpu", "cuda"])
def test_adjoint_of_other_tensors(dtype, strided, couplings):
    import torch

    from chllmodel_b200.autograd import lattice_energy, tangent_gradient

    dt = getattr(torch, dtype)
    shape, values = (12, 10, 6), (1.2, 0.7, 0.3)
    N = shape[0] * shape[1] * shape[2]
    g = torch.Generator().manual_seed(1)
    # FP32 values in either type: the kernel's inputs are exactly these
    n = torch.nn.functional.normalize(torch.randn(N, 3, generator=g), dim=1).double()
    s = (torch.randint(0, 2, (N,), generator=g) * 2 - 1).double()
    r = n.clone().requires_grad_(True)
    rc = [torch.tensor(v, dtype=torch.float64, requires_grad=True) for v in values]
    E = _energy(r, s, *rc, shape, True)
    (2.5 * E).backward()
    with torch.cuda.stream(torch.cuda.Stream()):
        x = n.to(dt).cuda()
        t = s.to(dt).cuda()
        if strided:
            x = x.t().contiguous().t()
            t = torch.stack([t, -t], 1)[:, 0]
        x.requires_grad_(True)
        c = [torch.tensor(v, dtype=torch.float64, device=couplings, requires_grad=True)
             for v in values]
        e = lattice_energy(x, t, *c, shape)
        (2.5 * e).backward()
        torque = tangent_gradient(x, t, *values, shape)
        torch.cuda.current_stream().synchronize()
    assert x.grad.dtype == dt and x.grad.shape == x.shape
    # FP32 sums of six bonds of order 1, scaled by 2.5
    assert (x.grad.double().cpu() - r.grad).abs().max() < 2e-5
    G = r.grad / 2.5
    G = G - (G * n).sum(1, keepdim=True) * n / (n * n).sum(1, keepdim=True)
    assert (torque.double().cpu() - G).abs().max() < 2e-5
    assert e.item() == pytest.approx(E.item(), rel=1e-11, abs=1e-11)
    for a, b in zip(c, rc):
        assert a.grad.device == a.device
        assert a.grad.item() == pytest.approx(b.grad.item(), rel=1e-11, abs=1e-11)
