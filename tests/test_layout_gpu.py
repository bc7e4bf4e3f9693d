"""Uploads over a lattice that held something else: every site arrives, padding
slots read zero, and the state comes back unchanged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Slots:
    """One colour's storage as a CUDA array."""

    def __init__(self, ptr, slots):
        self.__cuda_array_interface__ = {"shape": (slots, 4), "typestr": "<f4",
                                         "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("how", ["f4", "f64", "random"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 7, 3), (2, 3, 5), (3, 2, 4), (4, 1, 2), (5, 6, 7),
                                   (64, 3, 2), (150, 25, 11)])
def test_uploads_fill_padded_rows(shape, how):
    import torch

    from chllmodel_b200.lattice import Lattice, from_f4

    N = shape[0] * shape[1] * shape[2]
    lat = Lattice(*shape, boundary="open")
    c0, c1, per_colour, hx = lat.storage()
    colours = [torch.as_tensor(_Slots(p, per_colour), device="cuda") for p in (c0, c1)]
    for t in colours:
        t.fill_(9.0)
    torch.cuda.synchronize()
    rng = np.random.default_rng(N)
    f4 = rng.standard_normal((N, 4)).astype(np.float32)
    f4[:, 3] = np.sign(f4[:, 3])
    if how == "f4":
        lat.upload_f4(f4)
    elif how == "f64":
        lat.upload_f64(*from_f4(f4, *shape))
    else:
        lat.init_random(3)
        lat.sync()
    out = torch.stack(colours).view(2, shape[2], shape[1], hx, 4).cpu().numpy()
    c, k, j, h = np.meshgrid(*(np.arange(v) for v in out.shape[:4]), indexing="ij")
    padding = 2 * h + ((c + j + k) & 1) >= shape[0]
    assert not out[padding].any()
    if how == "random":
        assert np.allclose(np.linalg.norm(out[~padding][:, :3], axis=1), 1.0, atol=1e-6)
    else:
        assert np.array_equal(lat.download_f4(), f4)
    lat.close()
