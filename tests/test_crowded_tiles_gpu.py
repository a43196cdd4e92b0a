"""The order of crowded tiles in the tile sort: lists of one bitmap window and of two, lists short enough
to be ranked by pairs (20M samples: segments of 312k, lists of 385 to 395), against exact sums.
Samples sit on a few positions, so their exact backprojection is that of the summed data
(float32 NUFFT tolerance, 1e-5 relative L2), and a second run has to give the same bits."""
import numpy as np
import pytest
import torch

from oracle import nudft
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,ns,nt", [((8, 8), 400, 3), ((16, 12), 30000, 4), ((80, 64), 5000000, 4), ((6, 8, 9), 60000, 3)])
def test_backprojection(mr, cuda, img, ns, nt):
    rng = np.random.default_rng(51)
    d, n = len(img), ns * nt
    pos = (rng.random((d, 60)) - 0.5).astype(np.float32)
    pos[:, :20] *= 0.05  # one crowded tile (wrapped: at most 2^d)
    p = np.full(60, 0.00125)
    p[:20] = (1 - 40 * 0.00125) / 20
    at = rng.choice(60, size=n, p=p)
    trj = np.ascontiguousarray(pos[:, at].reshape((d, ns, nt), order="F"))
    K, nc = (4, 4) if d == 3 else (2, 1)  # 32 parts: the 3D rule takes register rows
    data = rng.standard_normal((nc * n, 2), dtype=np.float32).view(np.complex64).reshape((ns, nt, nc), order="F")
    U = rng.standard_normal((nt, K)).astype(np.float32)
    got = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U))
    fr, c, k = np.repeat(np.arange(nt), ns), nc - 1, K - 1
    v = data[..., c].reshape(-1, order="F") * U[fr, k].astype(np.float64)
    s = np.bincount(at, v.real, 60) + 1j * np.bincount(at, v.imag, 60)
    assert rel_l2(got[..., k, c], nudft.adjoint(s, pos.astype(np.float64), img)) < 1e-5
    np.testing.assert_array_equal(got, mr.to_host(mr.calculate_backprojection(data, trj, img, U=U)))
    torch.cuda.empty_cache()
