"""Forward model over the plane groups of its interpolation (16 planes, whole coils): ranks 1 to 8
with coil counts that fill, split and leave a group, grids shorter than a window, against the exact
sums (float32 NUFFT tolerance, 1e-5 relative L2)."""
import numpy as np
import pytest

from oracle import nudft
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,K,nc,ns,nt,cplx", [
    ((8, 6), 1, 17, 40, 3, False),    # 16 coils a group; grid 16 x 12 < window 23
    ((16, 12), 2, 9, 70, 4, True),
    ((20, 20), 3, 6, 33, 5, False),   # five coils a group
    ((12, 30), 4, 4, 50, 3, True),
    ((24, 18), 5, 4, 1200, 2, False),  # more samples than an item takes in one tile: see the spread below
    ((9, 10), 6, 3, 60, 3, False),
    ((10, 8), 7, 3, 25, 4, True),
    ((18, 16), 8, 5, 64, 2, False),   # two coils a group
])
def test_against_exact_sums(mr, cuda, img, K, nc, ns, nt, cplx):
    rng = np.random.default_rng(11)
    spread = 0.05 if ns > 1000 else 1.0
    trj = (spread * (rng.random((2, ns, nt)) - 0.5)).astype(np.float32)
    U = rand_c(rng, (nt, K)) if cplx else rng.standard_normal((nt, K)).astype(np.float32)
    x, cm = rand_c(rng, img + (K,)), rand_c(rng, img + (nc,))
    got = mr.to_host(mr.forward_model(x, trj, U, cmaps=cm))
    pts = trj.reshape(2, -1, order="F").astype(np.float64)
    fr = np.repeat(np.arange(nt), ns)
    ref = np.zeros((ns, nt, nc), dtype=np.complex128)
    for c in range(nc):
        y = sum(U[fr, k] * nudft.forward(cm[..., c] * x[..., k], pts) for k in range(K))
        ref[:, :, c] = y.reshape(ns, nt, order="F")
    assert rel_l2(got, ref) < 1e-5
