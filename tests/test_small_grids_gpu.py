"""Operators whose passes do not fill the GPU: the column tiles and row blocks shrink with the grid.
Sizes on both sides of the rule (one coil to many, one tile to many), two- and three-step lines,
plain and stacked, against the float64 oracle (float32 bar, 1e-5 relative L2)."""
import numpy as np
import pytest

from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,K,nc", [((32, 32), 4, 1), ((32, 32), 4, 12), ((45, 36), 3, 2), ((64, 64), 2, 1), ((64, 128), 6, 1),
                                      ((256, 40), 2, 1), ((40, 256), 5, 1), ((40, 256), 5, 8), ((4, 32), 1, 1), ((1, 32), 2, 3)])
def test_apply(mr, cuda, img, K, nc):
    rng = np.random.default_rng(9)
    G = tuple(2 * n for n in img)
    cells = np.flatnonzero(rng.random(int(np.prod(G))) < 0.7) + 1
    lam = rng.standard_normal((K * (K + 1) // 2, cells.size)).astype(np.float32)
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm) @ x)
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(got, ref) < 1e-5


@pytest.mark.parametrize("img,n", [((32, 32), 2), ((32, 32), 40), ((16, 128), 3)])
def test_stacked(mr, cuda, img, n):
    rng = np.random.default_rng(10)
    cells = np.flatnonzero(rng.random(4 * int(np.prod(img))) < 0.7) + 1
    lam = rng.standard_normal((1, cells.size)).astype(np.float32)
    A = mr.NFFTNormalOp(img, lam, cells)
    x = rand_c(rng, img + (n,))
    got = mr.to_host(A.stack(n) @ x)
    full = onormal.unpack_lambda(lam.astype(np.complex128), 1)
    for i in range(n):
        assert rel_l2(got[..., i:i + 1], onormal.nfft_normalop_apply(x[..., i:i + 1], full, cells, img)) < 1e-5
