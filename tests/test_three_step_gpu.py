"""Three-step Λ pass on 256-, 384-, 512- and 768-point lines: every kernel size it takes, real and
complex, on tiles of 2, 4 and 8 columns (the plane's width and K choose) and beside the two-step
pass (a plane whose width is no multiple of the tile), against the float64 oracle (float32 bar,
1e-5 relative L2)."""
import numpy as np
import pytest

from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


def check(mr, img, K, nc, real, seed):
    rng = np.random.default_rng(seed)
    G = tuple(2 * n for n in img)
    cells = np.flatnonzero(rng.random(int(np.prod(G))) < 0.6) + 1
    shape = (K * (K + 1) // 2, cells.size)
    lam = rng.standard_normal(shape).astype(np.float32) if real else rand_c(rng, shape)
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm) @ x)
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(got, ref) < 1e-5


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("img", [(12, 192), (12, 384), (12, 128), (12, 256)])
def test_kernel_sizes(mr, cuda, img, K, real):
    check(mr, img, K, 2, real, 11)


@pytest.mark.parametrize("img,K,nc", [((80, 192), 3, 20), ((80, 192), 4, 20), ((80, 384), 1, 20), ((80, 384), 3, 20),
                                      ((9, 192), 3, 2), ((1, 384), 2, 3), ((6, 4, 192), 2, 3), ((80, 256), 2, 20)])
def test_tiles(mr, cuda, img, K, nc):
    check(mr, img, K, nc, True, 12)


@pytest.mark.parametrize("img", [(20, 192), (20, 384)])
def test_stacked(mr, cuda, img):
    rng = np.random.default_rng(13)
    n = 5
    cells = np.flatnonzero(rng.random(4 * int(np.prod(img))) < 0.7) + 1
    lam = rng.standard_normal((1, cells.size)).astype(np.float32)
    x = rand_c(rng, img + (n,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells).stack(n) @ x)
    full = onormal.unpack_lambda(lam.astype(np.complex128), 1)
    for i in range(n):
        assert rel_l2(got[..., i:i + 1], onormal.nfft_normalop_apply(x[..., i:i + 1], full, cells, img)) < 1e-5
