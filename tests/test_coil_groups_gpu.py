"""Coil counts around the largest group whose rows fit in a block's shared memory, on row lengths with
padded splits, unpadded ones and none, against the float64 oracle (float32 bar, 1e-5 relative L2)."""
import numpy as np
import pytest

from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1", [162, 160, 256, 128])
@pytest.mark.parametrize("nc", [40, 49, 60, 70, 73])
def test_nfft(mr, cuda, n1, nc):
    rng = np.random.default_rng(91)
    img, K = (n1, 4), 2
    cells = np.flatnonzero(rng.random(16 * n1) < 0.6) + 1
    lam = rng.standard_normal((3, cells.size)).astype(np.float32)
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm) @ x)
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(got, ref) < 1e-5


@pytest.mark.parametrize("nc", [64, 65, 90, 102])
def test_fft_generic(mr, cuda, nc):
    rng = np.random.default_rng(92)
    img, K = (225, 6), 2
    lam = rand_c(rng, (K, K) + img)
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.FFTNormalOp(lam, cmaps=cm) @ x)
    lc, km, _ = onormal.fft_normalop_from_lambda(lam.astype(np.complex128))
    assert rel_l2(got, onormal.fft_normalop_apply(x, lc, km, img, cmaps=cm)) < 1e-5
