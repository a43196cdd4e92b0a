"""Middle axes of 3D operators where their column tiles are as wide as shared memory allows: lines
up to 512 points on 16 columns, longer ones (compiled and generic) on 8."""
import numpy as np
import pytest

from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img", [(8, 256, 3), (8, 243, 2), (8, 300, 2), (8, 450, 2), (4, 486, 3), (8, 512, 2), (5, 40, 4), (9, 32, 3)])
def test_apply_3d(mr, cuda, img):
    rng = np.random.default_rng(7)
    K, nc = 2, 2
    G = tuple(2 * n for n in img)
    cells = np.flatnonzero(rng.random(int(np.prod(G))) < 0.6) + 1
    lam = rand_c(rng, (K * (K + 1) // 2, cells.size))
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm) @ x)
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(got, ref) < 1e-5
