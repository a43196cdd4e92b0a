"""The vector steps of CG at the edges of their batches: fewer unknowns than a block, one more and
one less than whole batches, and several batches per thread, against float64 CG
on the same operator (float32 bar over three iterations, 1e-5 relative L2)."""
import numpy as np
import pytest

from oracle import normalop as onormal
from oracle.cg import cg as ocg
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("img,K", [((3, 2), 1), ((16, 16), 1), ((27, 36), 1), ((32, 32), 1), ((25, 45), 1), ((64, 50), 3),
                                   ((1024, 1024), 1), ((1080, 1000), 1), ((960, 1000), 3)])
def test_solve(mr, cuda, img, K):
    rng = np.random.default_rng(21)
    lam = np.zeros((K, K) + img, np.complex64)  # diagonal kernel, eigenvalues within [1, 3] times the transform's scale
    for k in range(K):
        lam[k, k] = 1 + 2 * rng.random(img)
    lam_c, cells, _ = onormal.fft_normalop_from_lambda(lam)
    b = rand_c(rng, img + (K,))
    got = mr.to_host(mr.cg(mr.FFTNormalOp(lam), b, maxiter=3, reltol=0.0))
    ref = ocg(lambda x: onormal.fft_normalop_apply(x, lam_c, cells, img).ravel(order="F"), b, 3, reltol=0.0)[0]
    assert rel_l2(got, ref.reshape(b.shape, order="F")) < 1e-5
