"""Λ pass on 256-, 384-, 512- and 768-point lines: the tile rule gives every kernel size the three-step
pass on the width that lets two blocks share an SM (73 R1 columns K + 64 R1 + 128 float2 each,
R1 = L / 64), wide grids the widest, grids that do not fill the GPU the narrowest; operators that
do not run it keep wider tiles.  Results against the float64 oracle (float32 bar, 1e-5 relative L2)."""
import ctypes as C

import numpy as np
import pytest

from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu
WIDE = {256: lambda K: 8, 384: lambda K: 8 if K <= 3 else 4, 512: lambda K: 8 if K <= 2 else 4, 768: lambda K: 4 if K <= 3 else 2}
NARROW = {256: 4, 384: 4, 512: 4, 768: 2}


def lambda_pass(mr, A):
    steps, columns = C.c_int(-1), C.c_int(-1)
    assert mr.library().mrsr_test_lambda_pass(A.handle, C.byref(steps), C.byref(columns)) == 0
    return steps.value, columns.value


def operator(mr, rng, img, K, nc, real, precision="fp32"):
    cells = np.flatnonzero(rng.random(4 * int(np.prod(img))) < 0.6) + 1
    shape = (K * (K + 1) // 2, cells.size)
    lam = rng.standard_normal(shape).astype(np.float32) if real else rand_c(rng, shape)
    cm = [rand_c(rng, img) for _ in range(nc)]
    return mr.NFFTNormalOp(img, lam, cells, cmaps=cm, precision=precision), lam, cells, cm


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("L", [256, 384, 512, 768])
@pytest.mark.parametrize("n1,nc", [(40, 16), (12, 2)])
def test_kernel_sizes(mr, cuda, n1, nc, L, K, real):
    rng = np.random.default_rng(61)
    img = (n1, L // 2)
    A, lam, cells, cm = operator(mr, rng, img, K, nc, real)
    steps = 2 if L == 512 and K == 6 and not real else 3
    assert lambda_pass(mr, A) == (steps, WIDE[L](K) if nc == 16 else NARROW[L])
    x = rand_c(rng, img + (K,))
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(mr.to_host(A @ x), ref) < 1e-5


def test_other_operators(mr, cuda):
    rng = np.random.default_rng(62)
    A, _, _, _ = operator(mr, rng, (64, 192), 4, 12, True, "fp16")
    assert lambda_pass(mr, A) == (2, 8)
    F = mr.FFTNormalOp(rand_c(rng, (4, 4, 80, 384)), cmaps=[rand_c(rng, (80, 384)) for _ in range(16)])
    assert lambda_pass(mr, F) == (2, 8)
    A, _, _, _ = operator(mr, rng, (40, 192), 7, 16, True)
    assert lambda_pass(mr, A)[0] == 2
