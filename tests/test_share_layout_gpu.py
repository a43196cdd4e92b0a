"""Operators on a shared kernel run the tiles of their own coil count: results with the bits of an
operator built directly, the kernel read back unchanged, whatever the source was laid out for."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import rand_c

pytestmark = pytest.mark.gpu


def columns(mr, A):
    steps, cols = C.c_int(-1), C.c_int(-1)
    assert mr.library().mrsr_test_lambda_pass(A.handle, C.byref(steps), C.byref(cols)) == 0
    return cols.value


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("img,K,prec,one,many", [
    ((40, 192), 4, "fp32", 4, 4),   # 384 points: one layout
    ((40, 256), 2, "fp32", 4, 8),   # 512 points: copied for many coils
    ((40, 64), 4, "fp32", 2, 8),    # 128 points, two steps: the same
    ((45, 50), 3, "fp32", 2, 2),    # 100 points: 90 columns take no wider tile
    ((64, 192), 4, "fp16", 4, 8),   # fp16 tiles are not the float32 ones
    ((64, 64), 3, "fp16", 2, 8),
])
def test_share(mr, cuda, img, K, prec, one, many, real):
    rng = np.random.default_rng(71)
    cells = np.flatnonzero(rng.random(4 * int(np.prod(img))) < 0.6) + 1
    shape = (K * (K + 1) // 2, cells.size)
    lam = rng.standard_normal(shape).astype(np.float32) if real else rand_c(rng, shape)
    cm = [rand_c(rng, img) for _ in range(24)]
    x = rand_c(rng, img + (K,))
    direct = mr.NFFTNormalOp(img, lam, cells, cmaps=cm, precision=prec)
    ref = mr.to_host(direct @ x)
    assert columns(mr, direct) == many
    for maps, shared in ((None, False), (cm[:1], False), (None, True)):
        src = mr.NFFTNormalOp(img, lam, cells, cmaps=maps, shared=shared)
        assert shared or columns(mr, src) == one
        A, B = src.share(cmaps=cm, precision=prec), src.share(cmaps=cm, precision=prec)
        src.close()
        for op in (A, B):
            assert columns(mr, op) == many
            np.testing.assert_array_equal(mr.to_host(op @ x), ref)
            np.testing.assert_array_equal(mr.to_host(op.Λ), lam)
            np.testing.assert_array_equal(mr.to_host(op.kmask_indcs), cells)
        # few coils on a kernel for many: the wider tiles, shared
        np.testing.assert_array_equal(mr.to_host(A.share(cmaps=cm[:2], precision="fp32") @ x),
                                      mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm[:2]) @ x))
