"""3D spreading on both sides of the rule that picks its kernel (few parts, crowded grids and padded
lanes on shared-memory windows, the rest on register rows): against the float64 oracle with exact
sums (float32 tolerance of the NUFFT paths, 1e-5 relative L2), and the same bits twice."""
import numpy as np
import pytest

from oracle import backprojection as obp
from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,nc,ns,spread,cplx", [
    (1, 1, 900, 1.0, False), (2, 2, 300, 1.0, True), (1, 13, 200, 0.1, False),  # 2, 8, 26 parts
    (3, 5, 200, 1.0, False), (4, 4, 1500, 0.1, True), (5, 4, 200, 1.0, False),  # 30, 32, 40 parts
])
def test_backprojection(mr, cuda, K, nc, ns, spread, cplx):
    rng = np.random.default_rng(31)
    img, nt = (9, 8, 12), 3
    trj = (spread * (rng.random((3, ns, nt)) - 0.5)).astype(np.float32)
    U = rand_c(rng, (nt, K)) if cplx else rng.standard_normal((nt, K)).astype(np.float32)
    cml = [rand_c(rng, img) for _ in range(nc)]
    data = rand_c(rng, (ns, nt, nc))
    run = lambda: mr.to_host(mr.calculate_backprojection(data, trj, cml, U=U, density_compensation="radial_3D"))
    got = run()
    assert rel_l2(got, obp.calculate_backprojection(data, trj, cmaps=cml, U=U, density_compensation="radial_3D")) < 1e-5
    np.testing.assert_array_equal(got, run())


@pytest.mark.parametrize("img,K,cplx", [((20, 20, 24), 1, False), ((20, 20, 24), 3, False), ((20, 20, 24), 4, False),
                                        ((20, 20, 24), 3, True), ((8, 9, 10), 4, False)])
def test_kernel(mr, cuda, img, K, cplx):
    rng = np.random.default_rng(32)
    trj = (rng.random((3, 60, 2)) - 0.5).astype(np.float32)
    U = rand_c(rng, (2, K)) if cplx else rng.standard_normal((2, K)).astype(np.float32)
    got = mr.to_host(mr.NFFTNormalOp(img, trj, U).Λ)
    lam, _ = onormal.calculate_kernel_noncartesian(tuple(2 * n for n in img), trj, U)
    assert rel_l2(got, onormal.pack_lambda(lam, real=not cplx)) < 1e-5
    np.testing.assert_array_equal(got, mr.to_host(mr.NFFTNormalOp(img, trj, U).Λ))
