"""Tile-sorted spreading where it can go wrong: grids shorter than a window (taps wrap around),
ragged tiles, part counts at the edges of the lane groups (8, 16, 32), tiles with more samples
than a chunk, masks, density compensation, complex bases.

Against the float64 oracle with exact sums; float32 tolerance of the NUFFT paths, 1e-5 relative
L2.  Heavily sampled tiles also have to give the same bits twice: their chunks are cut from
sample lists that atomics filled in any order.
"""
import numpy as np
import pytest

from oracle import backprojection as obp
from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

TOL = 1e-5
pytestmark = pytest.mark.gpu


def _trj(rng, d, ns, nt, spread):
    return (spread * (rng.random((d, ns, nt)) - 0.5)).astype(np.float32)


@pytest.mark.parametrize("img,K,nc,ns,nt,spread,cplx,dcf,masked", [
    ((8, 8), 1, 1, 300, 5, 1.0, False, "none", False),        # 2 parts; grid 16 < window 23; a tile over a chunk
    ((8, 6), 2, 2, 50, 3, 1.0, True, "radial_2D", True),      # 8 parts
    ((16, 12), 3, 3, 120, 4, 1.0, False, "none", False),      # 18 parts: one group of 32
    ((20, 18), 2, 4, 100, 6, 1.0, True, "none", True),        # 16 parts
    ((24, 30), 5, 4, 200, 7, 0.9, False, "radial_3D", False),  # 40 parts: three groups of 16
    ((32, 32), 4, 9, 900, 6, 0.05, False, "none", False),     # 72 parts; one crowded tile
    ((8, 9, 10), 2, 2, 60, 4, 1.0, False, "none", True),      # 3D, 8 parts
    ((12, 8, 15), 3, 6, 150, 3, 1.0, True, "radial_3D", False),  # 3D, 36 parts
    ((9, 10, 8), 1, 3, 700, 2, 0.08, False, "none", False),   # 3D, crowded
])
def test_backprojection_against_exact_sums(mr, cuda, img, K, nc, ns, nt, spread, cplx, dcf, masked):
    rng = np.random.default_rng(3)
    trj = _trj(rng, len(img), ns, nt, spread)
    U = rand_c(rng, (nt, K)) if cplx else rng.standard_normal((nt, K)).astype(np.float32)
    cm = rand_c(rng, img + (nc,))
    data = rand_c(rng, (ns, nt, nc))
    data[0] *= 300.0  # a few samples far above the rest
    m = rng.random((ns, nt)) < 0.7 if masked else None
    cml = [cm[..., c] for c in range(nc)]
    got = mr.to_host(mr.calculate_backprojection(data, trj, cml, U=U, sample_mask=m, density_compensation=dcf))
    again = mr.to_host(mr.calculate_backprojection(data, trj, cml, U=U, sample_mask=m, density_compensation=dcf))
    ref = obp.calculate_backprojection(data, trj, cmaps=cml, U=U, sample_mask=m, density_compensation=dcf)
    assert rel_l2(got, ref) < TOL
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("img,K,ns,nt,spread,cplx", [
    ((8, 10), 3, 80, 4, 1.0, False),      # 6 parts
    ((12, 8), 4, 700, 3, 0.1, False),     # 10 parts, crowded
    ((8, 8), 4, 60, 5, 1.0, True),        # 20 parts
    ((6, 5, 8), 4, 90, 3, 1.0, False),    # 3D: batches of 8 and 2 parts where the grid is large, one here
    ((4, 6, 5), 3, 500, 2, 0.1, True),    # 3D, 12 parts, crowded
])
def test_kernel_against_exact_sums(mr, cuda, img, K, ns, nt, spread, cplx):
    rng = np.random.default_rng(5)
    trj = _trj(rng, len(img), ns, nt, spread)
    U = rand_c(rng, (nt, K)) if cplx else rng.standard_normal((nt, K)).astype(np.float32)
    A = mr.NFFTNormalOp(img, trj, U)
    B = mr.NFFTNormalOp(img, trj, U)
    lam, km = onormal.calculate_kernel_noncartesian(tuple(2 * n for n in img), trj, U)
    np.testing.assert_array_equal(mr.to_host(A.kmask_indcs), km)
    got = mr.to_host(A.Λ)
    assert rel_l2(got, onormal.pack_lambda(lam, real=not cplx)) < TOL
    np.testing.assert_array_equal(got, mr.to_host(B.Λ))
