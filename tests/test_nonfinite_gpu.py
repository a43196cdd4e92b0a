"""Non-finite input of the spreading on register rows: the images (and kernel entries) it reaches are
NaN, whichever component it is in, the others keep the bits they have without it, and a sample that
the mask leaves out does not count.  The entry that is replaced is a small one, so that no maximum
over the rest changes."""
import numpy as np
import pytest

from tests.helpers import rand_c

pytestmark = pytest.mark.gpu
NAN, INF = float("nan"), float("inf")


def _scan(img, K, nc, ns, nt, cplx):
    rng = np.random.default_rng(41)
    trj = (rng.random((len(img), ns, nt)) - 0.5).astype(np.float32)
    U = rand_c(rng, (nt, K)) if cplx else rng.standard_normal((nt, K)).astype(np.float32)
    return rng, trj, U, rand_c(rng, (ns, nt, nc))


@pytest.mark.parametrize("value", [NAN + 0.5j, complex(0.5, NAN), complex(NAN, NAN), complex(INF, 0.5), complex(0.5, -INF)])
@pytest.mark.parametrize("img,K,nc,cplx", [((16, 12), 3, 3, False), ((20, 18), 2, 4, True), ((8, 9, 10), 4, 4, False)])
def test_data(mr, cuda, img, K, nc, cplx, value):
    rng, trj, U, data = _scan(img, K, nc, 90, 4, cplx)
    clean = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U))
    s, t = np.unravel_index(np.argmin(np.abs(data[..., 1])), data.shape[:2])
    data[s, t, 1] = value
    got = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U))
    assert not np.isfinite(got[..., 1]).any()
    keep = [c for c in range(nc) if c != 1]
    np.testing.assert_array_equal(got[..., keep], clean[..., keep])
    # left out by the mask
    mask = np.ones(data.shape[:2], dtype=bool)
    mask[s, t] = False
    got = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U, sample_mask=mask))
    data[s, t, 1] = 0
    ref = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U, sample_mask=mask))
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("value", [NAN, INF])
@pytest.mark.parametrize("img,K,cplx", [((16, 12), 4, False), ((12, 10), 3, True)])
def test_basis(mr, cuda, img, K, cplx, value):
    rng, trj, U, data = _scan(img, K, 2, 90, 6, cplx)
    bp = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U))
    lam = mr.to_host(mr.NFFTNormalOp(img, trj, U).Λ)
    t = np.argmin(np.abs(U[:, 2]))
    U[t, 2] = value
    # a frame that the mask leaves out
    mask = np.ones(data.shape[:2], dtype=bool)
    mask[:, t] = False
    zero = np.where(np.isfinite(U), U, 0).astype(U.dtype)
    for call in (lambda u: mr.calculate_backprojection(data, trj, img, U=u, sample_mask=mask),
                 lambda u: mr.NFFTNormalOp(img, trj, u, sample_mask=mask).Λ):
        np.testing.assert_array_equal(mr.to_host(call(U)), mr.to_host(call(zero)))
    got = mr.to_host(mr.calculate_backprojection(data, trj, img, U=U))
    assert not np.isfinite(got[:, :, 2]).any()
    keep = [k for k in range(K) if k != 2]
    np.testing.assert_array_equal(got[:, :, keep], bp[:, :, keep])
    got = mr.to_host(mr.NFFTNormalOp(img, trj, U).Λ)
    pairs = [(k1, k2) for k2 in range(K) for k1 in range(k2 + 1)]
    for p, pair in enumerate(pairs):
        if 2 in pair:
            assert not np.isfinite(got[p]).any()
        else:
            np.testing.assert_array_equal(got[p], lam[p])


@pytest.mark.parametrize("value", [NAN, INF])
def test_density_compensation(mr, cuda, value):
    img = (16, 12)
    rng, trj, U, data = _scan(img, 3, 2, 90, 4, False)
    w = rng.random(data.shape[:2]).astype(np.float32)
    w[40, 2] = value
    assert not np.isfinite(mr.to_host(mr.calculate_backprojection(data, trj, img, U=U, density_compensation=w))).any()
