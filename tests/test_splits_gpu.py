"""Every line length with compiled two-step kernels (csrc/splits.cuh), in each role: first axis
(row passes), last axis (Λ pass) and middle axis (3D), zero-padded (NFFT operator) and whole (FFT
operator), and the batched transform of the Cartesian backprojection.  Float32 bar: 1e-5 relative
L2 against the float64 oracle."""
import re
from pathlib import Path

import numpy as np
import pytest

from oracle import backprojection as obp
from oracle import normalop as onormal
from tests.helpers import rand_c, rel_l2

TOL = 1e-5
pytestmark = pytest.mark.gpu
SPLITS = Path(__file__).resolve().parents[1] / "mrfingerprintingrecon.jl_gb300" / "csrc" / "splits.cuh"
LENGTHS = sorted({int(m) for m in re.findall(r"X\((\d+), \d+, \d+\)", SPLITS.read_text())})


def test_list_of_lengths():
    assert len(LENGTHS) == 41 and all(n % 2 == 0 for n in LENGTHS)


def _nfft(mr, rng, img, K, nc, cplx):
    G = tuple(2 * n for n in img)
    cells = np.flatnonzero(rng.random(int(np.prod(G))) < 0.6) + 1
    P = K * (K + 1) // 2
    lam = rand_c(rng, (P, cells.size)) if cplx else rng.standard_normal((P, cells.size)).astype(np.float32)
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.NFFTNormalOp(img, lam, cells, cmaps=cm) @ x)
    ref = onormal.nfft_normalop_apply(x, onormal.unpack_lambda(lam.astype(np.complex128), K), cells, img, cmaps=cm)
    assert rel_l2(got, ref) < TOL


def _fft(mr, rng, img, K, nc):
    lam = rand_c(rng, (K, K) + img)
    lam[0, 0][rng.random(img) < 0.4] = 0
    cm = [rand_c(rng, img) for _ in range(nc)]
    x = rand_c(rng, img + (K,))
    got = mr.to_host(mr.FFTNormalOp(lam, cmaps=cm) @ x)
    lc, km, _ = onormal.fft_normalop_from_lambda(lam.astype(np.complex128))
    assert rel_l2(got, onormal.fft_normalop_apply(x, lc, km, img, cmaps=cm)) < TOL


@pytest.mark.parametrize("L", LENGTHS)
def test_operators(mr, cuda, L):
    rng = np.random.default_rng(L)
    _nfft(mr, rng, (L // 2, 9), 3, 3, False)
    _nfft(mr, rng, (10, L // 2), 2, 2, True)
    _fft(mr, rng, (L, 15), 2, 2)
    _fft(mr, rng, (9, L), 3, 1)
    _nfft(mr, rng, (5, L // 2, 3), 2, 2, False)
    _fft(mr, rng, (4, L, 3), 1, 2)


@pytest.mark.parametrize("L", LENGTHS)
def test_batched_transform(mr, cuda, L):
    rng = np.random.default_rng(L)
    img, ns, nt, nc, K = (L, 6), 200, 3, 2, 2
    trj = np.stack([rng.integers(1, n + 1, (ns, nt)) for n in img]).astype(np.int32)
    data, U = rand_c(rng, (ns, nt, nc)), rand_c(rng, (nt, K))
    cm = [rand_c(rng, img) for _ in range(nc)]
    got = mr.to_host(mr.calculate_backprojection(data, trj, cm, U=U))
    assert rel_l2(got, obp.calculate_backprojection_cartesian(data, trj, cmaps=cm, U=U)) < TOL
