"""GROG kernels at the edges of their coil groups, against the float64 oracle (src/GROG.jl).

Calibration on spokes of known operators: rows d_{r+1} = G d_r, plus noise, with G = exp(B) of a
B whose eigenvalues stay clear of the logarithm's cut, so lnG is well conditioned.  Gridding with
random lnG of several norms (the table's spacing and the polynomial's degree follow them), sample
counts that leave ragged groups of 4 and 32, and repetitions.  Tolerance 1e-4 relative L2, the
bound of the float32 GROG paths.
"""
import numpy as np
import pytest
import torch

from oracle import grog as ogrog
from tests.helpers import rand_c, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 2, 7, 8, 15, 31, 32])
def test_calibration(mr, cuda, nc):
    rng = np.random.default_rng(nc)
    Nr, nspk = 4 * nc + 8, 40
    ang = 2 * np.pi * np.arange(nspk) / nspk * 0.618
    k = (np.arange(Nr) - (Nr - 1) / 2) / Nr
    trj = np.stack([np.outer(k, np.cos(ang)), np.outer(k, np.sin(ang))]).astype(np.float32)
    q = np.linalg.qr(rng.standard_normal((nc, nc)) + 1j * rng.standard_normal((nc, nc)))[0]
    gen = [(q * (1j * rng.uniform(-1.5, 1.5, nc))) @ q.conj().T for _ in range(2)]  # commuting, unitary shifts
    data = np.empty((Nr, nspk, nc), dtype=np.complex64)
    for s in range(nspk):
        b = np.cos(ang[s]) * gen[0] + np.sin(ang[s]) * gen[1]
        lam, vec = np.linalg.eig(b)
        d = rng.standard_normal(nc) + 1j * rng.standard_normal(nc)
        for r in range(Nr):  # G of one sample step is exp(b)
            data[r, s] = vec @ (np.exp(lam * r) * np.linalg.solve(vec, d))
    data += (0.01 * rand_c(rng, data.shape)).astype(np.complex64)
    got = [mr.to_host(m) for m in mr.grog_calib(data, trj, Nr)]
    for a, b in zip(got, ogrog.grog_calib(data, trj, Nr)):
        assert rel_l2(a, b) < 1e-4


@pytest.mark.parametrize("nc,norm,ns,nrep", [(1, 1.0, 31, 1), (3, 0.1, 45, 2), (8, 2.0, 64, 1), (9, 6.0, 33, 1), (16, 20.0, 40, 1),
                                             (24, 1.0, 7, 3), (31, 3.0, 50, 1), (32, 5.0, 128, 2)])
def test_gridding(mr, cuda, nc, norm, ns, nrep):
    rng = np.random.default_rng(100 + nc)
    Nr, img, nt = ns, (16, 12), 5
    trj = (rng.random((2, ns, nt)) - 0.5).astype(np.float32)
    lnG = []
    for _ in range(2):
        m = rand_c(rng, (nc, nc))
        m = (m - m.conj().T) / 2 + 0.05 * m  # close to unitary shifts
        lnG.append((m * (norm / np.abs(m).sum(0).max())).astype(np.complex64))
    data = rand_c(rng, (ns, nt, nc, nrep))
    d = mr.to_jl(data, torch.complex64)
    idx = mr.to_host(mr.grog_gridding(d, trj, lnG, Nr, img))
    ref_idx, ref = ogrog.grog_gridding(data, trj, lnG, Nr, img)
    np.testing.assert_array_equal(idx, ref_idx)
    assert rel_l2(mr.to_host(d), ref) < 1e-4
