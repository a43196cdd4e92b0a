"""The server's estimate of a request covers the backprojection's grids, whose accumulators are padded to
the lanes of the spreading kernel."""
import importlib

import pytest


@pytest.fixture(scope="module")
def sv(mr):
    return importlib.import_module(mr.__name__ + ".serving")


@pytest.mark.parametrize("parts,padded", [(1, 8), (2, 8), (8, 8), (10, 16), (18, 32), (32, 32), (40, 48), (72, 80), (96, 96), (200, 224)])
def test_padding(sv, parts, padded):
    assert sv.spread_parts(parts) == padded


@pytest.mark.parametrize("img,K,nc", [((192, 192), 1, 1), ((384, 384), 1, 4), ((256, 256), 3, 3), ((384, 384), 6, 32)])
def test_estimate(sv, img, K, nc):
    G = 4 * img[0] * img[1]
    cb = min(nc, max(1, (2 << 30) // (8 * K * G)))
    assert sv.request_bytes(img, K, nc) > 8 * G * (K * cb + sv.spread_parts(2 * K * cb))
