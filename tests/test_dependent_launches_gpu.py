"""Passes that are launched before the pass ahead of them has ended (grids of 304 to 4096 blocks): the
same bits as plain launches (an apply captured in a caller's graph) with a caller's kernels writing
x right before and reading y, overwriting x and y right after, and with two operators in flight on
two streams."""
import numpy as np
import pytest
import torch

from tests.helpers import rand_c

pytestmark = pytest.mark.gpu


def _operator(mr, rng, img, K, nc, kind):
    cm = [rand_c(rng, img) for _ in range(nc)]
    if kind == "fft":
        return mr.FFTNormalOp(rand_c(rng, (K, K) + img), cmaps=cm)
    cells = np.flatnonzero(rng.random(4 * int(np.prod(img))) < 0.6) + 1
    return mr.NFFTNormalOp(img, rand_c(rng, (K * (K + 1) // 2, cells.size)), cells, cmaps=cm)


def _plain(mr, A, x):
    """One apply as the launches of a graph."""
    y = torch.zeros_like(x)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        A.mul(y, x, stream=s)
    torch.cuda.synchronize()
    y.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.mul(y, x, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert not y.any()
    g.replay()
    torch.cuda.synchronize()
    return y.clone()


CASES = [((180, 150), 3, 12, "nfft"), ((256, 256), 6, 32, "fft"), ((225, 150), 2, 6, "fft"), ((64, 64), 4, 32, "nfft")]


@pytest.mark.parametrize("img,K,nc,kind", CASES)
def test_neighbours(mr, cuda, img, K, nc, kind):
    rng = np.random.default_rng(101)
    A = _operator(mr, rng, img, K, nc, kind)
    inputs = [mr.to_jl(rand_c(rng, img + (K,)), torch.complex64) for _ in range(3)]
    refs = [_plain(mr, A, x) for x in inputs]
    x, y = torch.zeros_like(inputs[0]), torch.zeros_like(inputs[0])
    out = []
    for i in range(30):
        x.copy_(inputs[i % 3])
        A.mul(y, x)
        x.fill_(float("nan"))
        out.append(y * 2)
        y.fill_(float("nan"))
    for i, z in enumerate(out):
        assert torch.equal(z, refs[i % 3] * 2)


def test_two_streams(mr, cuda):
    rng = np.random.default_rng(102)
    ops = [_operator(mr, rng, *c) for c in CASES[:2]]
    xs = [mr.to_jl(rand_c(rng, c[0] + (c[1],)), torch.complex64) for c in CASES[:2]]
    refs = [_plain(mr, A, x) for A, x in zip(ops, xs)]
    ys = [[torch.zeros_like(x) for _ in range(40)] for x in xs]
    streams = [torch.cuda.Stream() for _ in ops]
    torch.cuda.synchronize()
    for i in range(40):
        for A, x, y, s in zip(ops, xs, ys, streams):
            A.mul(y[i], x, stream=s)
    torch.cuda.synchronize()
    for y, ref in zip(ys, refs):
        assert all(torch.equal(v, ref) for v in y)
