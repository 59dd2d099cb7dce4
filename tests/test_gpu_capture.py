"""Transforms of points inside a stream capture, their buffers grown and their
plans uploaded during it, replayed on new inputs; and beside a pipeline call of
the same default context on another stream."""
import numpy as np
import pytest

import oracle as O
from conftest import fk20_setup_data

pytestmark = pytest.mark.gpu


def points(seed, count):
    return O.g1_op("mul", np.repeat(O.g1_generator().reshape(1, 18), count, 0), O.seeded_fr(seed, count))


@pytest.mark.parametrize("log_m,inverse", [(3, 1), (6, 0)])
def test_transform_captured_and_replayed(engine, log_m, inverse):
    import torch
    m, count = 1 << log_m, 3
    x, y = points(5, count * m).reshape(count, m, 18), points(6, count * m).reshape(count, m, 18)
    src, out = engine.to_device(x), engine.empty(x.shape)
    # the default context exists before the capture; this size's plan and buffers do not
    engine.call("g1p_fft_n", engine._ptr(out), engine._ptr(src), 1, 1, 0, engine._stream())
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        engine.call("g1p_fft_n", engine._ptr(out), engine._ptr(src), log_m, count, inverse, engine._stream())
    for v in (x, y):
        src.copy_(engine.to_device(v))
        g.replay()
        torch.cuda.synchronize()
        got = O.g1_normalize(engine.to_host(out).reshape(-1, 18)).reshape(v.shape)
        assert np.array_equal(got, O.g1_fft(v, inverse=bool(inverse)))


def test_transform_beside_a_pipeline_call(engine):
    import torch
    rows, n = 40, 4096
    xext = engine.to_device(fk20_setup_data(n)[2])
    poly = engine.to_device(O.seeded_fr(8, rows * n).reshape(rows, n, 4))
    src = engine.to_device(points(9, 512).reshape(1, 512, 18))
    ref, out = engine.empty((1, 512, 18)), engine.empty((1, 512, 18))
    h0, h1 = engine.empty((rows, 512, 18)), engine.empty((rows, 512, 18))
    P = engine._ptr
    engine.call("fk20_poly2h_fft", P(h0), P(poly), P(xext), rows)
    torch.cuda.synchronize()
    engine.call("g1p_fft", P(ref), P(src), 1, engine._stream())
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(3):
        engine.call("fk20_poly2h_fft", P(h1), P(poly), P(xext), rows)
        with torch.cuda.stream(side):
            engine.call("g1p_fft", P(out), P(src), 1, engine._stream())
        torch.cuda.synchronize()
        assert torch.equal(h1, h0) and torch.equal(out, ref)
