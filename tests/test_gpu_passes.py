"""Batches of more rows of a length than one pass of the pipeline takes (1024):
every output form, contiguous and ragged, equal to the same polynomials in a
small call, which other tests compare with the oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import fk20_setup_data

pytestmark = pytest.mark.gpu

DISTINCT = 24


def words(t):  # indexing wants a signed type
    import torch
    return t.view(torch.int64)


@pytest.fixture(scope="module")
def ctx(engine):
    c = engine.Context(0, 8)
    for n in (1024, 2048):
        c.load_xext_fft(n, engine.to_device(fk20_setup_data(n)[2]))
    yield c
    c.close()


def forms(engine, ctx, poly, rows, n):
    import torch
    m = n // 8
    h, hext = words(engine.empty((rows, m, 18))), words(engine.empty((rows, m, 18)))
    proofs = torch.empty((rows, m, 48), dtype=torch.uint8, device="cuda")
    ctx.poly2h_fft(h, poly, rows, n)
    ctx.poly2hext_fft(hext, poly, rows, n)
    ctx.poly2proofs(proofs, poly, rows, n)
    return h, hext, proofs


@pytest.mark.parametrize("n,rows", [(1024, 1025), (1024, 2048 + 19), (2048, 1040)])
def test_rows_in_passes(engine, ctx, n, rows):
    import torch
    poly = words(engine.to_device(O.seeded_fr(500 + n, DISTINCT * n).reshape(DISTINCT, n, 4)))
    index = torch.arange(rows, device="cuda") % DISTINCT
    small, large = forms(engine, ctx, poly, DISTINCT, n), forms(engine, ctx, poly[index].contiguous(), rows, n)
    assert ctx.status() == 0
    for a, b in zip(small, large):
        assert torch.equal(a[index], b)


@pytest.mark.parametrize("form", ["batch", "proofs", "plan"])
def test_ragged_rows_in_passes(engine, ctx, form):
    """1,100 of one length and 40 of another, in an order and at offsets of their own."""
    import torch
    rng = np.random.default_rng(4)
    ns = [int(v) for v in rng.permutation([1024] * 1100 + [2048] * 40)]
    size = 48 if form == "proofs" else 18
    base = {n: words(engine.to_device(O.seeded_fr(600 + n, DISTINCT * n).reshape(DISTINCT, n, 4))) for n in (1024, 2048)}
    small = {n: forms(engine, ctx, base[n], DISTINCT, n)[2 if form == "proofs" else 0] for n in base}
    place = rng.permutation(len(ns))  # where each request's polynomial and proofs lie
    poly_off, out_off, at = [0] * len(ns), [0] * len(ns), 0
    for j in place:
        poly_off[j], out_off[j] = at, at // 8
        at += ns[j]
    polys = torch.cat([base[ns[j]][j % DISTINCT] for j in place])
    out = torch.zeros((at // 8, size), dtype=small[1024].dtype, device="cuda")
    if form == "plan":
        p = engine.Plan(ctx, out, polys, ns, poly_off, out_off)
        p.launch()
        torch.cuda.synchronize()
        p.close()
    else:
        (ctx.batch if form == "batch" else ctx.batch_proofs)(out, polys, ns, poly_off, out_off)
    assert ctx.status() == 0
    expected = torch.cat([small[ns[j]][j % DISTINCT] for j in place])
    assert torch.equal(out, expected)


@pytest.mark.parametrize("call,rows", [("fk20_hext_fft2h_fft", 1041), ("g1p_fft", 1027), ("g1p_ift", 1057)])
def test_points_in_passes(engine, ctx, call, rows):
    import torch
    k = DISTINCT * 512
    gen = engine.to_device(np.repeat(O.g1_generator().reshape(1, 18), k, 0))
    src, small = words(engine.empty((DISTINCT, 512, 18))), words(engine.empty((DISTINCT, 512, 18)))
    scal = engine.to_device(O.seeded_fr(9, k))
    engine.call("g1p_op_n", engine.G1_OPS["mul"], engine._ptr(src), engine._ptr(gen), engine._ptr(scal), k, engine._stream())
    index = torch.arange(rows, device="cuda") % DISTINCT
    large = src[index].contiguous()
    engine.call(call, engine._ptr(small), engine._ptr(src), DISTINCT, engine._stream())
    engine.call(call, engine._ptr(large), engine._ptr(large), rows, engine._stream())
    assert torch.equal(small[index], large)


@pytest.mark.parametrize("shift", [-3, 3])
def test_points_over_a_shifted_input(engine, ctx, shift):
    """Output and input share a buffer, the output some rows before or behind."""
    import torch
    rows, k = 1060, DISTINCT * 512
    gen = engine.to_device(np.repeat(O.g1_generator().reshape(1, 18), k, 0))
    src, small = words(engine.empty((DISTINCT, 512, 18))), words(engine.empty((DISTINCT, 512, 18)))
    scal = engine.to_device(O.seeded_fr(10, k))
    engine.call("g1p_op_n", engine.G1_OPS["mul"], engine._ptr(src), engine._ptr(gen), engine._ptr(scal), k, engine._stream())
    engine.call("g1p_fft", engine._ptr(small), engine._ptr(src), DISTINCT, engine._stream())
    index = torch.arange(rows, device="cuda") % DISTINCT
    buf = torch.zeros((rows + 3, 512, 18), dtype=torch.int64, device="cuda")
    a, b = buf[max(0, -shift):][:rows], buf[max(0, shift):][:rows]
    a.copy_(src[index])
    engine.call("g1p_fft", engine._ptr(b), engine._ptr(a), rows, engine._stream())
    assert torch.equal(small[index], b)


@pytest.mark.parametrize("shape", ["rows behind", "rows at the start", "ragged"])
def test_proofs_over_their_coefficients(engine, ctx, shape):
    """1,060 rows' proofs written into the buffer of the coefficients."""
    import torch
    n, rows, m = 1024, 1060, 128
    base = words(engine.to_device(O.seeded_fr(777, DISTINCT * n).reshape(DISTINCT, n, 4)))
    small = forms(engine, ctx, base, DISTINCT, n)[0]
    index = torch.arange(rows, device="cuda") % DISTINCT
    buf = base[index].reshape(-1).clone()
    at = {"rows behind": buf.numel() - rows * m * 18, "rows at the start": 0, "ragged": 18 * m}[shape]
    at -= at % 18
    out = buf[at:at + rows * m * 18].reshape(rows, m, 18)
    if shape == "ragged":
        order = list(range(rows))[::-1]  # of coefficients and proofs alike
        ctx.batch(buf, buf, [n] * rows, [r * n for r in order], [at // 18 + r * m for r in order])
    else:
        ctx.poly2h_fft(out, buf, rows, n)
    assert ctx.status() == 0
    assert torch.equal(out, small[index])
