"""The cuts of the fixed-base sums: rows packed on part of a warp's lanes with
the terms of a column shared by the others, four warps per column, a remainder
of rows with a packing of its own, both projection instances in one group; and
the commitments' lane groups and reduction tree."""
import numpy as np
import pytest

import oracle as O
from conftest import fk20_setup_data

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(engine):
    c = engine.Context(0, 8)
    c.load_xext_fft(1024, engine.to_device(fk20_setup_data(1024)[2]))
    c.load_commit(1024, engine.to_device(fk20_setup_data(1024)[1][:1024]), 8)
    yield c
    c.close()


@pytest.mark.parametrize("rows", [1, 2, 3, 8, 16, 17, 40, 48, 50])
def test_rows_of_every_packing(engine, ctx, rows):
    n, m = 1024, 128
    tau, _, xext = fk20_setup_data(n)
    poly = O.seeded_fr(300 + rows, rows * n).reshape(rows, n, 4)
    d = engine.to_device(poly)
    h, hext = engine.empty((rows, m, 18)), engine.empty((rows, m, 18))
    ctx.poly2h_fft(h, d, rows, n)
    ctx.poly2hext_fft(hext, d, rows, n)
    assert ctx.status() == 0
    got, gx = engine.to_host(h), engine.to_host(hext)
    for r in sorted({0, rows // 2, rows - 1}):
        ref = O.fk20_row(poly[r], xext)
        assert np.array_equal(O.g1_normalize(got[r]), ref["h_fft"]), r
        assert np.array_equal(O.g1_normalize(gx[r]), ref["hext_fft"]), r


@pytest.mark.parametrize("rows,n", [(1, 32), (1, 1024), (5, 96), (33, 1024), (48, 64)])
def test_commitments_of_every_packing(engine, ctx, rows, n):
    tau = O.limbs_to_int(fk20_setup_data(1024)[0])
    poly = O.seeded_fr(900 + rows, rows * n).reshape(rows, n, 4)
    out = engine.empty((rows, 18))
    ctx.commit(out, engine.to_device(poly), rows, n)
    ks = []
    for r in range(rows):
        acc = 0
        for v in reversed(poly[r]):
            acc = (acc * tau + O.limbs_to_int(v)) % O.R
        ks.append(acc)
    exp = O.g1_op("mul", np.repeat(O.g1_generator().reshape(1, 18), rows, 0), O.ints_to_array(ks, 4))
    assert np.array_equal(O.g1_normalize(engine.to_host(out)), O.g1_normalize(exp))


@pytest.mark.parametrize("rows,n", [(296, 32), (297, 32), (1183, 64), (2100, 32), (9000, 32), (18000, 64), (40001, 32)])
def test_many_commitments(engine, ctx, rows, n):
    """The partial sums of a row added by a block, or by 32 down to one lanes;
    several waves of the first pass.  Rows repeat 61 polynomials."""
    tau = O.limbs_to_int(fk20_setup_data(1024)[0])
    poly = O.seeded_fr(77, 61 * n).reshape(61, n, 4)
    ks = []
    for p in poly:
        acc = 0
        for v in reversed(p):
            acc = (acc * tau + O.limbs_to_int(v)) % O.R
        ks.append(acc)
    exp = O.g1_normalize(O.g1_op("mul", np.repeat(O.g1_generator().reshape(1, 18), 61, 0), O.ints_to_array(ks, 4)))
    out, aff = engine.empty((rows, 18)), engine.empty((rows, 18))
    d = engine.to_device(poly).repeat((rows + 60) // 61, 1, 1)[:rows].contiguous()
    ctx.commit(out, d, rows, n)
    engine.call("g1p_op_n", engine.G1_OPS["normalize"], engine._ptr(aff), engine._ptr(out), None, rows, engine._stream())
    got = engine.to_host(aff)
    assert np.array_equal(got, np.tile(exp, ((rows + 60) // 61, 1))[:rows])
