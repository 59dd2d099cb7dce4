"""Pairing checks on both sides of the line between the two kernels (a warp per
check up to 10,240, a thread per check beyond): true and false equations and
points at infinity on either side, by known scalars."""
import numpy as np
import pytest

import oracle as O
import pairing_py as PP

pytestmark = pytest.mark.gpu


def g2_rows(pts):
    out = np.zeros((len(pts), 36), np.uint64)
    for i, q in enumerate(pts):
        if q is None:
            out[i, 12] = 1
            continue
        for k, v in enumerate((q[0][0], q[0][1], q[1][0], q[1][1], 1, 0)):
            out[i, 6 * k:6 * k + 6] = O.int_to_limbs(v, 6)
    return out


@pytest.mark.parametrize("count", [1, 2, 3, 37, 10240, 10241])
def test_checks_by_known_scalars(engine, count):
    import torch
    ks = [O.limbs_to_int(v) for v in O.seeded_fr(77, 8)]
    # (a, b, c, d): e([a]G1, [b]G2) == e([c]G1, [d]G2) exactly when ab = cd
    rows = [(ks[0], ks[1], ks[0] * ks[1] % O.R, 1), (ks[2], ks[3], (ks[2] * ks[3] + 1) % O.R, 1), (0, ks[1], 0, ks[2]),
            (0, ks[1], 5, ks[2]), (ks[4], 0, ks[5], 0), (ks[4], 0, 0, ks[6]), (ks[4], ks[5], ks[5], ks[4]),
            (ks[4], ks[5], ks[4], ks[6])]
    want = [int(a * b % O.R == c * d % O.R) for a, b, c, d in rows]
    assert want == [1, 0, 1, 0, 1, 1, 1, 0]
    g1 = O.g1_generator().reshape(1, 18)
    g2 = PP.g2_generator()
    mul1 = lambda v: O.g1_op("mul", np.repeat(g1, len(v), 0), O.ints_to_array(v, 4))
    A, C = mul1([r[0] for r in rows]), mul1([r[2] for r in rows])
    Bq, D = (g2_rows([PP.g2mul(r[k], g2) if r[k] else None for r in rows]) for k in (1, 3))
    idx = np.arange(count) % len(rows)
    dev = [engine.to_device(np.ascontiguousarray(v[idx])) for v in (A, Bq, C, D)]
    ok = torch.full((count,), 7, dtype=torch.uint8, device="cuda")
    engine.call("fk20_pairing_check_n", engine._ptr(ok), *[engine._ptr(v) for v in dev], count, engine._stream())
    assert ok.cpu().numpy().tolist() == [want[i] for i in idx]


@pytest.mark.parametrize("count", [5, 2048, 2049])
def test_check_proof_multi_on_both_point_kernels(engine, count):
    """check_proof_multi with its points a warp each and two lanes each, checks of
    every verdict with a zero coset shift, an infinite proof and an infinite
    commitment among them (scalars known: C = [c], proof = [q], I from ys)."""
    import torch
    l, R = 4, O.R
    t = 1234567
    rng = np.random.default_rng(12)
    word = lambda: int.from_bytes(rng.bytes(32), "little") % R
    w = O.root_of_unity(l)
    rows = []
    for kind in range(6):
        x, r = (0 if kind == 3 else word()), [word() for _ in range(l)]
        rt = sum(v * pow(t, k, R) for k, v in enumerate(r)) % R
        d = (pow(t, l, R) - pow(x, l, R)) % R
        c = 0 if kind == 4 else rt if kind == 2 else word()  # kind 2: quotient 0
        q = (c - rt) * pow(d, -1, R) % R
        if kind == 3:  # every value of a coset at 0 is r_0
            r = [r[0]] + [0] * (l - 1)
            rt, q = r[0], (c - r[0]) * pow(d, -1, R) % R
        ys = [sum(v * pow(x * pow(w, k, R) % R, e, R) for e, v in enumerate(r)) % R for k in range(l)]
        rows.append((c, q, x, ys, 1))
        rows.append((c, q, x, [(ys[0] + 1) % R] + ys[1:], 0))
    idx = np.arange(count) % len(rows)
    g1 = O.g1_generator().reshape(1, 18)
    mul1 = lambda v: O.g1_op("mul", np.repeat(g1, len(v), 0), O.ints_to_array(v, 4))
    c = engine.Context(0, 8)
    c.load_commit(32, engine.to_device(mul1([pow(t, k, R) for k in range(32)])), 8)
    dev = lambda a: engine.to_device(np.ascontiguousarray(a[idx]))
    C, Q = dev(mul1([r[0] for r in rows])), dev(mul1([r[1] for r in rows]))
    X = dev(O.ints_to_array([r[2] for r in rows], 4))
    Y = dev(np.stack([O.ints_to_array(r[3], 4) for r in rows]))
    s2 = engine.to_device(g2_rows([PP.g2mul(pow(t, k, R), PP.g2_generator()) for k in range(l + 1)]))
    ok = torch.full((count,), 7, dtype=torch.uint8, device="cuda")
    c.check_proof_multi(ok, C, Q, X, Y, l, s2, count)
    got = ok.cpu().numpy().tolist()
    c.close()
    # at x = 0 the interpolation keeps coefficient 0 only, as before: ys[0] alone moves the mean
    assert got == [rows[i][4] for i in idx]


@pytest.mark.parametrize("count", [8192, 8193])
def test_pairing_values_on_both_sides_of_their_line(engine, count):
    """The same words from a warp and from a thread a pairing, infinities and a
    point off the curve among the inputs."""
    g1, g2 = O.g1_generator().reshape(1, 18), PP.g2_generator()
    a = O.g1_op("mul", np.repeat(g1, 6, 0), O.ints_to_array([3, 5, 0, 7, O.R - 1, 11], 4))
    b = g2_rows([PP.g2mul(k, g2) if k else None for k in (1, 9, 4, 0, 2, 6)])
    b[5, :12] = b[1, 12:24]  # no point of the twist
    idx = np.arange(count) % 6
    few, many = engine.empty((6, 72)), engine.empty((count, 72))
    d = [engine.to_device(np.ascontiguousarray(v)) for v in (a, b, a[idx], b[idx])]
    engine.call("fk20_pairing_n", engine._ptr(few), engine._ptr(d[0]), engine._ptr(d[1]), 6, engine._stream())
    engine.call("fk20_pairing_n", engine._ptr(many), engine._ptr(d[2]), engine._ptr(d[3]), count, engine._stream())
    ref = engine.to_host(few)
    assert np.array_equal(engine.to_host(many), ref[idx])
    one = np.zeros(72, np.uint64)
    one[0] = 1
    assert [bool(np.array_equal(v, one)) for v in ref] == [False, False, True, True, False, False]
