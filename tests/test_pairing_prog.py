"""The pairing's rounds (csrc/gen_pairing_prog.py): the committed tables are the
generator's output, and each program, run lane by lane on integers as the
kernel runs it, computes its step -- Miller doubling and addition with both
lines against the affine restatement, products, cyclotomic squares and the
inverse in Fp12."""
import os
import random
import subprocess
import sys

import pytest

import pairing_py as PP
from conftest import ROOT

CSRC = os.path.join(ROOT, "fk20-cuda_b200", "csrc")
sys.path.insert(0, CSRC)
import gen_pairing_prog as G  # noqa: E402

P = PP.P


def test_tables_are_the_generators_output():
    out = subprocess.run([sys.executable, "gen_pairing_prog.py"], cwd=CSRC, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    with open(os.path.join(CSRC, "pairing_prog.inc")) as f:
        assert out.stdout == f.read()


@pytest.fixture(scope="module")
def progs():
    p, slots = G.build()
    assert slots <= 255
    return p, slots


def run(progs, st, name):
    for kind, lanes in progs[0][name]:
        assert len(lanes) <= 32 and len({d for d, _ in lanes}) == len(lanes)
        new = []
        for d, refs in lanes:  # every lane reads before any writes
            if kind == "prod":
                new.append((d, sum(st[s] * c for s, c in refs[:2]) * sum(st[s] * c for s, c in refs[2:]) % P))
            else:  # the kernel's column sums hold 2^7 p
                assert sum(abs(c) for _, c in refs) <= 120
                new.append((d, sum(st[s] * c for s, c in refs) % P))
        for d, v in new:
            st[d] = v


def state(progs, seed):
    rng = random.Random(seed)
    st = [rng.randrange(P) for _ in range(progs[1])]
    st[G.ZERO], st[G.ONE] = 0, 1
    return st


def f12(st, at):
    return tuple((st[at + 2 * k], st[at + 2 * k + 1]) for k in range(6))


def put(st, at, vals):
    for k, v in enumerate(vals):
        st[at + 2 * k], st[at + 2 * k + 1] = v


def test_products_and_inverse(progs):
    st = state(progs, 1)
    a, b = f12(st, G.ACC), f12(st, G.B)
    run(progs, st, "MUL")
    assert f12(st, G.ACC) == PP.f12mul(a, b) and f12(st, G.B) == b
    a = f12(st, G.ACC)
    run(progs, st, "INV1")
    st[G.X + 8] = pow(st[G.X + 8], P - 2, P)
    run(progs, st, "INV2")
    assert PP.f12mul(a, f12(st, G.B)) == PP.ONE12


def test_cyclotomic_square(progs):
    st = state(progs, 2)
    a = PP.f12pow(f12(st, G.ACC), (P ** 6 - 1) * (P ** 2 + 1))
    put(st, G.ACC, a)
    run(progs, st, "CYC")
    assert f12(st, G.ACC) == PP.f12mul(a, a)


def proportional(a, b):
    """a = c b for some c in Fp2"""
    k = next(i for i in range(6) if b[i] != (0, 0))
    c = PP.f2mul(a[k], PP.f2inv(b[k]))
    return all(PP.f2mul(c, b[i]) == a[i] for i in range(6))


@pytest.mark.parametrize("add", [False, True])
def test_miller_steps(progs, add):
    """f and T after a step, up to Fp2 factors (of the lines) and Z"""
    st = state(progs, 3)
    rng = random.Random(4)
    f = f12(st, G.ACC)
    g2 = PP.g2_generator()
    exp = f if add else PP.f12mul(f, f)
    pts = []
    for j in range(2):
        q, t = PP.g2mul(rng.randrange(PP.R), g2), PP.g2mul(rng.randrange(PP.R), g2)
        z = (rng.randrange(P), rng.randrange(P))
        put(st, G.T + 6 * j, (PP.f2mul(t[0], z), PP.f2mul(t[1], z), z))
        put(st, G.Q + 4 * j, q)
        xp, yp = rng.randrange(P), rng.randrange(P)
        st[G.PT + 2 * j], st[G.PT + 2 * j + 1] = xp, yp
        if add:
            lam = PP.f2mul(PP.f2sub(q[1], t[1]), PP.f2inv(PP.f2sub(q[0], t[0])))
            pts.append(PP.g2add(t, q))
        else:
            lam = PP.f2mul(PP.f2mul((3, 0), PP.f2mul(t[0], t[0])), PP.f2inv(PP.f2add(t[1], t[1])))
            pts.append(PP.g2add(t, t))
        exp = PP.f12mul(exp, PP._line(lam, t, xp, yp))
    run(progs, st, "ADD" if add else "DBL")
    assert proportional(f12(st, G.ACC), exp)
    for j in range(2):
        x, y, z = ((st[G.T + 6 * j + 2 * k], st[G.T + 6 * j + 2 * k + 1]) for k in range(3))
        zi = PP.f2inv(z)
        assert (PP.f2mul(x, zi), PP.f2mul(y, zi)) == pts[j]


def test_generator_keeps_the_constant_term_of_every_line():
    """a pair with a point at infinity runs with P = (0, 0) and Q the generator:
    its lines are their constant terms, none of them zero"""
    t = q = PP.g2_generator()
    for bit in bin(PP.Z_ABS)[3:]:
        lam = PP.f2mul(PP.f2mul((3, 0), PP.f2mul(t[0], t[0])), PP.f2inv(PP.f2add(t[1], t[1])))
        assert PP.f2sub(PP.f2mul(lam, t[0]), t[1]) != (0, 0)
        t = PP.g2add(t, t)
        if bit == "1":
            lam = PP.f2mul(PP.f2sub(q[1], t[1]), PP.f2inv(PP.f2sub(q[0], t[0])))
            assert PP.f2sub(PP.f2mul(lam, t[0]), t[1]) != (0, 0)
            t = PP.g2add(t, q)


def g1_jac(st, at):
    x, y, z = st[at:at + 3]
    if z == 0:
        return None
    zi = pow(z, -1, P)
    return x * zi % P, y * zi % P


def test_g1_sums(progs):
    """Both sums of a doubling and an addition round sequence, with equal points,
    opposite points and infinity among the operands (homogeneous coordinates)."""
    rng = random.Random(6)
    gen = (0x17F1D3A73197D7942695638C4FA9AC0FC3688C4F9774B905A14E3A3F171BAC586C55E83FF97A1AEFFB3AF00ADB22C6BB,
           0x08B3F481E3AAA0F1A09E30ED741D8AE4FCF5E095D5D00AF600DB18CB2C04B3EDD03CC744A2888AE40CAA232946C5E7E1)
    a, b = PP.g1mul(rng.randrange(PP.R), gen), PP.g1mul(rng.randrange(PP.R), gen)

    def put3(st, at, p):
        z = rng.randrange(1, P)
        st[at:at + 3] = (0, z, 0) if p is None else (p[0] * z % P, p[1] * z % P, z)

    cases = [(a, b), (a, a), (a, PP.g1neg(a)), (None, b), (a, None), (None, None)]
    for x, y in zip(cases, cases[1:] + cases[:1]):
        st = state(progs, 7)
        for j, (p, q) in enumerate((x, y)):
            put3(st, G.VA + 3 * j, p)
            put3(st, G.VQ + 3 * j, q)
        run(progs, st, "VADD")
        for j, (p, q) in enumerate((x, y)):
            assert g1_jac(st, G.VA + 3 * j) == PP.g1add(p, q)
        run(progs, st, "VDBL")
        for j, (p, q) in enumerate((x, y)):
            s = PP.g1add(p, q)
            assert g1_jac(st, G.VA + 3 * j) == PP.g1add(s, s)
