"""The plans of additions and one layer of fixed-scalar products
(csrc/proj_plan.cuh), hext_fft -> h_fft and whole transforms, replayed on Fr
values against the transforms they replace; the dependencies and slot reuse the kernel relies on;
the launch order; the shared P + Q / P - Q formulas."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle as O
from conftest import ROOT
from test_host_emulation import HOST, LAMBDA, P, program_partial_sums

R = O.R
LIN, SHL, MUL, OUT, NONE = 0, 1, 2, 3, 0xFFFF


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("emul") / "libemul.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fk20-cuda_b200", "csrc"), os.path.join(HOST, "emul.cpp"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def ints(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def load_plan(emul, log_m, half):
    head = np.zeros(5, np.int32)
    emul.emul_proj_plan(log_m, half, ints(head), None, None, None, None)
    slots, nt, muls, nout, nlev = (int(v) for v in head)
    tasks = np.zeros((nt, 16), np.int32)
    sc = np.zeros((muls, 4), np.uint64)
    out = np.zeros(nout, np.int32)
    lev = np.zeros((nlev, 3), np.int32)
    emul.emul_proj_plan(log_m, half, ints(head), ints(tasks), P(sc), ints(out), ints(lev))
    return slots, tasks.tolist(), [O.limbs_to_int(v) for v in sc], out.tolist(), lev.tolist()


def unordered_overwrites(tasks):
    """(task, slot, reader) for every write over a value that a reader may not have
    read yet.  What a task waits for: the writers of the versions that it asks for
    and, in the last phase, all products of its group; so also all that these wait for."""
    wrote, readers, above, produced, bad = {}, {}, [], set(), []
    for k, (op, sh, ph, neg, d0, d1, a, b, b2, va, vb, vb2, w0, w1, phase, prog) in enumerate(tasks):
        anc = set(produced) if phase == 2 else set()
        for s, v in ((a, va), (b, vb), (b2, vb2)):
            # an output's b and b2 are the other instance's, written at the same place there
            if s != NONE and v:
                anc |= above[wrote[s, v]] | {wrote[s, v]}
        above.append(anc)
        if op == MUL:
            produced |= anc | {k}
        for s in (a,) if op in (OUT, SHL, MUL) else (a, b):  # b2 is waited for, not read
            readers.setdefault(s, []).append(k)
        for d, w in ((d0, w0), (d1, w1)):
            if d != NONE:
                bad += [(k, d, r) for r in readers.get(d, []) if r != k and r not in anc]
                wrote[d, w], readers[d] = k, []
    return bad


def test_an_overwrite_that_nothing_orders_is_seen():
    """After the products a task writes over slot 0, which a doubling that feeds no
    product reads: seen, unless the task waits for the doubling's result; the sum
    that reads it too is above the product."""
    def tasks(b2, vb2):
        return [(SHL, 3, 0, 0, 2, NONE, 0, NONE, NONE, 0, 0, 0, 1, 0, 0, 0),
                (LIN, 0, 0, 0, 3, 4, 0, 1, NONE, 0, 0, 0, 1, 1, 0, 0),
                (MUL, 0, 0, 0, 5, NONE, 3, NONE, NONE, 1, 0, 0, 1, 0, 1, 0),
                (LIN, 0, 0, 0, 0, NONE, 5, 4, b2, 1, 1, vb2, 1, 0, 2, 0)]
    assert unordered_overwrites(tasks(NONE, 0)) == [(3, 0, 0)]
    assert unordered_overwrites(tasks(2, 1)) == []


PLANS = [(7, 0), (8, 0), (9, 0), (9, 1)] + [(l, k) for l in range(1, 10) for k in (2, 3)]


@pytest.mark.parametrize("log_m,kind", PLANS)
def test_plan_replayed_on_scalars(emul, log_m, kind):
    """In task order every read finds the version it asks for; the outputs are
    FFT(upper half zeroed(IFFT)) of the inputs (kinds 0 and 1, two instances a
    row) or their transform (2) or inverse transform (3); and no slot is written over
    while a reader of the old value may still run."""
    m, H = 1 << log_m, 1 << (log_m - 1)
    slots, tasks, scalars, out, levels = load_plan(emul, log_m, kind)
    rng = np.random.default_rng(log_m)
    x = [int(v) for v in rng.integers(0, 2**62, m)]
    w = O.root_of_unity(m)
    inv_m = pow(m, R - 2, R)
    val = [[0] * slots, [0] * slots]
    s_, i_ = ctypes.c_int(), ctypes.c_int()
    seen = set()
    for c in range(m):
        if kind > 1:
            val[0][c] = x[c]
            continue
        emul.emul_proj_in(c, log_m, ctypes.byref(s_), ctypes.byref(i_))
        assert 0 <= s_.value < H and (s_.value, i_.value) not in seen
        seen.add((s_.value, i_.value))
        val[i_.value][s_.value] = x[c] if kind else x[c] * inv_m % R
    ver = [0] * slots
    assert unordered_overwrites(tasks) == []
    wrote = {}
    above = []
    cross = set()
    phi = [1, LAMBDA, LAMBDA * LAMBDA % R]
    phase_before = 0
    last = [0] * slots  # final version of each slot
    for t in tasks:
        for d, wv in ((t[4], t[12]), (t[5], t[13])):
            if d != NONE:
                last[d] = max(last[d], wv)
    for k, (op, sh, ph, neg, d0, d1, a, b, b2, va, vb, vb2, w0, w1, phase, prog) in enumerate(tasks):
        assert phase >= phase_before and (op == MUL) == (phase == 1)
        phase_before = phase
        deps = set()
        reads = [(a, va)] + ([(b, vb)] if b != NONE else []) + ([(b2, vb2)] if b2 != NONE else [])
        for s, v in reads:
            assert ver[s] == v or (op != OUT and s == b2 and ver[s] >= v), k
            if v:
                deps.add(wrote[s, v])
                assert tasks[wrote[s, v]][14] <= phase
        anc = set()
        for d in deps:
            anc |= above[d] | {d}
        above.append(anc)
        if op == OUT:  # b, b2: the other instance's
            cross |= {b, b2}
        res = []
        for inst in (0, 1):
            A = val[inst][a]
            if op == LIN:
                B = val[inst][b] * phi[ph] % R * (1 << sh) % R * (-1 if neg else 1)
                res.append(((A + B) % R, (A - B) % R))
            elif op == SHL:
                res.append((A * (1 << sh) % R,))
            elif op == MUL:
                res.append((A * scalars[prog] % R,))
            else:
                res.append(((A * phi[ph] * (-1 if neg else 1) + val[1 - inst][b2 if inst else b]) % R,))
        for n, (d, wv) in enumerate([(d0, w0)] + ([(d1, w1)] if d1 != NONE else [])):
            assert not any(e & 0xFFFF == d and ver[d] == last[d] for e in out)  # outputs stay
            assert d not in cross and wv == ver[d] + 1 and wv < 256
            ver[d], wrote[d, wv] = wv, k
            for inst in (0, 1):
                val[inst][d] = res[inst][n]
    for first, count, phase in levels:  # no dependency inside a level
        for k in range(first, first + count):
            assert not any(first <= d < first + count for d in above[k]) and tasks[k][14] == phase
    wi = pow(w, R - 2, R)
    pw, pi = [1], [1]
    for _ in range(m - 1):
        pw.append(pw[-1] * w % R)
        pi.append(pi[-1] * wi % R)
    h = [sum(x[c] * pi[j * c % m] for c in range(m)) * inv_m % R for j in range(H)] if kind < 2 else []
    for k in range(0, m, 1 if m < 512 else 5):
        if kind < 2:
            got, exp = val[k & 1][out[k >> 1]], sum(h[j] * pw[j * k % m] for j in range(H)) % R
        else:
            e = out[k]
            got = val[0][e & 0xFFFF] * phi[e >> 17] * (-1 if (e >> 16) & 1 else 1) % R
            tw, f = (pw, 1) if kind == 2 else (pi, inv_m)
            exp = sum(x[j] * tw[j * k % m] for j in range(m)) * f % R
        assert got == exp, k


@pytest.mark.parametrize("log_m,half", PLANS)
def test_plan_programs_avoid_exceptional_additions(emul, log_m, half):
    """As for the twiddle programs: no partial sum of a product's program meets
    the added point, its negative or infinity."""
    prog = np.zeros(64, np.uint32)
    for k in load_plan(emul, log_m, half)[2]:
        emul.emul_make_program(prog.ctypes.data_as(ctypes.c_void_p), P(O.int_to_limbs(k, 4)))
        if int(prog[0]) & 0x300:
            assert k in (1, R - 1)
            continue
        adds, res = program_partial_sums(prog)
        assert res == k
        for a, q in adds:
            assert a != 0 and a != q and a != R - q


@pytest.mark.parametrize("rows", [[1], [16], [17], [600], [333, 320, 347], [1, 40, 16]])
def test_launch_order(emul, rows):
    """Every (segment, task, group) once, and never before a task it depends on."""
    log_m = [9, 8, 7][:len(rows)] if len(rows) > 1 else [7]
    plans = [load_plan(emul, l, 0) for l in log_m]
    G = [2 * (r // 32) + (r % 32 > 0) + (r % 32 > 16) for r in rows]
    cap = sum(len(p[1]) * g for p, g in zip(plans, G))
    order = np.zeros((cap, 3), np.int32)
    ci = lambda v: (ctypes.c_int * len(v))(*v)
    assert emul.emul_proj_order(len(rows), ci(log_m), ci(rows), ints(order), ctypes.c_long(cap)) == cap
    for k, (p, g) in enumerate(zip(plans, G)):
        sel = order[order[:, 0] == k]
        at = np.full((len(p[1]), g), -1, np.int64)
        at[sel[:, 1], sel[:, 2]] = np.nonzero(order[:, 0] == k)[0]
        assert (at >= 0).all() and len(sel) == len(p[1]) * g
        # task t waits for tasks of lower number of its level's predecessors: levels in order per group,
        # and outputs (they read the other instance's diagonal term) after every first-phase level
        starts = [f for f, _, _ in p[4]] + [len(p[1])]
        for a, b, c in zip(starts, starts[1:], starts[2:]):
            assert (at[a:b].max(axis=0) < at[b:c].min(axis=0)).all()
        first = [f for f, _, ph in p[4] if ph == 2][0]
        assert at[:first].max() < at[first:].min()


def test_addsub_formulas(emul):
    g = O.g1_generator().reshape(1, 18)
    ks = O.seeded_fr(3, 24)
    p = O.g1_op("mul", np.repeat(g, 24, 0), ks)
    q = O.g1_op("mul", np.repeat(g, 24, 0), O.seeded_fr(4, 24))
    inf = np.zeros(18, np.uint64)
    inf[6] = 1
    q[0] = p[0]
    q[1] = O.g1_op("neg", p[1:2])[0]
    q[2] = inf
    p[3] = inf
    p[4] = q[4] = inf
    s, d = np.zeros_like(p), np.zeros_like(p)
    emul.emul_g1_addsub(P(s), P(d), P(p), P(q), 24)
    assert np.array_equal(O.g1_normalize(s), O.g1_normalize(O.g1_op("add", p, q)))
    assert np.array_equal(O.g1_normalize(d), O.g1_normalize(O.g1_op("add", p, O.g1_op("neg", q))))
