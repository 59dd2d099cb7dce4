#!/usr/bin/env python3
"""Writes pairing_prog.inc: the steps of the pairing as rounds of a 32-lane
machine (kernels_pairing.cu runs one check per warp).

The state is a file of Fp values ("slots") in shared memory.  A PROD round
gives every lane one Fp product (+-a0 +-a1)(+-b0 +-b1) of slots, a LIN round
one sum of up to 7 slots with small integer coefficients; lanes read before
any lane writes.  The formulas below are traced on symbolic values: a value is
an integer combination of slots and earlier products, a product's operand of
more than two terms becomes a LIN result first, and the products and sums are
placed into rounds by a list scheduler (longest remaining path first).

Run from this directory: python gen_pairing_prog.py > pairing_prog.inc"""
import sys

LANES, TERMS, PROD_COST, LIN_COST = 32, 7, 15, 8
# fixed slots
ZERO, ONE, DUMP = 0, 1, 2
ACC, B, M, S1, S2 = 4, 16, 28, 40, 52
T, PT, Q = 64, 76, 80  # two points: X, Y, Z (6 each); xP, yP (2 each); xQ, yQ (4 each)
X = 88                 # the inverse's intermediates: t0, t1, t2, n, 1/norm
TMP = 97
VA, VQ, VT = 4, 10, 16  # the G1 machine: two sums, two addends, 2 x 8 multiples (inside the pairing's slots)
Z_ABS = 0xD201000000010000


class Trace:
    """One program: nodes are ('in', slot), ('prod', a, b) or ('lin', terms)."""

    def __init__(self):
        self.nodes = []
        self.memo = {}

    def node(self, key):
        if key not in self.memo:
            self.memo[key] = len(self.nodes)
            self.nodes.append(key)
        return self.memo[key]

    def slot(self, s):
        return LC(self, {self.node(("in", s)): 1})

    def atom(self, v):
        """a value as at most two terms of coefficient +-1"""
        if len(v.t) <= 2 and all(abs(c) == 1 for c in v.t.values()):
            return tuple(sorted(v.t.items()))
        return ((self.lin(v), 1),)

    def lin(self, v):
        """a node that holds the value v"""
        terms = sorted(v.t.items())
        if len(terms) == 1 and terms[0][1] == 1:
            return terms[0][0]
        while len(terms) > TERMS:
            n = min(TERMS, len(terms) - TERMS + 1)
            head, terms = terms[:n], terms[n:]
            terms.append((self.node(("lin", tuple(head))), 1))
        assert sum(abs(c) for _, c in terms) <= 120
        return self.node(("lin", tuple(terms)))

    def mul(self, a, b):
        if not a.t or not b.t:
            return LC(self, {})
        x, y = sorted([self.atom(a), self.atom(b)])
        return LC(self, {self.node(("prod", x, y)): 1})


class LC:
    def __init__(self, tr, t):
        self.tr, self.t = tr, {k: c for k, c in t.items() if c}

    def __add__(self, o):
        t = dict(self.t)
        for k, c in o.t.items():
            t[k] = t.get(k, 0) + c
        return LC(self.tr, t)

    def __rmul__(self, k):
        return LC(self.tr, {i: k * c for i, c in self.t.items()})

    def __sub__(self, o):
        return self + (-1) * o

    def __neg__(self):
        return (-1) * self


class F2:
    def __init__(self, a, b):
        self.a, self.b = a, b

    def __add__(self, o): return F2(self.a + o.a, self.b + o.b)
    def __sub__(self, o): return F2(self.a - o.a, self.b - o.b)
    def __neg__(self): return F2(-self.a, -self.b)
    def __rmul__(self, k): return F2(k * self.a, k * self.b)

    def __mul__(self, o):  # Karatsuba
        m = self.a.tr.mul
        t0, t1, t2 = m(self.a, o.a), m(self.b, o.b), m(self.a + self.b, o.a + o.b)
        return F2(t0 - t1, t2 - t0 - t1)

    def school(self, o):
        m = self.a.tr.mul
        return F2(m(self.a, o.a) - m(self.b, o.b), m(self.a, o.b) + m(self.b, o.a))

    def sqr(self):
        m = self.a.tr.mul
        return F2(m(self.a + self.b, self.a - self.b), 2 * m(self.a, self.b))

    def scale(self, s):  # by an Fp value
        return F2(self.a.tr.mul(self.a, s), self.a.tr.mul(self.b, s))

    def xi(self): return F2(self.a - self.b, self.a + self.b)

    def hold(self):
        """as stored values"""
        tr = self.a.tr
        return F2(LC(tr, {tr.lin(self.a): 1}) if self.a.t else self.a, LC(tr, {tr.lin(self.b): 1}) if self.b.t else self.b)


def f2at(tr, s): return F2(tr.slot(s), tr.slot(s + 1))
def f12at(tr, s): return [f2at(tr, s + 2 * k) for k in range(6)]


def poly_mul(a, b, mul):
    """coefficients of w (None: zero), w^6 = xi"""
    out = [None] * 6
    for i, x in enumerate(a):
        for j, y in enumerate(b):
            if x is None or y is None:
                continue
            p = mul(x, y)
            k = i + j
            if k >= 6:
                k, p = k - 6, p.xi()
            out[k] = p if out[k] is None else out[k] + p
    return out


def poly_sqr(a):
    out = [None] * 6
    for i in range(6):
        for j in range(i, 6):
            p = a[i].sqr() if i == j else 2 * (a[i] * a[j])
            k = i + j
            if k >= 6:
                k, p = k - 6, p.xi()
            out[k] = p if out[k] is None else out[k] + p
    return out


def put(out, s, v):
    out[s], out[s + 1] = v.a, v.b


def put12(out, s, f):
    for k in range(6):
        put(out, s + 2 * k, f[k])


def lines_into(tr, out, f, lines):
    l0, l1 = [[c0, None, c2, c3, None, None] for c0, c2, c3 in lines]
    L = [None if v is None else v.hold() for v in poly_mul(l0, l1, lambda x, y: x * y)]
    put12(out, ACC, poly_mul(f, L, lambda x, y: x * y))


def prog_dbl():
    """f = f^2 l0 l1, T_j = 2 T_j (tangent lines at T_j evaluated at P_j)"""
    tr, out = Trace(), {}
    f = [v.hold() for v in poly_sqr(f12at(tr, ACC))]
    lines = []
    for j in range(2):
        x, y, z = (f2at(tr, T + 6 * j + 2 * k) for k in range(3))
        xp, yp = tr.slot(PT + 2 * j), tr.slot(PT + 2 * j + 1)
        Bq, C, XX, YZ, XY = y.sqr().hold(), z.sqr(), x.sqr(), y * z, x * y
        E = (12 * C.xi()).hold()  # 3 b' Z^2
        H = (2 * YZ).hold()
        lines.append(((Bq - E).hold(), (-(3 * XX)).hold().scale(xp).hold(), H.scale(yp).hold()))
        put(out, T + 6 * j, 2 * (XY.hold() * (Bq - 3 * E).hold()))
        put(out, T + 6 * j + 2, (Bq + 3 * E).hold().sqr() - 12 * E.sqr())
        put(out, T + 6 * j + 4, 4 * (Bq * H))
    lines_into(tr, out, f, lines)
    return tr, out


def prog_add():
    """f = f l0 l1, T_j = T_j + Q_j (chord lines evaluated at P_j)"""
    tr, out = Trace(), {}
    f = f12at(tr, ACC)
    lines = []
    for j in range(2):
        x, y, z = (f2at(tr, T + 6 * j + 2 * k) for k in range(3))
        xp, yp = tr.slot(PT + 2 * j), tr.slot(PT + 2 * j + 1)
        xq, yq = f2at(tr, Q + 4 * j), f2at(tr, Q + 4 * j + 2)
        th, la = (y - yq * z).hold(), (x - xq * z).hold()
        lines.append(((th * xq - la * yq).hold(), (-th).hold().scale(xp).hold(), la.scale(yp).hold()))
        C, D = th.sqr().hold(), la.sqr().hold()
        E, F, G = (la * D).hold(), (z * C).hold(), (x * D).hold()
        Hh = (E + F - 2 * G).hold()
        put(out, T + 6 * j, la * Hh)
        put(out, T + 6 * j + 2, th * (G - Hh).hold() - y * E)
        put(out, T + 6 * j + 4, z * E)
    lines_into(tr, out, f, lines)
    return tr, out


def prog_mul():
    """ACC = ACC B"""
    tr, out = Trace(), {}
    put12(out, ACC, poly_mul(f12at(tr, ACC), f12at(tr, B), lambda x, y: x * y))
    return tr, out


def prog_cyc():
    """ACC = ACC^2 in the cyclotomic subgroup (Granger and Scott)"""
    tr, out = Trace(), {}
    g = f12at(tr, ACC)

    def f4(x0, x1):  # (x0^2 + xi x1^2, 2 x0 x1)
        return x0.sqr() + x1.sqr().xi(), 2 * x0.school(x1)
    A, Bq, C = f4(g[0], g[3]), f4(g[1], g[4]), f4(g[2], g[5])
    put(out, ACC + 0, 3 * A[0] - 2 * g[0])
    put(out, ACC + 6, 3 * A[1] + 2 * g[3])
    put(out, ACC + 2, 3 * C[1].xi() + 2 * g[1])
    put(out, ACC + 8, 3 * C[0] - 2 * g[4])
    put(out, ACC + 4, 3 * Bq[0] - 2 * g[2])
    put(out, ACC + 10, 3 * Bq[1] + 2 * g[5])
    return tr, out


def f6mul(a, b):  # coefficients of v, v^3 = xi
    out = [None] * 3
    for i in range(3):
        for j in range(3):
            p, k = a[i] * b[j], i + j
            if k >= 3:
                k, p = k - 3, p.xi()
            out[k] = p if out[k] is None else out[k] + p
    return out


def prog_inv1():
    """X: t0, t1, t2, n and the norm whose inverse finishes ACC^-1"""
    tr, out = Trace(), {}
    f = f12at(tr, ACC)
    a0, a1 = [f[0], f[2], f[4]], [f[1], f[3], f[5]]
    q, r = f6mul(a0, a0), f6mul(a1, a1)
    s = [(q[0] - r[2].xi()).hold(), (q[1] - r[0]).hold(), (q[2] - r[1]).hold()]  # a0^2 - v a1^2
    t0 = (s[0].sqr() - (s[1] * s[2]).xi()).hold()
    t1 = (s[2].sqr().xi() - s[0] * s[1]).hold()
    t2 = (s[1].sqr() - s[0] * s[2]).hold()
    n = (s[0] * t0 + (s[2] * t1 + s[1] * t2).xi()).hold()
    for k, v in enumerate((t0, t1, t2, n)):
        put(out, X + 2 * k, v)
    out[X + 8] = tr.mul(n.a, n.a) + tr.mul(n.b, n.b)
    return tr, out


def prog_inv2():
    """B = ACC^-1 from X"""
    tr, out = Trace(), {}
    f = f12at(tr, ACC)
    t = [f2at(tr, X + 2 * k) for k in range(3)]
    n, ni = f2at(tr, X + 6), tr.slot(X + 8)
    ninv = F2(tr.mul(n.a, ni), -tr.mul(n.b, ni)).hold()
    s = [(v * ninv).hold() for v in t]
    r0, r1 = f6mul([f[0], f[2], f[4]], s), f6mul([f[1], f[3], f[5]], s)
    for k in range(3):
        put(out, B + 4 * k, r0[k])
        put(out, B + 4 * k + 2, -r1[k])
    return tr, out


def g1at(tr, s): return tr.slot(s), tr.slot(s + 1), tr.slot(s + 2)


def prog_vdbl():
    """A_j = 2 A_j on G1 (complete, Renes-Costello-Batina algorithm 9), j = 0, 1"""
    tr, out = Trace(), {}
    m = tr.mul

    def hold(v): return LC(tr, {tr.lin(v): 1})
    for j in range(2):
        x, y, z = g1at(tr, VA + 3 * j)
        yy, yz, zz, xy = m(y, y), m(y, z), m(z, z), m(x, y)
        t2, z3, u, t0 = hold(12 * zz), hold(8 * yy), hold(yy + 12 * zz), hold(yy - 36 * zz)
        out[VA + 3 * j] = 2 * m(t0, xy)
        out[VA + 3 * j + 1] = m(t0, u) + m(t2, z3)
        out[VA + 3 * j + 2] = m(yz, z3)
    return tr, out


def prog_vadd():
    """A_j = A_j + Q_j on G1 (complete, algorithm 7), j = 0, 1"""
    tr, out = Trace(), {}
    m = tr.mul

    def hold(v): return LC(tr, {tr.lin(v): 1})
    for j in range(2):
        x1, y1, z1 = g1at(tr, VA + 3 * j)
        x2, y2, z2 = g1at(tr, VQ + 3 * j)
        t0, t1, t2 = m(x1, x2), m(y1, y2), m(z1, z2)
        t3 = hold(m(x1 + y1, x2 + y2) - t0 - t1)
        t4 = hold(m(y1 + z1, y2 + z2) - t1 - t2)
        s = hold(12 * (m(x1 + z1, x2 + z2) - t0 - t2))
        w, u, v = hold(3 * t0), hold(t1 - 12 * t2), hold(t1 + 12 * t2)
        out[VA + 3 * j] = m(t3, u) - m(t4, s)
        out[VA + 3 * j + 1] = m(s, w) + m(u, v)
        out[VA + 3 * j + 2] = m(v, t4) + m(w, t3)
    return tr, out


def schedule(tr, out):
    """rounds [(kind, [(dst slot, node)])] and the slots used"""
    nodes = tr.nodes
    writes = {s: tr.lin(v) if v.t else None for s, v in out.items()}
    nodes = tr.nodes
    reads = [[] if n[0] == "in" else [k for k, _ in n[1]] + ([k for k, _ in n[2]] if n[0] == "prod" else []) for n in nodes]
    # an output that is an input or shared by two slots is copied
    taken, final = set(), {}
    for s in sorted(writes):
        v = writes[s]
        if v is None:
            nodes.append(("lin", ((tr.node(("in", ZERO)), 1),)))
            reads.append([tr.node(("in", ZERO))])
            v = len(nodes) - 1
        elif nodes[v][0] == "in" or v in taken:
            nodes.append(("lin", ((v, 1),)))
            reads.append([v])
            v = len(nodes) - 1
        taken.add(v)
        final[v] = s
    while len(reads) < len(nodes):
        reads.append([])
    users = [[] for _ in nodes]
    live, stack = set(), list(final)
    while stack:
        v = stack.pop()
        if v in live:
            continue
        live.add(v)
        stack += reads[v]
    for v in live:
        for r in set(reads[v]):
            users[r].append(v)
    cost = {"prod": PROD_COST, "lin": LIN_COST, "in": 0}
    prio = {}

    def path(v):
        if v not in prio:
            prio[v] = cost[nodes[v][0]] + max([path(u) for u in users[v]], default=0)
        return prio[v]
    sys.setrecursionlimit(10000)
    for v in live:
        path(v)
    in_slot = {n[1]: k for k, n in enumerate(nodes) if n[0] == "in" and k in live}
    done = {v for v in live if nodes[v][0] == "in"}
    place = {v: nodes[v][1] for v in done}
    left = {v: len(users[v]) for v in live}
    free, top, rounds = [], TMP, []
    todo = live - done
    while todo:
        ready = [v for v in todo if all(r in done for r in reads[v])]
        # an output may replace an input once all readers of the input are issued (this round's read first)
        def fits(v, batch):
            if v not in final or final[v] not in in_slot:
                return True
            return all(u in done or u in batch or u == v for u in users[in_slot[final[v]]])
        kinds = {}
        for kind in ("prod", "lin"):
            c = sorted([v for v in ready if nodes[v][0] == kind], key=lambda v: -prio[v])
            batch = []
            for v in c:
                if len(batch) < LANES and fits(v, ()):
                    batch.append(v)
            for v in c:
                if len(batch) < LANES and v not in batch and fits(v, batch):
                    batch.append(v)
            kinds[kind] = batch
        if not kinds["prod"] and not kinds["lin"]:
            # outputs that wait only for each other's reads: no reader is left outside them
            c = [v for v in ready if v in final]
            raise SystemExit("stuck with %d" % len(c))
        best = {k: max([prio[v] for v in b], default=-1) for k, b in kinds.items()}
        kind = "lin" if kinds["lin"] and (best["lin"] >= best["prod"] or not kinds["prod"]) else "prod"
        if kind == "lin" and kinds["prod"] and len(kinds["prod"]) >= LANES and best["prod"] + LIN_COST > best["lin"]:
            kind = "prod"
        batch = kinds[kind]
        ops = []
        for v in batch:
            if v in final:
                place[v] = final[v]
            elif free:
                place[v] = free.pop()
            else:
                place[v] = top
                top += 1
            ops.append(v)
        for v in batch:
            for r in set(reads[v]):
                left[r] -= 1
                if left[r] == 0 and nodes[r][0] != "in" and r not in final:
                    free.append(place[r])
        done |= set(batch)
        todo -= set(batch)
        rounds.append((kind, [(place[v], v) for v in ops]))
    assert top <= 255
    code = []
    for kind, ops in rounds:
        lanes = []
        for d, v in ops:
            n = nodes[v]
            if kind == "prod":
                ref = []
                for side in (n[1], n[2]):
                    side = list(side) + [(None, 1)] * (2 - len(side))
                    ref += [(ZERO if k is None else place_at(place, k), c) for k, c in side]
                lanes.append((d, ref))
            else:
                lanes.append((d, [(place_at(place, k), c) for k, c in n[1]]))
        code.append((kind, lanes))
    return code, top


def place_at(place, k):
    return place[k]


PROGRAMS = (("DBL", prog_dbl), ("ADD", prog_add), ("MUL", prog_mul), ("CYC", prog_cyc), ("INV1", prog_inv1),
            ("INV2", prog_inv2), ("VDBL", prog_vdbl), ("VADD", prog_vadd))


def build():
    """{name: rounds}, slots used; each round (kind, [(dst, [(slot, coefficient)])])"""
    progs, slots = {}, 0
    for name, fn in PROGRAMS:
        code, top = schedule(*fn())
        progs[name] = code
        slots = max(slots, top)
    return progs, slots


def words(kind, lanes):
    """16 bytes per lane as 4 little-endian words, and the round's header:
    0 PROD with single operands, 1 PROD, 8 + n LIN of up to n terms"""
    out, head = [], 0
    for k in range(LANES):
        d, refs = lanes[k] if k < len(lanes) else (DUMP, [])
        b = [d]
        if kind == "prod":
            refs = refs + [(ZERO, 1)] * (4 - len(refs))
            b += [s for s, _ in refs] + [sum((c < 0) << i for i, (_, c) in enumerate(refs))]
            if refs[1][0] != ZERO or refs[3][0] != ZERO:
                head = 1
        else:
            head = max(head, len(refs))
            b += [0]
            refs = refs + [(ZERO, 0)] * (TERMS - len(refs))
            for s, c in refs:
                b += [s, c & 0xFF]
        b += [0] * (16 - len(b))
        out.append([int.from_bytes(bytes(b[i:i + 4]), "little") for i in range(0, 16, 4)])
    return head + (8 if kind == "lin" else 0), out


def main():
    progs, slots = build()
    print("// pairing_prog.inc -- written by gen_pairing_prog.py (run it to regenerate; do not edit).")
    print("// clang-format off")
    print("constexpr int PV_SLOTS = %d;" % slots)
    names = ("ZERO", ZERO), ("ONE", ONE), ("DUMP", DUMP), ("ACC", ACC), ("B", B), ("M", M), ("S1", S1), ("S2", S2), ("T", T), ("PT", PT), ("Q", Q), ("X", X), ("VA", VA), ("VQ", VQ), ("VT", VT)
    for n, v in names:
        print("constexpr int PV_%s = %d;" % (n, v))
    at, heads, data = 0, [], []
    for name, rounds in progs.items():
        print("constexpr int PV_%s_AT = %d, PV_%s_ROUNDS = %d;  // %d products, %d sums" % (
            name, at, name, len(rounds), sum(len(l) for k, l in rounds if k == "prod"),
            sum(len(l) for k, l in rounds if k == "lin")))
        for kind, lanes in rounds:
            h, w = words(kind, lanes)
            heads.append(h)
            data.append(w)
        at += len(rounds)
    print("__device__ const unsigned char c_pv_head[%d] = {%s};" % (len(heads), ", ".join(map(str, heads))))
    print("__device__ const uint4 c_pv_code[%d][32] = {" % len(data))
    for w in data:
        print("    {" + ", ".join("{0x%xu, 0x%xu, 0x%xu, 0x%xu}" % tuple(x) for x in w) + "},")
    print("};")
    print("// clang-format on")


if __name__ == "__main__":
    main()
