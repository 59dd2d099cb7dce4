#!/usr/bin/env python3
"""Writes chains.inc: the carry chains of the Fp (12 x 32-bit limbs) and Fr
(8 limbs) arithmetic in field.cuh, each chain ONE inline-PTX statement.

A chain of add.cc / addc.cc / mad.lo.cc / madc.hi.cc ... instructions passes
the carry flag CC.CF from one instruction to the next.  The flag is invisible
to the compiler, so a chain written as separate asm statements depends on
nothing being placed between them that also writes the flag.  Here every
chain starts with an instruction that does not read the flag and ends with
one whose flag output is not used, and lives entirely inside one asm
statement, so no code can come between its links.

The generated functions are specialisations for the two descriptors FpDesc
and FrDesc (field.cuh); the modulus enters as immediates ("n" operands) read
from the descriptor, so the constants have one source.  Host builds use the
portable stand-ins in field.cuh instead (ch_* there call these in
device code).

Run from this directory: python gen_chains.py > chains.inc"""

FIELDS = (("FpDesc", 12), ("FrDesc", 8))


def block(name, sig, lines, outs, ins):
    """One device function whose body is a single asm statement."""
    body = ['"%s;\\n\\t"' % l for l in lines]
    txt = "template <> FK_D %s %s<%s>(%s) {\n" % (sig[0], name, sig[1], sig[2])
    txt += sig[3]
    txt += "    asm volatile(" + "\n        ".join(body) + "\n"
    txt += "        : " + ", ".join(outs) + "\n"
    txt += "        : " + ", ".join(ins) + ");\n"
    txt += sig[4]
    txt += "}\n"
    return txt


def gen(desc, n):
    out = []
    half = n // 2

    # r = a + b (the carry out of the top word is dropped: callers keep sums < 2^(32n))
    outs = ['"=r"(r[%d])' % i for i in range(n)]
    ins = ['"r"(a[%d])' % i for i in range(n)] + ['"r"(b[%d])' % i for i in range(n)]
    A = lambda i: "%%%d" % (n + i)
    B = lambda i: "%%%d" % (2 * n + i)
    lines = ["add.cc.u32 %%0, %s, %s" % (A(0), B(0))]
    lines += ["addc.cc.u32 %%%d, %s, %s" % (i, A(i), B(i)) for i in range(1, n - 1)]
    lines += ["addc.u32 %%%d, %s, %s" % (n - 1, A(n - 1), B(n - 1))]
    out.append(block("ptx_add", ("void", desc, "uint32_t *r, const uint32_t *a, const uint32_t *b", "", ""),
                     lines, outs, ins))

    # r = a - b; returns all ones when a < b (a borrow out of the top word), else 0
    outs = ['"=r"(r[%d])' % i for i in range(n)] + ['"=r"(mask)']
    Ai = lambda i: "%%%d" % (n + 1 + i)
    Bi = lambda i: "%%%d" % (2 * n + 1 + i)
    lines = ["sub.cc.u32 %%0, %s, %s" % (Ai(0), Bi(0))]
    lines += ["subc.cc.u32 %%%d, %s, %s" % (i, Ai(i), Bi(i)) for i in range(1, n)]
    lines += ["subc.u32 %%%d, 0, 0" % n]
    out.append(block("ptx_sub", ("uint32_t", desc, "uint32_t *r, const uint32_t *a, const uint32_t *b",
                                "    uint32_t mask;\n", "    return mask;\n"), lines, outs, ins))

    # r = t - modulus; returns all ones when t < modulus
    ins = ['"r"(t[%d])' % i for i in range(n)] + ['"n"(%s::mod(%d))' % (desc, i) for i in range(n)]
    lines = ["sub.cc.u32 %%0, %s, %s" % (Ai(0), Bi(0))]
    lines += ["subc.cc.u32 %%%d, %s, %s" % (i, Ai(i), Bi(i)) for i in range(1, n)]
    lines += ["subc.u32 %%%d, 0, 0" % n]
    out.append(block("ptx_sub_mod", ("uint32_t", desc, "uint32_t *r, const uint32_t *t",
                                    "    uint32_t mask;\n", "    return mask;\n"), lines, outs, ins))

    # product row, even half: e[0..n-1] += a[j] * b for even j (lo word at j,
    # hi word at j + 1); e[n] = the carry out (its old value is not read)
    outs = ['"+r"(e[%d])' % i for i in range(n)] + ['"=r"(e[%d])' % n]
    ins = ['"r"(a[%d])' % (2 * k) for k in range(half)] + ['"r"(b)']
    a_ = lambda k: "%%%d" % (n + 1 + k)
    b_ = "%%%d" % (n + 1 + half)
    lines = []
    for k in range(half):
        lo, hi = 2 * k, 2 * k + 1
        lines.append("%s.u32 %%%d, %s, %s, %%%d" % ("mad.lo.cc" if k == 0 else "madc.lo.cc", lo, a_(k), b_, lo))
        lines.append("madc.hi.cc.u32 %%%d, %s, %s, %%%d" % (hi, a_(k), b_, hi))
    lines.append("addc.u32 %%%d, 0, 0" % n)
    out.append(block("ptx_row_even", ("void", desc, "uint32_t *e, const uint32_t *a, uint32_t b", "", ""),
                     lines, outs, ins))

    # product row, odd half (o[k] is word k + 1): o[0..n-1] += a[j] * b for odd j
    # (lo word at o[j-1], hi word at o[j]); no carry out of o[n-1], whose old
    # value is 0
    outs = ['"+r"(o[%d])' % i for i in range(n - 1)] + ['"=r"(o[%d])' % (n - 1)]
    ins = ['"r"(a[%d])' % (2 * k + 1) for k in range(half)] + ['"r"(b)']
    a_ = lambda k: "%%%d" % (n + k)
    b_ = "%%%d" % (n + half)
    lines = []
    for k in range(half):
        lo, hi = 2 * k, 2 * k + 1
        lines.append("%s.u32 %%%d, %s, %s, %%%d" % ("mad.lo.cc" if k == 0 else "madc.lo.cc", lo, a_(k), b_, lo))
        if k < half - 1:
            lines.append("madc.hi.cc.u32 %%%d, %s, %s, %%%d" % (hi, a_(k), b_, hi))
        else:
            lines.append("madc.hi.u32 %%%d, %s, %s, 0" % (hi, a_(k), b_))
    out.append(block("ptx_row_odd", ("void", desc, "uint32_t *o, const uint32_t *a, uint32_t b", "", ""),
                     lines, outs, ins))

    # reduction, even half: e[0..n-1] += m * mod[j] for even j; e[n] += carry
    outs = ['"+r"(e[%d])' % i for i in range(n + 1)]
    ins = ['"r"(m)'] + ['"n"(%s::mod(%d))' % (desc, 2 * k) for k in range(half)]
    m_ = "%%%d" % (n + 1)
    p_ = lambda k: "%%%d" % (n + 2 + k)
    lines = []
    for k in range(half):
        lo, hi = 2 * k, 2 * k + 1
        lines.append("%s.u32 %%%d, %s, %s, %%%d" % ("mad.lo.cc" if k == 0 else "madc.lo.cc", lo, m_, p_(k), lo))
        lines.append("madc.hi.cc.u32 %%%d, %s, %s, %%%d" % (hi, m_, p_(k), hi))
    lines.append("addc.u32 %%%d, %%%d, 0" % (n, n))
    out.append(block("ptx_red_even", ("void", desc, "uint32_t *e, uint32_t m", "", ""), lines, outs, ins))

    # reduction, odd half: e0 += x (word 0; the carry goes on to word 1), then
    # o[0..n-1] += m * mod[j] for odd j (lo word at o[j-1], hi word at o[j])
    outs = ['"+r"(o[%d])' % i for i in range(n)] + ['"+r"(e0)']
    ins = ['"r"(m)', '"r"(x)'] + ['"n"(%s::mod(%d))' % (desc, 2 * k + 1) for k in range(half)]
    m_, x_ = "%%%d" % (n + 1), "%%%d" % (n + 2)
    q_ = lambda k: "%%%d" % (n + 3 + k)
    lines = ["add.cc.u32 %%%d, %%%d, %s" % (n, n, x_)]
    for k in range(half):
        lo, hi = 2 * k, 2 * k + 1
        lines.append("madc.lo.cc.u32 %%%d, %s, %s, %%%d" % (lo, m_, q_(k), lo))
        lines.append("%s.u32 %%%d, %s, %s, %%%d" % ("madc.hi.cc" if k < half - 1 else "madc.hi", hi, m_, q_(k), hi))
    out.append(block("ptx_red_odd", ("void", desc, "uint32_t *o, uint32_t m, uint32_t &e0, uint32_t x", "", ""), lines, outs, ins))

    # squaring rows I = 1 .. n-1 (row 0 is plain products): e[j0..n-1] += v[j] * b
    # for even j >= I (lo word at j, hi word at j + 1), e[n] = the carry out;
    # odd j >= I: lo word at o[j-1], hi word at o[j], no carry out of o[n-1],
    # whose old value is 0
    for I in range(1, n):
        for par, acc in ((0, "e"), (1, "o")):
            js = [j for j in range(I, n) if j % 2 == par]
            name = "ptx_sqrow_even" if par == 0 else "ptx_sqrow_odd"
            sig = ("void", "%s, %d" % (desc, I), "uint32_t *%s, const uint32_t *v, uint32_t b" % acc, "", "")
            if not js:
                out.append("template <> FK_D void %s<%s, %d>(uint32_t *, const uint32_t *, uint32_t) {}\n" % (name, desc, I))
                continue
            words = list(range(js[0] - par, n))
            outs = ['"%s"(%s[%d])' % ("=r" if par == 1 and w == n - 1 else "+r", acc, w) for w in words]
            if par == 0:
                outs.append('"=r"(%s[%d])' % (acc, n))
            op = {w: "%%%d" % k for k, w in enumerate(words + ([n] if par == 0 else []))}
            base = len(outs)
            ins = ['"r"(v[%d])' % j for j in js] + ['"r"(b)']
            vj = {j: "%%%d" % (base + k) for k, j in enumerate(js)}
            b_ = "%%%d" % (base + len(js))
            lines = []
            for k, j in enumerate(js):
                lo, hi = j - par, j - par + 1
                lines.append("%s.u32 %s, %s, %s, %s" % ("mad.lo.cc" if k == 0 else "madc.lo.cc", op[lo], vj[j], b_, op[lo]))
                if par == 1 and j == js[-1]:
                    lines.append("madc.hi.u32 %s, %s, %s, 0" % (op[hi], vj[j], b_))
                else:
                    lines.append("madc.hi.cc.u32 %s, %s, %s, %s" % (op[hi], vj[j], b_, op[hi]))
            if par == 0:
                lines.append("addc.u32 %s, 0, 0" % op[n])
            out.append(block(name, sig, lines, outs, ins))

    # t[k] = e[k+1] + o[k], k < n (the carry out of the top word is dropped)
    outs = ['"=r"(t[%d])' % i for i in range(n)]
    ins = ['"r"(e[%d])' % i for i in range(1, n + 1)] + ['"r"(o[%d])' % i for i in range(n)]
    lines = ["add.cc.u32 %%0, %%%d, %%%d" % (n, 2 * n)]
    lines += ["addc.cc.u32 %%%d, %%%d, %%%d" % (k, n + k, 2 * n + k) for k in range(1, n - 1)]
    lines += ["addc.u32 %%%d, %%%d, %%%d" % (n - 1, 2 * n - 1, 3 * n - 1)]
    out.append(block("ptx_final", ("void", desc, "uint32_t *t, const uint32_t *e, const uint32_t *o", "", ""),
                     lines, outs, ins))
    return out


def main():
    print("// chains.inc -- written by gen_chains.py (run it to regenerate; do not edit).")
    print("// One asm statement per carry chain of the Fp and Fr arithmetic (field.cuh).")
    print("// clang-format off")
    for desc, n in FIELDS:
        print("\n// ---------------------------------------------------------------- %s (%d limbs)\n" % (desc, n))
        for f in gen(desc, n):
            print(f)
    print("// clang-format on")


if __name__ == "__main__":
    main()
