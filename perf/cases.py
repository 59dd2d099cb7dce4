"""Performance cases of the FK20 engine: the calls a program makes through the
Python binding of the C ABI, from one blob of 1024 coefficients to the
512 x 4096 batch, with the reference's own entry points, commitments, proof
verification and the request server beside them.

Points leave a case as affine coordinates or as 48-byte compressed proofs: a
projective result has no unique words, and a consumer of proofs reads one of
these two forms.  Everything is whole numbers, so results are compared
exactly; `exact` computes them from the known secret tau in Python integers.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "fk20-cuda_b200"))
import fk20b200 as E  # noqa: E402

P = 0x1A0111EA397FE69A4B1BA7B6434BACD764774B84F38512BF6730D2A0F6B0F6241EABFFFEB153FFFFB9FEFFFFFFFFAAAB
R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
G1 = (0x17F1D3A73197D7942695638C4FA9AC0FC3688C4F9774B905A14E3A3F171BAC586C55E83FF97A1AEFFB3AF00ADB22C6BB,
      0x08B3F481E3AAA0F1A09E30ED741D8AE4FCF5E095D5D00AF600DB18CB2C04B3EDD03CC744A2888AE40CAA232946C5E7E1)
G2 = ((0x024AA2B2F08F0A91260805272DC51051C6E47AD4FA403B02B4510B647AE3D1770BAC0326A805BBEFD48056C8C121BDB8,
       0x13E02B6052719F607DACD3A088274F65596BD0D09920B61AB5DA61BBDC7F5049334CF11213945D57E5AC7D055D042B7E),
      (0x0CE5D527727D6E118CC9CDC6DA2E351AADFD9BAA8CBDD3A76D429A695160D12C923AC9CC3BACA289E193548608B82801,
       0x0606C4A02EA734CC32ACD2B02BC28B99CB3E287E85A763AF267492AB572E99AB3F370D275CEC1DA1AAA9075FF05F79BE))
# the secret of the reference harness's test setup (FK20Py/fk20_multi_cuda.py:290-313)
TAU = 1927409816240961209460912649124
LENGTHS = (1024, 2048, 4096)


def listed():
    return [
        # one short blob, one full blob: a node proving a single blob waits for these
        {"name": "proofs_1x1024", "kind": "proofs", "rows": 1, "n": 1024, "window": 10},
        {"name": "proofs_1x4096", "kind": "proofs", "rows": 1, "n": 4096, "window": 10},
        # a handful of blobs, not a whole group of 32 rows
        {"name": "proofs_19x2048", "kind": "proofs", "rows": 19, "n": 2048, "window": 10},
        # the request server's default pack size as one plain batch
        {"name": "h_fft_160x4096", "kind": "h_fft", "rows": 160, "n": 4096, "window": 10},
        # the headline batch, with the larger tables a prover of many batches keeps
        {"name": "h_fft_512x4096", "kind": "h_fft", "rows": 512, "n": 4096, "window": 13},
        # a mixed backlog of blobs of all three lengths in one call
        {"name": "ragged_250", "kind": "ragged", "count": 250, "window": 10},
        # a burst of requests through the continuous-batching server, host buffers in and out
        {"name": "served_48", "kind": "served", "count": 48, "window": 10},
        # the reference's second half alone: points in, proofs out (fk20_hext_fft2h_fft.cu:27)
        {"name": "hext2h_fft_40", "kind": "hext2h_fft", "rows": 40},
        # the reference's inverse G1 transform (g1p_fft.cu:350)
        {"name": "g1_ift_32x512", "kind": "g1_fft", "count": 32, "log_m": 9, "inverse": True},
        # commitments of a block's blobs
        {"name": "commit_48x4096", "kind": "commit", "rows": 48, "n": 4096, "window": 10},
        # a sampling node checks proofs it was sent, some of them wrong
        {"name": "verify_300", "kind": "verify", "count": 300, "l": 16},
        # the reference's Fr transforms in bulk (fr_fft.cu:318)
        {"name": "fr_fft_4000x512", "kind": "fr_fft", "count": 4000, "log_m": 9, "inverse": False},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["proofs", "h_fft", "proofs", "h_fft", "ragged", "served", "hext2h_fft", "g1_fft", "commit",
                       "verify", "fr_fft"])
    if kind in ("proofs", "h_fft"):
        return {"kind": kind, "rows": size(1, 400), "n": rng.choice(LENGTHS), "window": rng.choice([8, 10, 11])}
    if kind == "ragged":
        return {"kind": kind, "count": size(2, 400), "window": rng.choice([8, 10])}
    if kind == "served":
        return {"kind": kind, "count": size(1, 100), "window": 10}
    if kind == "hext2h_fft":
        return {"kind": kind, "rows": size(1, 160)}
    if kind == "g1_fft":
        return {"kind": kind, "count": size(1, 64), "log_m": rng.randint(3, 9), "inverse": rng.random() < 0.5}
    if kind == "commit":
        return {"kind": kind, "rows": size(1, 96), "n": 32 * size(1, 128), "window": rng.choice([8, 10])}
    if kind == "verify":
        return {"kind": kind, "count": size(1, 600), "l": rng.choice([4, 8, 16, 32])}
    return {"kind": kind, "count": size(1, 4000), "log_m": rng.randint(4, 9), "inverse": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
def limbs(values, words):
    data = b"".join(v.to_bytes(8 * words, "little") for v in values)
    return torch.from_numpy(np.frombuffer(data, np.int64).reshape(len(values), words).copy())


def integers(t):
    a = np.ascontiguousarray(t.cpu().numpy())
    w = a.shape[-1] * 8
    b = a.tobytes()
    return [int.from_bytes(b[i:i + w], "little") for i in range(0, len(b), w)]


def scalars(seed, count, device="cuda"):
    """uniform below 2^254 < r"""
    g = torch.Generator(device=device).manual_seed(seed)
    t = torch.randint(-(1 << 63), (1 << 63) - 1, (count, 4), generator=g, device=device, dtype=torch.int64)
    t[:, 3] &= (1 << 62) - 1
    return t


def empty(*shape):
    return torch.empty(shape, dtype=torch.int64, device="cuda")


def g1_multiples(k):
    """[k_i] G1 as g1p_t rows, k on the device"""
    gen = limbs([G1[0], G1[1], 1], 6).reshape(1, 18).cuda().repeat(k.shape[0], 1)
    out = empty(k.shape[0], 18)
    E.call("g1p_op_n", E.G1_OPS["mul"], E._ptr(out), E._ptr(gen), E._ptr(k), k.shape[0], E._stream())
    return out


def powers(count):
    t, out = 1, []
    for _ in range(count):
        out.append(t)
        t = t * TAU % R
    return out


def setup(n):
    return g1_multiples(limbs(powers(n + 1), 4).cuda())


def context(case, lengths):
    c = E.Context(0, case["window"])
    for n in lengths:
        c.load_setup(n, setup(n))
    return c


def ragged_lengths(case):
    """lengths of the requests, in an order of their own for each count"""
    rng = np.random.default_rng(case["count"])
    return [int(v) for v in rng.choice(LENGTHS, case["count"])]


def verify_scalars(case, seed):
    """per check: commitment, quotient, coset x, values ys, expected verdict"""
    rng = np.random.default_rng(seed)
    l, out = case["l"], []
    w = pow(5, (R - 1) // l, R)
    wk = [pow(w, k, R) for k in range(l)]
    tl = pow(TAU, l, R)

    def word():
        return int.from_bytes(rng.bytes(32), "little") % R

    for i in range(case["count"]):
        c, x, r = word(), word(), [word() for _ in range(l)]
        rt = sum(v * pow(TAU, k, R) for k, v in enumerate(r)) % R
        q = (c - rt) * pow(tl - pow(x, l, R), -1, R) % R
        rx = [v * pow(x, k, R) % R for k, v in enumerate(r)]
        ys = [sum(rx[t] * wk[k * t % l] for t in range(l)) % R for k in range(l)]
        wrong = rng.random() < 0.2
        if wrong:
            ys[i % l] = (ys[i % l] + 1) % R
        out.append((c, q, x, ys, 0 if wrong else 1))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("proofs", "h_fft"):
        rows, n = case["rows"], case["n"]
        s["ctx"] = context(case, [n])
        s["poly"] = scalars(seed, rows * n).reshape(rows, n, 4)
        s["out"] = torch.empty((rows, n // 8, 48), dtype=torch.uint8, device="cuda") if kind == "proofs" else empty(rows, n // 8, 18)
    elif kind in ("ragged", "served"):
        s["ctx"] = context(case, LENGTHS)
        s["ns"] = ns = ragged_lengths(case)
        s["poly_off"] = [int(v) for v in np.cumsum([0] + ns[:-1])]
        s["out_off"] = [v // 8 for v in s["poly_off"]]
        polys = scalars(seed, sum(ns))
        if kind == "ragged":
            s["polys"] = polys
            s["out"] = torch.empty((sum(ns) // 8, 48), dtype=torch.uint8, device="cuda")
        else:
            host = polys.cpu().numpy().view(np.uint64)
            s["polys"] = [host[o:o + n] for o, n in zip(s["poly_off"], ns)]
            s["out"] = torch.empty((sum(ns) // 8, 18), dtype=torch.int64).pin_memory()
            s["server"] = E.Server(s["ctx"])
    elif kind == "hext2h_fft":
        s["points"] = g1_multiples(scalars(seed, case["rows"] * 512))
        s["out"] = empty(case["rows"], 512, 18)
    elif kind == "g1_fft":
        m = 1 << case["log_m"]
        s["points"] = g1_multiples(scalars(seed, case["count"] * m))
        s["out"] = empty(case["count"], m, 18)
    elif kind == "commit":
        s["ctx"] = E.Context(0)
        s["ctx"].load_commit(case["n"], setup(case["n"] - 1), case["window"])
        s["poly"] = scalars(seed, case["rows"] * case["n"])
        s["out"] = empty(case["rows"], 18)
    elif kind == "verify":
        s["ctx"] = E.Context(0)
        s["ctx"].load_commit(32, setup(31), 10)
        v = verify_scalars(case, seed)
        s["commitment"] = g1_multiples(limbs([t[0] for t in v], 4).cuda())
        s["proof"] = g1_multiples(limbs([t[1] for t in v], 4).cuda())
        s["x"] = limbs([t[2] for t in v], 4).cuda()
        s["ys"] = limbs([y for t in v for y in t[3]], 4).cuda()
        l = case["l"]
        g2 = limbs([G2[0][0], G2[0][1], G2[1][0], G2[1][1], 1, 0], 6).reshape(1, 36).cuda().repeat(l + 1, 1)
        k = limbs(powers(l + 1), 4).cuda()
        s["setup_g2"] = empty(l + 1, 36)
        E.call("g2p_op_n", E.G2_OPS["mul"], E._ptr(s["setup_g2"]), E._ptr(g2), E._ptr(k), l + 1, E._stream())
        s["out"] = torch.empty(case["count"], dtype=torch.uint8, device="cuda")
    else:
        s["x"] = scalars(seed, case["count"] << case["log_m"])
        s["out"] = torch.empty_like(s["x"])
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def affine(points):
    a = empty(*points.shape[:-1], 12)
    E.call("g1a_fromG1p_n", E._ptr(a), E._ptr(points), points.numel() // 18, E._stream())
    return a


def run(s):
    kind = s["kind"]
    if kind == "proofs":
        s["ctx"].poly2proofs(s["out"], s["poly"], s["rows"], s["n"])
        return s["out"]
    if kind == "h_fft":
        s["ctx"].poly2h_fft(s["out"], s["poly"], s["rows"], s["n"])
        return affine(s["out"])
    if kind == "ragged":
        s["ctx"].batch_proofs(s["out"], s["polys"], s["ns"], s["poly_off"], s["out_off"])
        return s["out"]
    if kind == "served":
        host = s["out"].numpy()
        tickets = [s["server"].submit(p, host[o:o + n // 8]) for p, n, o in zip(s["polys"], s["ns"], s["out_off"])]
        for t in tickets:
            E.check("fk20_server_wait", s["server"].wait(t, 60000))
        return affine(s["out"].cuda())
    if kind == "hext2h_fft":
        E.call("fk20_hext_fft2h_fft", E._ptr(s["out"]), E._ptr(s["points"]), s["rows"], E._stream())
        return affine(s["out"])
    if kind == "g1_fft":
        E.call("g1p_fft_n", E._ptr(s["out"]), E._ptr(s["points"]), s["log_m"], s["count"], int(s["inverse"]), E._stream())
        return affine(s["out"])
    if kind == "commit":
        s["ctx"].commit(s["out"], s["poly"], s["rows"], s["n"])
        return affine(s["out"])
    if kind == "verify":
        s["ctx"].check_proof_multi(s["out"], s["commitment"], s["proof"], s["x"], s["ys"], s["l"], s["setup_g2"],
                                   s["count"])
        return s["out"]
    E.call("fr_fft_n", E._ptr(s["out"]), E._ptr(s["x"]), s["log_m"], s["count"], int(s["inverse"]), E._stream())
    return s["out"]


def work(case):
    """Bytes in and out.  The arithmetic is exact integer work whose least
    amount depends on the algorithm, so no operations are claimed."""
    kind = case["kind"]
    if kind in ("proofs", "h_fft"):
        return {"bytes": case["rows"] * case["n"] * 32 + case["rows"] * case["n"] // 8 * (48 if kind == "proofs" else 96)}
    if kind in ("ragged", "served"):
        return {"bytes": sum(LENGTHS) / 3 * case["count"] * (32 + (48 if kind == "ragged" else 144) / 8)}
    if kind == "hext2h_fft":
        return {"bytes": case["rows"] * 512 * (144 + 96)}
    if kind == "g1_fft":
        return {"bytes": (case["count"] << case["log_m"]) * (144 + 96)}
    if kind == "commit":
        return {"bytes": case["rows"] * (case["n"] * 32 + 96)}
    if kind == "verify":
        return {"bytes": case["count"] * (2 * 144 + 32 + 32 * case["l"] + 1)}
    return {"bytes": (case["count"] << case["log_m"]) * 64}


def tolerance(case):
    return "exact"


# ------------------------------------------------------------------ exact values
def fr_transform(x, inverse):
    m = len(x)
    if m == 1:
        return x
    a = list(x)
    log_m = m.bit_length() - 1
    a = [a[int(format(i, "0%db" % log_m)[::-1], 2)] for i in range(m)]
    w = pow(5, (R - 1) // m, R)
    if inverse:
        w = pow(w, -1, R)
    half = 1
    while half < m:
        step = pow(w, m // (2 * half), R)
        tw = [1]
        for _ in range(half - 1):
            tw.append(tw[-1] * step % R)
        for i in range(0, m, 2 * half):
            for j in range(half):
                u, v = a[i + j], a[i + j + half] * tw[j] % R
                a[i + j], a[i + j + half] = (u + v) % R, (u - v) % R
        half *= 2
    if inverse:
        k = pow(m, -1, R)
        a = [v * k % R for v in a]
    return a


def to_affine(pts):
    """Jacobian points with nonzero Z, one inversion"""
    acc, pre = 1, []
    for q in pts:
        pre.append(acc)
        acc = acc * q[2] % P
    inv, out = pow(acc, -1, P), []
    for q, f in zip(reversed(pts), reversed(pre)):
        zi = inv * f % P
        inv = inv * q[2] % P
        z2 = zi * zi % P
        out.append((q[0] * z2 % P, q[1] * z2 * zi % P))
    return out[::-1]


def jac_dbl(q):
    x, y, z = q
    b = y * y % P
    d = 4 * x * b % P
    e = 3 * x * x % P
    x3 = (e * e - 2 * d) % P
    return x3, (e * (d - x3) - 8 * b * b) % P, 2 * y * z % P


def jac_madd(q, a):
    if q is None:
        return a[0], a[1], 1
    x, y, z = q
    zz = z * z % P
    h, s = (a[0] * zz - x) % P, (a[1] * zz * z - y) % P
    if h == 0:
        return jac_dbl(q) if s == 0 else None
    hh = h * h % P
    hhh, v = h * hh % P, x * hh % P
    x3 = (s * s - hhh - 2 * v) % P
    return x3, (s * (v - x3) - y * hhh) % P, z * h % P


COMB = []


def multiples_of_g(ks):
    """affine (x, y) of [k] G1 for each k, (0, 0) at infinity; 8-bit comb"""
    if not COMB:
        base = G1
        for _ in range(32):
            row = [(base[0], base[1], 1), jac_dbl((base[0], base[1], 1))]
            while len(row) < 255:
                row.append(jac_madd(row[-1], base))
            nxt = jac_madd(row[-1], base)
            row = to_affine(row + [nxt])
            COMB.append(row[:255])
            base = row[255]
    out = []
    for k in ks:
        q = None
        for row in COMB:
            if k & 255:
                q = jac_madd(q, row[(k & 255) - 1])
            k >>= 8
        out.append(q)
    live = iter(to_affine([q for q in out if q is not None]))
    return [(0, 0) if q is None else next(live) for q in out]


def affine_rows(pts, shape):
    return limbs([v for q in pts for v in q], 6).reshape(*shape, 12)


def compressed(pts):
    out = np.zeros((len(pts), 48), np.uint8)
    for i, (x, y) in enumerate(pts):
        b = bytearray(x.to_bytes(48, "big"))
        b[0] |= 0x80 | (0x40 if x == 0 and y == 0 else 0x20 if y > (P - 1) // 2 else 0)
        out[i] = np.frombuffer(bytes(b), np.uint8)
    return torch.from_numpy(out)


def proof_scalars(f):
    """[q_j(tau)] for every j: q_j = f div (X^16 - w_m^j)"""
    n = len(f)
    m = n // 8
    t16, pw = pow(TAU, 16, R), powers(16)
    w = pow(5, (R - 1) // m, R)
    # f = sum_k X^(16 k) f_k: f_k(tau) once, then each remainder at tau is a value of a polynomial in w^j
    fk = [sum(f[16 * k + t] * pw[t] for t in range(16)) % R for k in range(n // 16)]
    total = sum(v * pow(t16, k, R) for k, v in enumerate(fk)) % R
    rem = fr_transform(fk + [0] * (m - len(fk)), False)
    return [(total - rem[j]) * pow(t16 - pow(w, j, R), -1, R) % R for j in range(m)]


def bit_reversed(v):
    bits = len(v).bit_length() - 1
    return [v[int(format(i, "0%db" % bits)[::-1], 2)] for i in range(len(v))]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("proofs", "h_fft"):
        rows, n = case["rows"], case["n"]
        if rows * n > 40000:
            return None
        f = integers(scalars(seed, rows * n))
        ks = [proof_scalars(f[r * n:(r + 1) * n]) for r in range(rows)]
        if kind == "proofs":
            return compressed(multiples_of_g([k for row in ks for k in bit_reversed(row)])).reshape(rows, n // 8, 48)
        return affine_rows(multiples_of_g([k for row in ks for k in row]), (rows, n // 8))
    if kind in ("ragged", "served"):
        ns = ragged_lengths(case)
        if sum(ns) > 130000:
            return None
        f = integers(scalars(seed, sum(ns)))
        ks, at = [], 0
        for n in ns:
            row = proof_scalars(f[at:at + n])
            ks += bit_reversed(row) if kind == "ragged" else row
            at += n
        pts = multiples_of_g(ks)
        return compressed(pts) if kind == "ragged" else affine_rows(pts, (len(pts),))
    if kind in ("hext2h_fft", "g1_fft"):
        m = 512 if kind == "hext2h_fft" else 1 << case["log_m"]
        count = case["rows"] if kind == "hext2h_fft" else case["count"]
        if count * m > 21000:
            return None
        x, ks = integers(scalars(seed, count * m)), []
        for r in range(count):
            row = x[r * m:(r + 1) * m]
            if kind == "hext2h_fft":
                h = fr_transform(row, True)
                ks += fr_transform(h[:m // 2] + [0] * (m // 2), False)
            else:
                ks += fr_transform(row, case["inverse"])
        return affine_rows(multiples_of_g(ks), (count, m))
    if kind == "commit":
        n = case["n"]
        f, pw = integers(scalars(seed, case["rows"] * n)), powers(n)
        ks = [sum(a * b for a, b in zip(f[r * n:(r + 1) * n], pw)) % R for r in range(case["rows"])]
        return affine_rows(multiples_of_g(ks), (case["rows"],))
    if kind == "verify":
        return torch.tensor([t[4] for t in verify_scalars(case, seed)], dtype=torch.uint8)
    m = 1 << case["log_m"]
    if case["count"] * m * case["log_m"] > 20_000_000:
        return None
    x, out = integers(scalars(seed, case["count"] * m)), []
    for r in range(case["count"]):
        out += fr_transform(x[r * m:(r + 1) * m], case["inverse"])
    return limbs(out, 4)
