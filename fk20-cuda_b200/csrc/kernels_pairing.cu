// kernels_pairing.cu -- BLS12-381 pairing checks, for verifying KZG proofs.
//
// The reference verifies multiproofs with py_ecc's pairing (check_proof_multi,
// FK20Py/kzg_proofs.py:207-232; no CUDA counterpart).  This is the optimal
// ate pairing of BLS12 curves computed with the standard techniques:
//   * Fp2 = Fp[u]/(u^2 + 1), Fp6 = Fp2[v]/(v^3 - xi), Fp12 = Fp6[w]/(w^2 - v),
//     xi = 1 + u (so w^6 = xi); Karatsuba products at every level (an Fp12
//     product is 18 Fp2 products, a square 12, a product by a line 13; a
//     square in the cyclotomic subgroup, where the final exponentiation
//     works, 9 Fp2 squares).
//   * G2 on the M-type twist E': y^2 = x^3 + 4 xi, mapped into E(Fp12) by
//     psi(x', y') = (x'/w^2, y'/w^3).
//   * Miller loop over the bits of |z| = 0xd201000000010000 with T in
//     homogeneous projective coordinates (no inversions); the line through T
//     (tangent, or chord through Q) evaluated at P is c0 + c2 w^2 + c3 w^3
//     up to a factor in Fp2, which the final exponentiation removes:
//       tangent: c0 = Y^2 - 3b'Z^2, c2 = -3X^2 xP, c3 = 2YZ yP;
//       chord:   c0 = th xQ - la yQ, c2 = -th xP, c3 = la yP,
//                th = Y - yQ Z, la = X - xQ Z.
//     Both pairings of a check share one loop (one squaring of f per bit).
//     As z < 0 and the loop runs over |z|, the value is the inverse of the
//     usual normalisation: non-degenerate and bilinear all the same.
//   * Final exponentiation by 3 (p^12 - 1)/r: the easy part
//     m = f^((p^6 - 1)(p^2 + 1)) by conjugation, one inversion and a
//     Frobenius map; the hard part by the decomposition
//     3 (p^4 - p^2 + 1)/r = (z - 1)^2 (z + p)(z^2 + p^2 - 1) + 3
//     (five exponentiations by z, Frobenius maps, conjugations for the
//     inverses of the cyclotomic subgroup).  A fixed exponent coprime to r
//     keeps a check's answer the same: f^(3(p^12-1)/r) == 1 exactly when
//     f^((p^12-1)/r) == 1.
// Two kernels.  One warp per pairing or check (k_pairing): its Fp values are
// slots in shared memory and the steps above are programs of rounds
// (pairing_prog.inc, traced and scheduled by gen_pairing_prog.py); a round
// gives every lane one Fp product or one sum, so a Miller step with both lines
// is 8 products deep instead of 226, and a cyclotomic square 1 instead of 18.
// One thread per check (k_pairing_threads), its values in local memory and the
// Fp2 / Fp6 / Fp12 products out of line, is thousands of products
// deep but needs fewer instructions, so it takes over where checks fill the
// chip (launch_pairing).
#define FK_FP_MUL_OUTLINE 1
#include "glv.cuh"
#include "launch.h"
#include "layout.cuh"
#include "tower.cuh"
#include "pairing_prog.inc"

namespace fk {

constexpr unsigned long long Z_ABS = 0xd201000000010000ull;

// ---------------------------------------------------------------- Miller loop
struct G2H {  // homogeneous projective point of the twist
    Fp2 x, y, z;
};
// T = 2T; l = (c0, c2, c3) of the tangent at T evaluated at P
static __device__ __noinline__ void dbl_step(G2H *T, Fp2 *l, const Fp *xp, const Fp *yp) {
    Fp2 B = f2s(T->y), C = f2s(T->z), E, F, XX = f2s(T->x), H, t, u, c2, c3;
    f2_xi(t, C);
    f2_mul12(E, t);  // 3 b' Z^2 = 12 xi Z^2
    f2_add(F, E, E);
    f2_add(F, F, E);  // 3 E
    H = f2m(T->y, T->z);
    f2_add(H, H, H);  // 2 Y Z
    f2_sub(t, B, E);
    f2_add(u, XX, XX);
    f2_add(u, u, XX);
    f2_mul_fp(c2, u, *xp);
    f2_neg(c2, c2);
    f2_mul_fp(c3, H, *yp);
    l[0] = t;
    l[1] = c2;
    l[2] = c3;
    t = f2m(T->x, T->y);
    f2_add(t, t, t);
    f2_sub(u, B, F);
    T->x = f2m(t, u);  // 2 X Y (B - F)
    f2_add(t, B, F);
    T->y = f2s(t);
    u = f2s(E);
    f2_mul12(u, u);
    f2_sub(T->y, T->y, u);  // (B + F)^2 - 12 E^2
    t = f2m(B, H);
    f2_add(t, t, t);
    f2_add(T->z, t, t);  // 4 B H
}
// T = T + Q (Q affine); l = (c0, c2, c3) of the chord through T and Q evaluated at P
static __device__ __noinline__ void add_step(G2H *T, Fp2 *l, const Fp2 *xq, const Fp2 *yq, const Fp *xp,
                                             const Fp *yp) {
    Fp2 th, la, t, u, c0, c2, c3, C, D, E, F, G, H;
    t = f2m(*yq, T->z);
    f2_sub(th, T->y, t);
    t = f2m(*xq, T->z);
    f2_sub(la, T->x, t);
    t = f2m(th, *xq);
    u = f2m(la, *yq);
    f2_sub(c0, t, u);
    f2_mul_fp(c2, th, *xp);
    f2_neg(c2, c2);
    f2_mul_fp(c3, la, *yp);
    l[0] = c0;
    l[1] = c2;
    l[2] = c3;
    C = f2s(th);
    D = f2s(la);
    E = f2m(la, D);
    F = f2m(T->z, C);
    G = f2m(T->x, D);
    f2_add(H, E, F);
    f2_sub(H, H, G);
    f2_sub(H, H, G);
    T->x = f2m(la, H);
    f2_sub(t, G, H);
    t = f2m(th, t);
    u = f2m(T->y, E);
    f2_sub(T->y, t, u);
    T->z = f2m(T->z, E);
}
// f = prod over the n (<= 2) pairs of their Miller values (P affine over Fp,
// Q affine on the twist, neither infinity)
static __device__ __noinline__ void miller(Fp12 *f, int n, const Fp *xp, const Fp *yp, const Fp2 *xq, const Fp2 *yq) {
    G2H T[2];
    Fp2 l[3];
#pragma unroll 1
    for (int j = 0; j < n; j++) {
        T[j].x = xq[j];
        T[j].y = yq[j];
        f2_one(T[j].z);
    }
    f12_one(*f);
#pragma unroll 1
    for (int i = 62; i >= 0; i--) {
        f12_sqr(f, f);
#pragma unroll 1
        for (int j = 0; j < n; j++) {
            dbl_step(&T[j], l, &xp[j], &yp[j]);
            f12_mul_line(f, l);
        }
        if ((Z_ABS >> i) & 1ull) {
#pragma unroll 1
            for (int j = 0; j < n; j++) {
                add_step(&T[j], l, &xq[j], &yq[j], &xp[j], &yp[j]);
                f12_mul_line(f, l);
            }
        }
    }
}

// ---------------------------------------------------------------- final exponentiation
// r = a^z (z = -|z| < 0, a in the cyclotomic subgroup, where the inverse is
// the conjugate); r may alias a
static __device__ __noinline__ void exp_z(Fp12 *r, const Fp12 *a) {
    Fp12 acc = *a;
#pragma unroll 1
    for (int i = 62; i >= 0; i--) {
        f12_cyc_sqr(&acc, &acc);
        if ((Z_ABS >> i) & 1ull) f12_mul(&acc, &acc, a);
    }
    f12_conj(*r, acc);
}
// r = f^(3 (p^12 - 1) / r)
static __device__ __noinline__ void final_exp(Fp12 *r, const Fp12 *f) {
    Fp12 m, t, a, b, c;
    f12_inv(&t, f);  // easy part: m = f^((p^6 - 1)(p^2 + 1))
    f12_conj(m, *f);
    f12_mul(&m, &m, &t);
    f12_frob(&t, &m, false);
    f12_mul(&m, &t, &m);
    exp_z(&a, &m);  // a = m^(z - 1)
    f12_conj(t, m);
    f12_mul(&a, &a, &t);
    exp_z(&t, &a);  // a = a^(z - 1)
    f12_conj(a, a);
    f12_mul(&a, &t, &a);
    exp_z(&b, &a);  // b = a^(z + p)
    f12_frob(&t, &a, true);
    f12_mul(&b, &b, &t);
    exp_z(&c, &b);  // c = b^(z^2 + p^2 - 1)
    exp_z(&c, &c);
    f12_frob(&t, &b, false);
    f12_mul(&c, &c, &t);
    f12_conj(t, b);
    f12_mul(&c, &c, &t);
    f12_cyc_sqr(&t, &m);  // times m^3
    f12_mul(&t, &t, &m);
    f12_mul(r, &c, &t);
}

// ---------------------------------------------------------------- conversions
FK_D void fp_from_words(Fp &m, const uint64_t *w) {
    Fp t;
#pragma unroll
    for (int k = 0; k < 6; k++) { t.w[2 * k] = (uint32_t)w[k]; t.w[2 * k + 1] = (uint32_t)(w[k] >> 32); }
    f_to_mont(m, t);
}
FK_D void fp_to_words(uint64_t *w, const Fp &m) {
    Fp t;
    f_from_mont(t, m);
#pragma unroll
    for (int k = 0; k < 6; k++) w[k] = (uint64_t)t.w[2 * k] | ((uint64_t)t.w[2 * k + 1] << 32);
}
// reference g1p_t -> affine (Montgomery); false for infinity
FK_D bool g1_affine(Fp &x, Fp &y, const uint64_t *g) {
    G1P p;
    g1p_from_ref(p, g);
    if (f_is_zero(p.z)) return false;
    g1_normalize(p);
    x = p.x;
    y = p.y;
    return true;
}
// g2p_t {x0, x1, y0, y1, z0, z1} (36 words, standard form) -> affine; false for infinity
FK_D bool g2_affine(Fp2 &x, Fp2 &y, const uint64_t *g) {
    Fp2 z;
    fp_from_words(x.c0, g);
    fp_from_words(x.c1, g + 6);
    fp_from_words(y.c0, g + 12);
    fp_from_words(y.c1, g + 18);
    fp_from_words(z.c0, g + 24);
    fp_from_words(z.c1, g + 30);
    if (f2_is_zero(z)) return false;
    f2_inv(&z, &z);
    x = f2m(x, z);
    y = f2m(y, z);
    return true;
}
FK_D void g2_store(uint64_t *g, const Fp2 &x, const Fp2 &y, bool inf) {
    if (inf) {
#pragma unroll 1
        for (int k = 0; k < 36; k++) g[k] = 0;
        g[12] = 1;  // (0, 1, 0)
        return;
    }
    fp_to_words(g, x.c0);
    fp_to_words(g + 6, x.c1);
    fp_to_words(g + 12, y.c0);
    fp_to_words(g + 18, y.c1);
    Fp one;
    f_set_one(one);
    fp_to_words(g + 24, one);
#pragma unroll 1
    for (int k = 30; k < 36; k++) g[k] = 0;
}

// affine G2 addition with its special cases; inf flags
static __device__ __noinline__ void g2_add(Fp2 *xr, Fp2 *yr, bool *ir, Fp2 x1, Fp2 y1, bool i1, Fp2 x2, Fp2 y2,
                                           bool i2) {
    if (i1 || i2) {
        *ir = i1 && i2;
        *xr = i1 ? x2 : x1;
        *yr = i1 ? y2 : y1;
        return;
    }
    Fp2 lam, t, u;
    if (f2_eq(x1, x2)) {
        f2_add(t, y1, y2);
        if (f2_is_zero(t)) {  // P + (-P)
            *ir = true;
            return;
        }
        t = f2m(x1, x1);
        f2_add(u, t, t);
        f2_add(t, u, t);
        f2_add(u, y1, y1);
    } else {
        f2_sub(t, y2, y1);
        f2_sub(u, x2, x1);
    }
    f2_inv(&u, &u);
    lam = f2m(t, u);
    t = f2m(lam, lam);
    f2_sub(t, t, x1);
    f2_sub(t, t, x2);
    f2_sub(u, x1, t);
    u = f2m(lam, u);
    f2_sub(*yr, u, y1);
    *xr = t;
    *ir = false;
}

// ---------------------------------------------------------------- the 32-lane machine
constexpr int PV_WARPS = 2;  // checks per block

FK_D void pv_load(Fp &f, const uint32_t *sm, int slot) {
    const uint4 *q = reinterpret_cast<const uint4 *>(sm + 12 * slot);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint4 v = q[k];
        f.w[4 * k] = v.x; f.w[4 * k + 1] = v.y; f.w[4 * k + 2] = v.z; f.w[4 * k + 3] = v.w;
    }
}
FK_D void pv_store(uint32_t *sm, int slot, const Fp &f) {
    uint4 *q = reinterpret_cast<uint4 *>(sm + 12 * slot);
#pragma unroll
    for (int k = 0; k < 3; k++) q[k] = make_uint4(f.w[4 * k], f.w[4 * k + 1], f.w[4 * k + 2], f.w[4 * k + 3]);
}
// x or p - x (p for x = 0: a product or a sum takes it)
FK_D void pv_load_signed(Fp &f, const uint32_t *sm, int slot, bool neg) {
    pv_load(f, sm, slot);
    uint32_t m[12], t[12];
#pragma unroll
    for (int k = 0; k < 12; k++) m[k] = FpDesc::mod(k);
    (void)ch_sub<FpDesc>(t, m, f.w);
#pragma unroll
    for (int k = 0; k < 12; k++) f.w[k] = neg ? t[k] : f.w[k];
}
// acc < 2^7 p as 12 column sums below 2^39, reduced
FK_D void pv_reduce(Fp &r, const uint64_t acc[12]) {
    uint32_t t[13];
    uint64_t c = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        c += acc[k];
        t[k] = (uint32_t)c;
        c >>= 32;
    }
    t[12] = (uint32_t)c;
    // q = floor(top / (top of p + 1)): at most one below acc div p
    const uint64_t h = ((uint64_t)t[12] << 32) | t[11];
    const uint32_t q = (uint32_t)(h / (FpDesc::mod(11) + 1u));
    int64_t b = 0;
    uint32_t u[12];
#pragma unroll
    for (int k = 0; k < 12; k++) {
        b += (int64_t)t[k] - (int64_t)((uint64_t)q * FpDesc::mod(k));
        u[k] = (uint32_t)b;
        b >>= 32;
    }
    f_reduce_once<FpDesc>(r.w, u);
}
static __device__ __noinline__ void pv_run(uint32_t *sm, int at, int rounds, int lane) {
#pragma unroll 1
    for (int i = 0; i < rounds; i++) {
        const int head = c_pv_head[at + i];
        const uint4 w = c_pv_code[at + i][lane];
        Fp r;
        if (head < 8) {
            Fp a, b, t;
            pv_load_signed(a, sm, (w.x >> 8) & 255, w.y & 0x100u);
            pv_load_signed(b, sm, w.x >> 24, w.y & 0x400u);
            if (head) {
                pv_load_signed(t, sm, (w.x >> 16) & 255, w.y & 0x200u);
                f_add(a, a, t);
                pv_load_signed(t, sm, w.y & 255, w.y & 0x800u);
                f_add(b, b, t);
            }
            fp_mul(r, a, b);
        } else {
            uint64_t acc[12];
#pragma unroll
            for (int k = 0; k < 12; k++) acc[k] = 0;
            const int n = head - 8;
#pragma unroll 1
            for (int k = 1; k <= n; k++) {
                const uint32_t word = k < 2 ? w.x : k < 4 ? w.y : k < 6 ? w.z : w.w;
                const uint32_t e = (k & 1) ? word >> 16 : word & 0xffffu;
                const int cf = (int)(int8_t)(e >> 8);
                const uint32_t mag = (uint32_t)(cf < 0 ? -cf : cf);
                Fp x;
                pv_load_signed(x, sm, e & 255, cf < 0);
#pragma unroll
                for (int j = 0; j < 12; j++) acc[j] += (uint64_t)x.w[j] * mag;
            }
            pv_reduce(r, acc);
        }
        __syncwarp();
        pv_store(sm, w.x & 255, r);
        __syncwarp();
    }
}
#define PV_RUN(name) pv_run(sm, PV_##name##_AT, PV_##name##_ROUNDS, lane)

// an Fp12 value to other slots, conjugated over Fp6 if conj
FK_D void pv_copy12(uint32_t *sm, int dst, int src, bool conj, int lane) {
    Fp f;
    if (lane < 12) {
        pv_load(f, sm, src + lane);
        if (conj && ((lane >> 1) & 1)) f_neg(f, f);
    }
    __syncwarp();
    if (lane < 12) pv_store(sm, dst + lane, f);
    __syncwarp();
}
// dst = src^p (conj) or src^(p^2)
FK_D void pv_frob(uint32_t *sm, int dst, int src, bool conj, int lane) {
    Fp2 x, g;
    if (lane < 6) {
        pv_load(x.c0, sm, src + 2 * lane);
        pv_load(x.c1, sm, src + 2 * lane + 1);
        if (conj) f_neg(x.c1, x.c1);
        frob_coef(g, conj ? c_frob1[lane] : c_frob2[lane]);
        x = f2m(x, g);
    }
    __syncwarp();
    if (lane < 6) {
        pv_store(sm, dst + 2 * lane, x.c0);
        pv_store(sm, dst + 2 * lane + 1, x.c1);
    }
    __syncwarp();
}
// ACC = ACC^z in the cyclotomic subgroup (z = -|z|); B is overwritten
static __device__ __noinline__ void pv_exp_z(uint32_t *sm, int lane) {
    pv_copy12(sm, PV_B, PV_ACC, false, lane);
#pragma unroll 1
    for (int i = 62; i >= 0; i--) {
        PV_RUN(CYC);
        if ((Z_ABS >> i) & 1ull) PV_RUN(MUL);
    }
    pv_copy12(sm, PV_ACC, PV_ACC, true, lane);
}

// ---------------------------------------------------------------- kernels
// op 0: out[i] = e(a[i], b[i]) (12 fp_t: the 6 Fp2 coefficients of w);
// op 1: ok[i] = e(a[i], b[i]) == e(c[i], d[i]).
// bcast bit 0: b is one point for every i; bit 1: d likewise.
__global__ void __launch_bounds__(32 * PV_WARPS) k_pairing(int op, uint64_t *out, uint8_t *ok, const uint64_t *a,
                                                          const uint64_t *b, const uint64_t *c, const uint64_t *d,
                                                          size_t count, int bcast) {
    __shared__ __align__(16) uint32_t file[PV_WARPS][PV_SLOTS * 12];
    const int lane = threadIdx.x & 31;
    uint32_t *sm = file[threadIdx.x >> 5];
    const size_t i = blockIdx.x * (size_t)PV_WARPS + (threadIdx.x >> 5);
    if (i >= count) return;
    Fp one, zero;
    f_set_one(one);
    f_set_zero(zero);
    if (lane == 0) {
        pv_store(sm, PV_ZERO, zero);
        pv_store(sm, PV_ONE, one);
    }
    if (lane < 12) pv_store(sm, PV_ACC + lane, lane ? zero : one);
    // lanes 0, 1: the G1 points; 2, 3: the G2 points
    const int j = lane & 1;
    bool finite = false;
    if (lane < 2 && (j == 0 || op == 1)) {
        Fp x, y;
        finite = g1_affine(x, y, (j ? c : a) + 18 * i);
        if (finite) {
            if (j) f_neg(y, y);  // e(c, d)^-1 = e(-c, d)
            pv_store(sm, PV_PT + 2 * j, x);
            pv_store(sm, PV_PT + 2 * j + 1, y);
        }
    }
    Fp2 xq, yq;
    if ((lane == 2 || lane == 3) && (j == 0 || op == 1)) {
        const bool same = bcast & (j ? 2 : 1);
        finite = g2_affine(xq, yq, (j ? d : b) + (same ? 0 : 36 * i));
    }
    // A pair with a point at infinity (or op 0's second) contributes 1: P = (0, 0)
    // leaves of each line its Fp2 term, which the final exponentiation removes;
    // any finite Q whose multiples keep that term nonzero will do: the generator.
    const unsigned fin = __ballot_sync(0xffffffffu, finite);
    const bool pair = ((fin >> j) & (fin >> (2 + j))) & 1u;
    if (lane < 2 && !pair) {
        pv_store(sm, PV_PT + 2 * j, zero);
        pv_store(sm, PV_PT + 2 * j + 1, zero);
    }
    if (lane == 2 || lane == 3) {
        if (!pair) {
#pragma unroll
            for (int k = 0; k < 12; k++) {
                xq.c0.w[k] = c_g2_gen[0][k];
                xq.c1.w[k] = c_g2_gen[1][k];
                yq.c0.w[k] = c_g2_gen[2][k];
                yq.c1.w[k] = c_g2_gen[3][k];
            }
        }
        for (int t = 0; t < 2; t++) {  // Q, and T = Q
            const int at = t ? PV_T + 6 * j : PV_Q + 4 * j;
            pv_store(sm, at, xq.c0);
            pv_store(sm, at + 1, xq.c1);
            pv_store(sm, at + 2, yq.c0);
            pv_store(sm, at + 3, yq.c1);
        }
        pv_store(sm, PV_T + 6 * j + 4, one);
        pv_store(sm, PV_T + 6 * j + 5, zero);
    }
    __syncwarp();
#pragma unroll 1
    for (int k = 62; k >= 0; k--) {
        PV_RUN(DBL);
        if ((Z_ABS >> k) & 1ull) PV_RUN(ADD);
    }
    // easy part: m = f^((p^6 - 1)(p^2 + 1))
    PV_RUN(INV1);
    if (lane == 0) {
        Fp n;
        pv_load(n, sm, PV_X + 8);
        f_inv(n, n);
        pv_store(sm, PV_X + 8, n);
    }
    __syncwarp();
    PV_RUN(INV2);
    pv_copy12(sm, PV_ACC, PV_ACC, true, lane);
    PV_RUN(MUL);
    pv_frob(sm, PV_B, PV_ACC, false, lane);
    PV_RUN(MUL);
    pv_copy12(sm, PV_M, PV_ACC, false, lane);
    // hard part: (z - 1)^2 (z + p) (z^2 + p^2 - 1) + 3
    pv_exp_z(sm, lane);
    pv_copy12(sm, PV_B, PV_M, true, lane);
    PV_RUN(MUL);  // m^(z - 1)
    pv_copy12(sm, PV_S1, PV_ACC, false, lane);
    pv_exp_z(sm, lane);
    pv_copy12(sm, PV_B, PV_S1, true, lane);
    PV_RUN(MUL);  // m^((z - 1)^2)
    pv_copy12(sm, PV_S1, PV_ACC, false, lane);
    pv_exp_z(sm, lane);
    pv_frob(sm, PV_B, PV_S1, true, lane);
    PV_RUN(MUL);
    pv_copy12(sm, PV_S2, PV_ACC, false, lane);  // b = .. ^(z + p)
    pv_exp_z(sm, lane);
    pv_exp_z(sm, lane);
    pv_frob(sm, PV_B, PV_S2, false, lane);
    PV_RUN(MUL);
    pv_copy12(sm, PV_B, PV_S2, true, lane);
    PV_RUN(MUL);  // b^(z^2 + p^2 - 1)
    pv_copy12(sm, PV_S1, PV_ACC, false, lane);
    pv_copy12(sm, PV_ACC, PV_M, false, lane);
    pv_copy12(sm, PV_B, PV_M, false, lane);
    PV_RUN(CYC);
    PV_RUN(MUL);
    pv_copy12(sm, PV_B, PV_S1, false, lane);
    PV_RUN(MUL);  // times m^3
    Fp e;
    if (lane < 12) pv_load(e, sm, PV_ACC + lane);
    if (op == 1) {
        const bool is = lane >= 12 || f_eq(e, lane ? zero : one);
        const bool all = __all_sync(0xffffffffu, is);
        if (lane == 0) ok[i] = all ? 1 : 0;
    } else if (lane < 12) {
        fp_to_words(out + 72 * i + 6 * lane, e);
    }
}

// The same, one thread per check: under half of the warp kernel's instructions a
// check, nine times as deep.
__global__ void __launch_bounds__(64) k_pairing_threads(int op, uint64_t *out, uint8_t *ok, const uint64_t *a,
                                                const uint64_t *b, const uint64_t *c, const uint64_t *d,
                                                size_t count, int bcast) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= count) return;
    const size_t ib = (bcast & 1) ? 0 : i, id = (bcast & 2) ? 0 : i;
    Fp xp[2], yp[2];
    Fp2 xq[2], yq[2];
    int n = 0;
    if (g1_affine(xp[n], yp[n], a + 18 * i) && g2_affine(xq[n], yq[n], b + 36 * ib)) n++;
    if (op == 1 && g1_affine(xp[n], yp[n], c + 18 * i) && g2_affine(xq[n], yq[n], d + 36 * id)) {
        f_neg(yp[n], yp[n]);  // e(c, d)^-1 = e(-c, d)
        n++;
    }
    Fp12 f, e;
    if (n) miller(&f, n, xp, yp, xq, yq);
    else f12_one(f);
    final_exp(&e, &f);
    if (op == 1) {
        ok[i] = f12_is_one(e) ? 1 : 0;
        return;
    }
#pragma unroll 1
    for (int k = 0; k < 6; k++) {
        const Fp2 &v = (k & 1) ? e.a1.c[k >> 1] : e.a0.c[k >> 1];
        fp_to_words(out + 72 * i + 12 * k, v.c0);
        fp_to_words(out + 72 * i + 12 * k + 6, v.c1);
    }
}

// Interpolation for check_proof_multi (FK20Py/kzg_proofs.py:214-217): from the
// evaluations ys[k] = f(x w^k), k < l (w = w_l), the coefficients of the
// interpolation polynomial I(X) = sum_j c_j X^j, c_j = (1/l) sum_k ys[k] w^-jk
// / x^j, written as poly[32 i + j] (zero above l), and xl[i] = x^l.  Fr in
// Montgomery form inside; fr_t standard form (any representative) in,
// canonical out.  One warp per check, lane j its coefficient j.
__global__ void __launch_bounds__(64) k_interp(uint64_t *poly, uint64_t *xl, const uint64_t *x, const uint64_t *ys,
                                               int log_l, size_t count) {
    const size_t i = blockIdx.x * (size_t)2 + (threadIdx.x >> 5);
    if (i >= count) return;
    const int lane = threadIdx.x & 31, l = 1 << log_l, step = 32 >> log_l;
    Fr y, xm, p, t, acc, w;
    f_set_zero(y);
    if (lane < l) {
        fr_from_ref(t, ys + 4 * ((size_t)l * i + lane));
        f_to_mont(y, t);
    }
    fr_from_ref(t, x + 4 * i);
    f_to_mont(xm, t);
    f_set_zero(acc);
#pragma unroll 1
    for (int k = 0; k < l; k++) {
        Fr v;
#pragma unroll
        for (int q = 0; q < 8; q++) v.w[q] = __shfl_sync(0xffffffffu, y.w[q], k);
        const int e = (lane * k * step) & 31;
#pragma unroll
        for (int q = 0; q < 8; q++) w.w[q] = c_w32_inv[e][q];
        f_mul(t, v, w);
        f_add(acc, acc, t);
    }
    // lane j: x^j, then (1/l) x^-j (the lanes' inverses run together)
    f_set_one(p);
#pragma unroll 1
    for (int q = 4; q >= 0; q--) {
        f_mul(p, p, p);
        if ((lane >> q) & 1) f_mul(p, p, xm);
    }
    f_inv(p, p);
#pragma unroll
    for (int q = 0; q < 8; q++) t.w[q] = c_inv_pow2[log_l][q];
    f_mul(p, p, t);
    f_mul(acc, acc, p);
    f_from_mont(t, acc);
    if (lane >= l) f_set_zero(t);
    fr_to_ref(poly + 4 * (32 * i + lane), t);
    if (lane == 0) {
        t = xm;
#pragma unroll 1
        for (int q = 0; q < log_l; q++) f_mul(t, t, t);
        f_from_mont(acc, t);
        fr_to_ref(xl + 4 * i, acc);
    }
}

// signed 4-bit windows of the GLV half `half` (0: k mod lambda, 1: k div lambda)
// of a canonical scalar, least significant first
FK_D void glv_digits(int8_t dig[33], const Fr &s, int half) {
    uint32_t s1[4], s2[4];
    glv_split(s1, s2, s.w);
    int carry = 0;
#pragma unroll
    for (int w = 0; w < 32; w++) {
        const int v = (int)(((half ? s2[w >> 3] : s1[w >> 3]) >> (4 * (w & 7))) & 15u) + carry;
        carry = v > 8;
        dig[w] = (int8_t)(v - 16 * carry);
    }
    dig[32] = (int8_t)carry;
}

// k_verify_points' result with a warp per check: both halves' doublings and
// additions are rounds of the 32-lane machine, 2 products and 2 or 3 sums deep
// instead of 8 and 12 products.
__global__ void __launch_bounds__(32 * PV_WARPS) k_verify_points_warp(uint64_t *out, const uint64_t *C, const uint64_t *I,
                                                                     const uint64_t *P, const uint64_t *k,
                                                                     size_t count) {
    __shared__ __align__(16) uint32_t file[PV_WARPS][PV_SLOTS * 12];
    __shared__ int8_t digits[PV_WARPS][2][33];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    uint32_t *sm = file[wp];
    const size_t i = blockIdx.x * (size_t)PV_WARPS + wp;
    if (i >= count) return;
    const auto put = [&](int slot, const G1P &p) {
        pv_store(sm, slot, p.x);
        pv_store(sm, slot + 1, p.y);
        pv_store(sm, slot + 2, p.z);
    };
    // A_j = from[j] (j = 0, 1), three lanes each
    const auto copy = [&](int dst, int src0, int src1, bool neg0, bool neg1) {
        Fp f;
        const int j = lane / 3, c = lane % 3;
        if (lane < 6) {
            const int src = j ? src1 : src0;
            if (src < 0) {  // infinity
                f_set_zero(f);
                if (c == 1) f_set_one(f);
            } else {
                pv_load(f, sm, src + c);
                if (c == 1 && (j ? neg1 : neg0)) f_neg(f, f);
            }
        }
        __syncwarp();
        if (lane < 6) pv_store(sm, dst + lane, f);
        __syncwarp();
    };
    if (lane == 0) {
        Fp f;
        f_set_zero(f);
        pv_store(sm, PV_ZERO, f);
    }
    if (lane < 2) {  // P and phi(P): multiples 1 .. 8 of half j at PV_VT + 24 j
        Fr s;
        G1P p;
        fr_from_ref(s, k + 4 * i);
        glv_digits(digits[wp][lane], s, lane);
        g1p_from_ref(p, P + 18 * i);
        if (lane) g1_phi(p, p);
        put(PV_VT + 24 * lane, p);
    }
    __syncwarp();
    copy(PV_VA, PV_VT, PV_VT + 24, false, false);
    copy(PV_VQ, PV_VT, PV_VT + 24, false, false);
#pragma unroll 1
    for (int e = 1; e < 8; e++) {
        PV_RUN(VADD);
        Fp f;
        if (lane < 6) {
            pv_load(f, sm, PV_VA + lane);
            pv_store(sm, PV_VT + 24 * (lane / 3) + 3 * e + lane % 3, f);
        }
        __syncwarp();
    }
    copy(PV_VA, -1, -1, false, false);
#pragma unroll 1
    for (int w = 32; w >= 0; w--) {
        if (w < 32)
#pragma unroll 1
            for (int b = 0; b < 4; b++) PV_RUN(VDBL);
        const int v0 = digits[wp][0][w], v1 = digits[wp][1][w];
        if (!v0 && !v1) continue;
        copy(PV_VQ, v0 ? PV_VT + 3 * ((v0 < 0 ? -v0 : v0) - 1) : -1, v1 ? PV_VT + 24 + 3 * ((v1 < 0 ? -v1 : v1) - 1) : -1,
             v0 < 0, v1 < 0);
        PV_RUN(VADD);
    }
    // the two halves, then C and -I, each pair in one addition
    if (lane < 2) {
        G1P p;
        g1p_from_ref(p, (lane ? I : C) + 18 * i);
        if (lane) f_neg(p.y, p.y);
        put(PV_VT + 3 * lane, p);
    }
    __syncwarp();
    copy(PV_VQ, PV_VT, PV_VT + 3, false, false);
    PV_RUN(VADD);  // A_0 + C, A_1 - I
    copy(PV_VQ, PV_VA + 3, -1, false, false);
    PV_RUN(VADD);
    if (lane == 0) {
        G1P p;
        pv_load(p.x, sm, PV_VA);
        pv_load(p.y, sm, PV_VA + 1);
        pv_load(p.z, sm, PV_VA + 2);
        g1p_to_ref(out + 18 * i, p);
    }
}

// out[i] = C[i] - I[i] + [k_i] P_i for check_proof_multi: k = k1 + k2 lambda
// (glv.cuh), [k1] P and [k2] phi(P) on neighbouring lanes with signed 4-bit
// windows and complete formulas (32 x 4 doublings and 33 additions deep).  For
// a P with a part outside the order-r subgroup the two halves differ from
// [k] P by a point of the cofactor's order, which the pairing does not see.
// The element-wise product's 256 doublings and ~128 additions are 2.5 times as
// deep.  With the warp kernels of this file, 300 checks 40.6 -> 3.9 ms.
__global__ void __launch_bounds__(64) k_verify_points(uint64_t *out, const uint64_t *C, const uint64_t *I,
                                                      const uint64_t *P, const uint64_t *k, size_t count) {
    const size_t i = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 1;
    const int half = threadIdx.x & 1;
    const bool on = i < count;
    G1P acc, p, q;
    g1_set_inf(acc);
    g1_set_inf(p);
    int8_t dig[33];
    if (on) {
        Fr s;
        fr_from_ref(s, k + 4 * i);
        glv_digits(dig, s, half);
        g1p_from_ref(p, P + 18 * i);
        if (half) g1_phi(p, p);
        G1P tab[8];
        tab[0] = p;
        for (int e = 1; e < 8; e++) g1_add(tab[e], tab[e - 1], p);
#pragma unroll 1
        for (int w = 32; w >= 0; w--) {
            if (w < 32)
                for (int b = 0; b < 4; b++) g1_dbl(acc, acc);
            const int v = dig[w];
            if (v) {
                q = tab[(v < 0 ? -v : v) - 1];
                if (v < 0) f_neg(q.y, q.y);
                g1_add(acc, acc, q);
            }
        }
    }
    __syncwarp();
#pragma unroll
    for (int w = 0; w < 12; w++) {
        q.x.w[w] = __shfl_xor_sync(0xffffffffu, acc.x.w[w], 1);
        q.y.w[w] = __shfl_xor_sync(0xffffffffu, acc.y.w[w], 1);
        q.z.w[w] = __shfl_xor_sync(0xffffffffu, acc.z.w[w], 1);
    }
    if (!on || half) return;
    g1_add(acc, acc, q);
    g1p_from_ref(q, C + 18 * i);
    g1_add(acc, acc, q);
    g1p_from_ref(q, I + 18 * i);
    g1_neg(q, q);
    g1_add(acc, acc, q);
    g1p_to_ref(out + 18 * i, acc);
}

// G2 element-wise: 0 add, 1 dbl, 2 neg, 3 sub, 4 mul by fr_t scalar, 5 normalize,
// 6 on-curve flag (b: uint8 out)
__global__ void __launch_bounds__(64) k_g2_op(int op, uint64_t *out, const uint64_t *a, const void *b,
                                              size_t count) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= count) return;
    Fp2 x1, y1, x2, y2, xr, yr;
    const bool i1 = !g2_affine(x1, y1, a + 36 * i);
    bool ir = true;
    f2_zero(xr);
    f2_zero(yr);
    if (op == 6) {  // y^2 == x^3 + 4 xi, or infinity
        bool on = true;
        if (!i1) {
            Fp2 l = f2m(y1, y1), r = f2m(f2m(x1, x1), x1), bb;
            f_set_zero(bb.c0);
            f_set_zero(bb.c1);
            bb.c0.w[0] = 4;
            Fp t;
            f_to_mont(t, bb.c0);
            bb.c0 = t;
            bb.c1 = t;
            f2_add(r, r, bb);
            on = f2_eq(l, r);
        }
        ((uint8_t *)b)[i] = on ? 1 : 0;
        return;
    }
    if (op == 0 || op == 3) {
        const bool i2 = !g2_affine(x2, y2, (const uint64_t *)b + 36 * i);
        if (op == 3) f2_neg(y2, y2);
        g2_add(&xr, &yr, &ir, x1, y1, i1, x2, y2, i2);
    } else if (op == 1) {
        g2_add(&xr, &yr, &ir, x1, y1, i1, x1, y1, i1);
    } else if (op == 2) {
        xr = x1;
        f2_neg(yr, y1);
        ir = i1;
    } else if (op == 4) {
        const uint64_t *s = (const uint64_t *)b + 4 * i;
#pragma unroll 1
        for (int k = 255; k >= 0; k--) {
            g2_add(&xr, &yr, &ir, xr, yr, ir, xr, yr, ir);
            if ((s[k >> 6] >> (k & 63)) & 1ull) g2_add(&xr, &yr, &ir, xr, yr, ir, x1, y1, i1);
        }
    } else {
        xr = x1;
        yr = y1;
        ir = i1;
    }
    g2_store(out + 36 * i, xr, yr, ir);
}

// One warp each up to here, one thread each beyond: pairings (op 0) and checks (op
// 1).  B200: the warp kernel 2.8 ms to 300 of either (it runs both Miller loops'
// rounds for one pairing too), then 409 k/s: 20.8 ms at 8,288, 25.1 at 10,000; the
// thread kernel 26.2 ms to 10^4 checks, 20.4 to 20.8 to 10^4 pairings, 37.5 and 29.5
// at 37,888.
constexpr size_t PAIRING_WARP_MAX[2] = {8192, 10240};
void launch_pairing(int op, uint64_t *out, uint8_t *ok, const uint64_t *a, const uint64_t *b, const uint64_t *c,
                    const uint64_t *d, size_t count, cudaStream_t st, int bcast) {
    if (count <= PAIRING_WARP_MAX[op])
        k_pairing<<<blocks_for(count, PV_WARPS), 32 * PV_WARPS, 0, st>>>(op, out, ok, a, b, c, d, count, bcast);
    else
        k_pairing_threads<<<blocks_for(count, 64), 64, 0, st>>>(op, out, ok, a, b, c, d, count, bcast);
}
void launch_interp(uint64_t *poly, uint64_t *xl, const uint64_t *x, const uint64_t *ys, int log_l, size_t count,
                   cudaStream_t st) {
    k_interp<<<blocks_for(count, 2), 64, 0, st>>>(poly, xl, x, ys, log_l, count);
}
// Points one warp each up to here, two lanes each beyond.
constexpr size_t VERIFY_WARP_MAX = 2048;
void launch_verify_points(uint64_t *out, const uint64_t *C, const uint64_t *I, const uint64_t *P, const uint64_t *k,
                          size_t count, cudaStream_t st) {
    if (count <= VERIFY_WARP_MAX)
        k_verify_points_warp<<<blocks_for(count, PV_WARPS), 32 * PV_WARPS, 0, st>>>(out, C, I, P, k, count);
    else
        k_verify_points<<<blocks_for(2 * count, 64), 64, 0, st>>>(out, C, I, P, k, count);
}
void launch_g2_op(int op, uint64_t *out, const uint64_t *a, const void *b, size_t count, cudaStream_t st) {
    k_g2_op<<<blocks_for(count, 64), 64, 0, st>>>(op, out, a, b, count);
}

}  // namespace fk
