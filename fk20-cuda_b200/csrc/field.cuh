// field.cuh -- BLS12-381 Fp (381-bit) and Fr (255-bit) Montgomery arithmetic.
//
// Elements are little-endian arrays of 32-bit limbs (Fp: 12, Fr: 8).  Inside
// the engine Fp values are in Montgomery form (x*2^384 mod p) and always
// canonical (< p); Fr data keeps its standard form and is multiplied by
// Montgomery-form constants (x*y*2^-256 with y = w*2^256 gives x*w), so Fr
// FFT outputs are standard-form without conversions.  The reference stores
// plain (non-Montgomery) values with Barrett reduction (fp.cuh:10-14,
// fr.cuh:10-24, fr_mul.cu:58-186); conversion happens at the ABI boundary.
//
// Montgomery product r = A*B/2^(32N): word-serial CIOS with the partial products of each
// word b_i split between two accumulators, `e` (products a_j*b_i with j even:
// lo at word j, hi at word j+1) and `o` (j odd; o[k] is word k + 1).  Within one
// accumulator the lo/hi words of different j never overlap, so each half is a
// single mad.lo.cc/madc.hi.cc carry chain and the two chains are independent.
// The reduction multiple m*p is split the same way.  After it word 0 is 0 and
// everything moves down one word: the accumulators change roles, and the word
// left between them, e[1], joins the next word 0, whose carry goes into the
// next reduction's odd chain.  Bounds: with A < 2p (4p < 2^384) and B < 2^384
// every partial value stays below 2^416, so 13 words suffice, and the result is
// < 2p when A, B < 2p or when A < p (one conditional subtraction of p makes
// it canonical).  A must not exceed ~2^382: a full-width A overflows.
#pragma once
#include "limbs.cuh"

namespace fk {

// ---------------------------------------------------------------- moduli
struct FpDesc {
    static constexpr int N = 12;
    static constexpr uint32_t M0 = 0xfffcfffdu;  // -p^-1 mod 2^32
    FK_HD static constexpr uint32_t mod(int i) {
        return i == 0 ? 0xffffaaabu : i == 1 ? 0xb9feffffu : i == 2 ? 0xb153ffffu : i == 3 ? 0x1eabfffeu
             : i == 4 ? 0xf6b0f624u : i == 5 ? 0x6730d2a0u : i == 6 ? 0xf38512bfu : i == 7 ? 0x64774b84u
             : i == 8 ? 0x434bacd7u : i == 9 ? 0x4b1ba7b6u : i == 10 ? 0x397fe69au : 0x1a0111eau;
    }
    // 2^768 mod p (to Montgomery form)
    FK_HD static constexpr uint32_t r2(int i) {
        return i == 0 ? 0x1c341746u : i == 1 ? 0xf4df1f34u : i == 2 ? 0x09d104f1u : i == 3 ? 0x0a76e6a6u
             : i == 4 ? 0x4c95b6d5u : i == 5 ? 0x8de5476cu : i == 6 ? 0x939d83c0u : i == 7 ? 0x67eb88a9u
             : i == 8 ? 0xb519952du : i == 9 ? 0x9a793e85u : i == 10 ? 0x92cae3aau : 0x11988fe5u;
    }
    // 2^384 mod p (Montgomery one)
    FK_HD static constexpr uint32_t one(int i) {
        return i == 0 ? 0x0002fffdu : i == 1 ? 0x76090000u : i == 2 ? 0xc40c0002u : i == 3 ? 0xebf4000bu
             : i == 4 ? 0x53c758bau : i == 5 ? 0x5f489857u : i == 6 ? 0x70525745u : i == 7 ? 0x77ce5853u
             : i == 8 ? 0xa256ec6du : i == 9 ? 0x5c071a97u : i == 10 ? 0xfa80e493u : 0x15f65ec3u;
    }
};

struct FrDesc {
    static constexpr int N = 8;
    static constexpr uint32_t M0 = 0xffffffffu;  // -r^-1 mod 2^32
    FK_HD static constexpr uint32_t mod(int i) {
        return i == 0 ? 0x00000001u : i == 1 ? 0xffffffffu : i == 2 ? 0xfffe5bfeu : i == 3 ? 0x53bda402u
             : i == 4 ? 0x09a1d805u : i == 5 ? 0x3339d808u : i == 6 ? 0x299d7d48u : 0x73eda753u;
    }
    FK_HD static constexpr uint32_t r2(int i) {
        return i == 0 ? 0xf3f29c6du : i == 1 ? 0xc999e990u : i == 2 ? 0x87925c23u : i == 3 ? 0x2b6cedcbu
             : i == 4 ? 0x7254398fu : i == 5 ? 0x05d31496u : i == 6 ? 0x9f59ff11u : 0x0748d9d9u;
    }
    FK_HD static constexpr uint32_t one(int i) {
        return i == 0 ? 0xfffffffeu : i == 1 ? 0x00000001u : i == 2 ? 0x00034802u : i == 3 ? 0x5884b7fau
             : i == 4 ? 0xecbc4ff5u : i == 5 ? 0x998c4fefu : i == 6 ? 0xacc5056fu : 0x1824b159u;
    }
};

template <class F>
struct Elem {
    uint32_t w[F::N];
};
using Fp = Elem<FpDesc>;
using Fr = Elem<FrDesc>;

// ---------------------------------------------------------------- carry chains
// Each chain is one inline-PTX statement in device code (chains.inc, written
// by gen_chains.py): the carry flag CC.CF never has to survive from one asm
// statement to the next.  Host builds run the portable stand-ins below, which
// compute the same words.
template <class F> FK_D void ptx_add(uint32_t *r, const uint32_t *a, const uint32_t *b);
template <class F> FK_D uint32_t ptx_sub(uint32_t *r, const uint32_t *a, const uint32_t *b);
template <class F> FK_D uint32_t ptx_sub_mod(uint32_t *r, const uint32_t *t);
template <class F> FK_D void ptx_row_even(uint32_t *e, const uint32_t *a, uint32_t b);
template <class F> FK_D void ptx_row_odd(uint32_t *o, const uint32_t *a, uint32_t b);
template <class F> FK_D void ptx_red_even(uint32_t *e, uint32_t m);
template <class F> FK_D void ptx_red_odd(uint32_t *o, uint32_t m, uint32_t &e0, uint32_t x);
template <class F> FK_D void ptx_final(uint32_t *t, const uint32_t *e, const uint32_t *o);
template <class F, int I> FK_D void ptx_sqrow_even(uint32_t *e, const uint32_t *v, uint32_t b);
template <class F, int I> FK_D void ptx_sqrow_odd(uint32_t *o, const uint32_t *v, uint32_t b);
#if defined(__CUDA_ARCH__)
#include "chains.inc"
#endif

// r = a + b; the carry out of the top word is dropped (callers keep sums < 2^(32N))
template <class F>
FK_HD void ch_add(uint32_t *r, const uint32_t *a, const uint32_t *b) {
#if defined(__CUDA_ARCH__)
    ptx_add<F>(r, a, b);
#else
    uint64_t c = 0;
    for (int i = 0; i < F::N; i++) { c += (uint64_t)a[i] + b[i]; r[i] = (uint32_t)c; c >>= 32; }
#endif
}

// r = a - b; returns all ones when a < b, else 0
template <class F>
FK_HD uint32_t ch_sub(uint32_t *r, const uint32_t *a, const uint32_t *b) {
#if defined(__CUDA_ARCH__)
    return ptx_sub<F>(r, a, b);
#else
    uint64_t br = 0;
    for (int i = 0; i < F::N; i++) { uint64_t d = (uint64_t)a[i] - b[i] - br; r[i] = (uint32_t)d; br = d >> 63; }
    return br ? 0xffffffffu : 0u;
#endif
}

// r = t - modulus; returns all ones when t < modulus, else 0
template <class F>
FK_HD uint32_t ch_sub_mod(uint32_t *r, const uint32_t *t) {
#if defined(__CUDA_ARCH__)
    return ptx_sub_mod<F>(r, t);
#else
    uint32_t m[F::N];
    for (int i = 0; i < F::N; i++) m[i] = F::mod(i);
    return ch_sub<F>(r, t, m);
#endif
}

// e[0..N-1] += a[j]*b for even j (lo word at j, hi word at j+1); e[N] = carry out
template <class F>
FK_HD void ch_row_even(uint32_t *e, const uint32_t *a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    ptx_row_even<F>(e, a, b);
#else
    uint64_t c = 0;
    for (int w = 0; w < F::N; w++) {
        c += (uint64_t)e[w] + ((w & 1) ? mul_hi(a[w - 1], b) : mul_lo(a[w], b));
        e[w] = (uint32_t)c;
        c >>= 32;
    }
    e[F::N] = (uint32_t)c;
#endif
}

// o[0..N-1] (words 1..N) += a[j]*b for odd j (lo word at o[j-1], hi word at
// o[j]); o[N-1] is written, not read
template <class F>
FK_HD void ch_row_odd(uint32_t *o, const uint32_t *a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    ptx_row_odd<F>(o, a, b);
#else
    uint64_t s = 0;
    for (int w = 0; w < F::N - 1; w++) {
        s += (uint64_t)o[w] + ((w & 1) ? mul_hi(a[w], b) : mul_lo(a[w + 1], b));
        o[w] = (uint32_t)s;
        s >>= 32;
    }
    o[F::N - 1] = (uint32_t)(s + mul_hi(a[F::N - 1], b));
#endif
}

// e[0..N-1] += m*mod[j] for even j; e[N] += carry out
template <class F>
FK_HD void ch_red_even(uint32_t *e, uint32_t m) {
#if defined(__CUDA_ARCH__)
    ptx_red_even<F>(e, m);
#else
    uint64_t c = 0;
    for (int w = 0; w < F::N; w++) {
        c += (uint64_t)e[w] + ((w & 1) ? mul_hi(m, F::mod(w - 1)) : mul_lo(m, F::mod(w)));
        e[w] = (uint32_t)c;
        c >>= 32;
    }
    e[F::N] += (uint32_t)c;
#endif
}

// e0 += x (word 0), its carry and m*mod[j] for odd j into o[0..N-1] (words 1..N)
template <class F>
FK_HD void ch_red_odd(uint32_t *o, uint32_t m, uint32_t &e0, uint32_t x) {
#if defined(__CUDA_ARCH__)
    ptx_red_odd<F>(o, m, e0, x);
#else
    uint64_t c = (uint64_t)e0 + x;
    e0 = (uint32_t)c;
    c >>= 32;
    for (int w = 0; w < F::N - 1; w++) {
        c += (uint64_t)o[w] + ((w & 1) ? mul_hi(m, F::mod(w)) : mul_lo(m, F::mod(w + 1)));
        o[w] = (uint32_t)c;
        c >>= 32;
    }
    o[F::N - 1] += (uint32_t)c + mul_hi(m, F::mod(F::N - 1));
#endif
}

// t[k] = e[k+1] + o[k], k < N
template <class F>
FK_HD void ch_final(uint32_t *t, const uint32_t *e, const uint32_t *o) {
#if defined(__CUDA_ARCH__)
    ptx_final<F>(t, e, o);
#else
    uint64_t c = 0;
    for (int k = 0; k < F::N; k++) {
        c += (uint64_t)e[k + 1] + o[k];
        t[k] = (uint32_t)c;
        c >>= 32;
    }
#endif
}

// squaring row I >= 1, one parity P of j >= I: P = 0: e[j], e[j+1] += v[j] * b,
// the carry out into e[N]; P = 1: o[j-1], o[j] += v[j] * b, o[N-1] written, not
// read
template <class F, int I, int P>
FK_HD void ch_sqrow(uint32_t *acc, const uint32_t *v, uint32_t b) {
#if defined(__CUDA_ARCH__)
    if (P == 0) ptx_sqrow_even<F, I>(acc, v, b);
    else ptx_sqrow_odd<F, I>(acc, v, b);
#else
    constexpr int N = F::N;
    const int j0 = (I % 2 == P) ? I : I + 1;
    if (j0 >= N) return;  // no product of this parity
    uint64_t c = 0;
    for (int j = j0; j < N; j += 2) {
        const int w = j - P;
        c += (uint64_t)acc[w] + mul_lo(v[j], b);
        acc[w] = (uint32_t)c;
        c >>= 32;
        c += (P == 1 && j == N - 1 ? 0 : (uint64_t)acc[w + 1]) + mul_hi(v[j], b);
        acc[w + 1] = (uint32_t)c;
        c >>= 32;
    }
    if (P == 0) acc[N] = (uint32_t)c;
#endif
}

// ---------------------------------------------------------------- helpers
template <class F>
FK_HD void f_set_zero(Elem<F> &r) {
#pragma unroll
    for (int i = 0; i < F::N; i++) r.w[i] = 0;
}

template <class F>
FK_HD void f_set_one(Elem<F> &r) {  // Montgomery one
#pragma unroll
    for (int i = 0; i < F::N; i++) r.w[i] = F::one(i);
}

template <class F>
FK_HD bool f_is_zero(const Elem<F> &a) {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < F::N; i++) o |= a.w[i];
    return o == 0;
}

template <class F>
FK_HD bool f_eq(const Elem<F> &a, const Elem<F> &b) {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < F::N; i++) o |= a.w[i] ^ b.w[i];
    return o == 0;
}

// r = t - mod if t >= mod else t   (t < 2*mod < 2^(32N))
template <class F>
FK_HD void f_reduce_once(uint32_t r[F::N], const uint32_t t[F::N]) {
    constexpr int N = F::N;
    uint32_t s[N];
    const uint32_t borrow = ch_sub_mod<F>(s, t);  // 0xffffffff if t < mod
#pragma unroll
    for (int i = 0; i < N; i++) r[i] = (t[i] & borrow) | (s[i] & ~borrow);
}

// ---------------------------------------------------------------- Montgomery product
// One reduction step and the shift by one word.  Word 0 is e[0] + x, x the word
// left over from the step before; m makes it vanish.  The shift keeps each
// accumulator's lo/hi pairs on even register positions: the odd words 1..N
// become the even words 0..N-1, and e[2..N] the odd words (a lo/hi pair is one
// 64-bit multiply-add only on an even register; shifting both accumulators in
// place puts every second step's pairs on odd ones).  B200, 2^22 elements x 64
// dependent products: Fp product 26.2 -> 30.2 G/s (98 % of half the IMAD peak),
// square 31.3 -> 38.0 G/s; Fr 56.5 -> 56.9 G/s.
template <class F>
FK_HD void f_reduce_step(uint32_t *e, uint32_t *o, uint32_t &x, bool last) {
    constexpr int N = F::N;
    const uint32_t m = mul_lo(e[0] + x, F::M0);
    ch_red_odd<F>(o, m, e[0], x);
    ch_red_even<F>(e, m);
    if (last) return;
    uint32_t t[N + 1];
#pragma unroll
    for (int k = 0; k <= N; k++) t[k] = e[k];
#pragma unroll
    for (int k = 0; k < N; k++) e[k] = o[k];
    e[N] = 0;
#pragma unroll
    for (int k = 0; k < N - 1; k++) o[k] = t[k + 2];
    o[N - 1] = 0;
    x = t[1];
}

template <class F>
FK_HD void f_mul(Elem<F> &r, const Elem<F> &A, const Elem<F> &B) {
    constexpr int N = F::N;
    const uint32_t *a = A.w;
    uint32_t e[N + 1], o[N];
    uint32_t x = 0;

    // word 0 of b: plain products, no chains needed
    {
        const uint32_t bi = B.w[0];
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            e[j] = mul_lo(a[j], bi);
            e[j + 1] = mul_hi(a[j], bi);
            o[j] = mul_lo(a[j + 1], bi);
            o[j + 1] = mul_hi(a[j + 1], bi);
        }
        e[N] = 0;
    }

#pragma unroll
    for (int i = 0; i < N; i++) {
        if (i > 0) {
            ch_row_even<F>(e, a, B.w[i]);
            ch_row_odd<F>(o, a, B.w[i]);
        }
        f_reduce_step<F>(e, o, x, i == N - 1);
    }
    // the upper words, then one conditional subtraction
    uint32_t t[N];
    ch_final<F>(t, e, o);
    f_reduce_once<F>(r.w, t);
}

// ---------------------------------------------------------------- Montgomery square
// The same word-serial CIOS as f_mul, with the products of word i of A
// restricted to words j >= i (78 of 144 limb products for Fp, 36 of 64 for
// Fr): row i adds a_i * V_i, V_i = a_i 2^(32 i) + 2 sum_{j > i} a_j 2^(32 j),
// whose words are a_i, a_{i+1} << 1 and then the words of 2A (the top bit of
// a_i belongs to row i's own a_i, not to 2A's word i + 1).  Sum over i:
// sum a_i^2 2^(64 i) + 2 sum_{i<j} a_i a_j 2^(32(i+j)) = A^2.  Bounds: V_i <= 2A,
// so A < 2^(32N - 2) keeps every partial value where f_mul's do (A canonical:
// A < m), except the top word of the odd half, which holds hi(2 a_{N-1} a_i) +
// hi(m mod_{N-1}) and stays below 2^32 only for a modulus whose top word is
// below 2^30 (Fp: 0x1a0111ea; Fr's 0x73eda753 is not, so Fr squares are
// products).
template <class F, int I>
FK_HD void f_sqr_rows(uint32_t *e, uint32_t *o, uint32_t &x, const uint32_t *a, const uint32_t *a2) {
    constexpr int N = F::N;
    if constexpr (I > 0) {
        uint32_t v[N];
#pragma unroll
        for (int j = 0; j < N; j++) v[j] = j == I ? a[I] : j == I + 1 ? a[I + 1] << 1 : a2[j];
        ch_sqrow<F, I, 0>(e, v, a[I]);
        ch_sqrow<F, I, 1>(o, v, a[I]);
    }
    f_reduce_step<F>(e, o, x, I == N - 1);
    if constexpr (I < N - 1) f_sqr_rows<F, I + 1>(e, o, x, a, a2);
}

template <class F>
FK_HD void f_sqr(Elem<F> &r, const Elem<F> &A) {
    constexpr int N = F::N;
    if constexpr (F::mod(N - 1) >= (1u << 30)) {
        f_mul<F>(r, A, A);
    } else {
        const uint32_t *a = A.w;
        uint32_t a2[N];  // the words of 2A
        a2[0] = a[0] << 1;
#pragma unroll
        for (int j = 1; j < N; j++) a2[j] = (a[j] << 1) | (a[j - 1] >> 31);
        uint32_t e[N + 1], o[N];
        uint32_t x = 0;
        {
            // row 0: V_0 = (a_0, a_1 << 1, 2A's words 2..N-1), plain products
            const uint32_t b = a[0];
#pragma unroll
            for (int j = 0; j < N; j += 2) {
                const uint32_t v0 = j == 0 ? a[0] : a2[j], v1 = j == 0 ? a[1] << 1 : a2[j + 1];
                e[j] = mul_lo(v0, b);
                e[j + 1] = mul_hi(v0, b);
                o[j] = mul_lo(v1, b);
                o[j + 1] = mul_hi(v1, b);
            }
            e[N] = 0;
        }
        f_sqr_rows<F, 0>(e, o, x, a, a2);
        uint32_t t[N];
        ch_final<F>(t, e, o);
        f_reduce_once<F>(r.w, t);
    }
}

template <class F>
FK_HD void f_add(Elem<F> &r, const Elem<F> &a, const Elem<F> &b) {
    uint32_t t[F::N];
    ch_add<F>(t, a.w, b.w);
    f_reduce_once<F>(r.w, t);
}

template <class F>
FK_HD void f_sub(Elem<F> &r, const Elem<F> &a, const Elem<F> &b) {
    constexpr int N = F::N;
    uint32_t t[N], m[N];
    const uint32_t borrow = ch_sub<F>(t, a.w, b.w);
#pragma unroll
    for (int i = 0; i < N; i++) m[i] = F::mod(i) & borrow;
    ch_add<F>(r.w, t, m);
}

template <class F>
FK_HD void f_neg(Elem<F> &r, const Elem<F> &a) {
    Elem<F> z;
    f_set_zero(z);
    f_sub<F>(r, z, a);
}

template <class F>
FK_HD void f_dbl(Elem<F> &r, const Elem<F> &a) { f_add<F>(r, a, a); }

// r = 12 a  (3b for b = 4)
template <class F>
FK_HD void f_mul12(Elem<F> &r, const Elem<F> &a) {
    Elem<F> t;
    f_add<F>(t, a, a);
    f_add<F>(t, t, a);
    f_add<F>(t, t, t);
    f_add<F>(r, t, t);
}

template <class F>
FK_HD void f_cmov(Elem<F> &r, const Elem<F> &a, bool cond) {
    const uint32_t m = cond ? 0xffffffffu : 0u;
#pragma unroll
    for (int i = 0; i < F::N; i++) r.w[i] = (a.w[i] & m) | (r.w[i] & ~m);
}

// standard form (any value < 2^(32N)) -> Montgomery form, canonical.  The
// reduced constant R^2 mod m goes in the first (multiplicand) slot: f_mul's
// accumulator bound needs that operand below ~2^(32N - 2), while the second
// operand, scanned word by word, may be any 32N-bit value.
template <class F>
FK_HD void f_to_mont(Elem<F> &r, const Elem<F> &a) {
    Elem<F> r2;
#pragma unroll
    for (int i = 0; i < F::N; i++) r2.w[i] = F::r2(i);
    f_mul<F>(r, r2, a);
}

// Montgomery form -> canonical standard form
template <class F>
FK_HD void f_from_mont(Elem<F> &r, const Elem<F> &a) {
    Elem<F> one;
    f_set_zero(one);
    one.w[0] = 1;
    f_mul<F>(r, a, one);
}

// canonical reduction of any standard-form value < 2^(32N)
template <class F>
FK_HD void f_canon(Elem<F> &r, const Elem<F> &a) {
    Elem<F> t;
    f_to_mont<F>(t, a);
    f_from_mont<F>(r, t);
}

// r = a^e for a little-endian exponent of `nw` 32-bit words (Montgomery domain)
template <class F>
FK_HD void f_pow(Elem<F> &r, const Elem<F> &a, const uint32_t *e, int nw) {
    Elem<F> acc;
    f_set_one(acc);
    for (int i = 32 * nw - 1; i >= 0; i--) {
        f_sqr<F>(acc, acc);
        if ((e[i >> 5] >> (i & 31)) & 1) f_mul<F>(acc, acc, a);
    }
    r = acc;
}

// inverse by Fermat's little theorem, a^(m-2); inv(0) = 0
template <class F>
FK_HD void f_inv_pow(Elem<F> &r, const Elem<F> &a) {
    uint32_t e[F::N];
    uint64_t br = 2;
#pragma unroll
    for (int i = 0; i < F::N; i++) {
        const uint64_t d = (uint64_t)F::mod(i) - br;
        e[i] = (uint32_t)d;
        br = d >> 63;
    }
    f_pow<F>(r, a, e, F::N);
}

// Fp inverse by division steps (Bernstein and Yang, "Fast constant-time gcd
// computation and modular inversion", 2019): 30 steps at a time on the low
// words give a 2 x 2 matrix, which then updates f, g (the gcd pair, starting
// at p and a) and d, e (f = d a / c, g = e a / c mod p throughout, starting
// at 0 and c) by exact divisions by 2^30.  Numbers are 13 signed limbs of 30
// bits.  c = R^2 makes the result a^-1 R for a Montgomery-form input a R.
// Theorem 11.2 of the paper: g = 0 after (49 * 381 + 57) / 17 = 1101 steps, 37
// rounds; the loop ends as soon as g is 0 (25 rounds on average).  |d| and |e|
// grow by at most p / 2 a round and fit.  About 20,000 instructions against
// 320,000 for a^(p-2) (381 squares and ~190 products): one inverse per point
// of an output costs less than sharing a slow one did.
struct Limbs30 {
    int32_t v[13];
};
FK_HD int32_t l30_word(const uint32_t *w, int i) {  // bits 30 i .. 30 i + 29 of 12 words
    const int bit = 30 * i, k = bit >> 5, s = bit & 31;
    uint64_t x = w[k];
    if (k + 1 < 12) x |= (uint64_t)w[k + 1] << 32;
    return (int32_t)((uint32_t)(x >> s) & 0x3fffffffu);
}
FK_HD void l30_matrix(int32_t &delta, uint32_t f, uint32_t g, int32_t t[4]) {
    int32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 1
    for (int i = 0; i < 30; i++) {
        const bool odd = g & 1, swap = odd && delta > 0;
        const uint32_t f0 = f, g0 = g;
        const int32_t u0 = u, v0 = v, q0 = q, r0 = r;
        f = swap ? g0 : f0;
        u = swap ? q0 : u0;
        v = swap ? r0 : v0;
        g = odd ? g0 + (swap ? 0u - f0 : f0) : g0;
        q = odd ? q0 + (swap ? -u0 : u0) : q0;
        r = odd ? r0 + (swap ? -v0 : v0) : r0;
        delta = (swap ? -delta : delta) + 1;
        g >>= 1;
        u = (int32_t)((uint32_t)u << 1);
        v = (int32_t)((uint32_t)v << 1);
    }
    t[0] = u, t[1] = v, t[2] = q, t[3] = r;
}
FK_HD void fp_inv_steps(Elem<FpDesc> &res, const Elem<FpDesc> &a) {
    constexpr int32_t M = 0x3fffffff;
    Limbs30 f, g, d, e, p;
    uint32_t pw[12], cw[12];
#pragma unroll
    for (int i = 0; i < 12; i++) pw[i] = FpDesc::mod(i), cw[i] = FpDesc::r2(i);
#pragma unroll
    for (int i = 0; i < 13; i++) {
        p.v[i] = f.v[i] = l30_word(pw, i);
        g.v[i] = l30_word(a.w, i);
        d.v[i] = 0;
        e.v[i] = l30_word(cw, i);
    }
    int32_t delta = 1;
#pragma unroll 1
    for (int round = 0; round < 37; round++) {
        int32_t t[4];
        // the low 30 bits decide 30 steps
        l30_matrix(delta, (uint32_t)f.v[0] | ((uint32_t)f.v[1] << 30), (uint32_t)g.v[0] | ((uint32_t)g.v[1] << 30), t);
        const int64_t u = t[0], v = t[1], q = t[2], r = t[3];
        int64_t cf = u * f.v[0] + v * g.v[0], cg = q * f.v[0] + r * g.v[0];
        cf >>= 30;
        cg >>= 30;
        int64_t cd = u * d.v[0] + v * e.v[0], ce = q * d.v[0] + r * e.v[0];
        // the multiples of p (centred) that make the low 30 bits vanish
        int32_t md = (int32_t)(((uint32_t)cd * FpDesc::M0) << 2) >> 2, me = (int32_t)(((uint32_t)ce * FpDesc::M0) << 2) >> 2;
        cd = (cd + (int64_t)md * p.v[0]) >> 30;
        ce = (ce + (int64_t)me * p.v[0]) >> 30;
        int32_t any = 0;
#pragma unroll
        for (int i = 1; i < 13; i++) {
            cf += u * f.v[i] + v * g.v[i];
            cg += q * f.v[i] + r * g.v[i];
            cd += u * d.v[i] + v * e.v[i] + (int64_t)md * p.v[i];
            ce += q * d.v[i] + r * e.v[i] + (int64_t)me * p.v[i];
            f.v[i - 1] = (int32_t)cf & M;
            g.v[i - 1] = (int32_t)cg & M;
            d.v[i - 1] = (int32_t)cd & M;
            e.v[i - 1] = (int32_t)ce & M;
            any |= g.v[i - 1];
            cf >>= 30, cg >>= 30, cd >>= 30, ce >>= 30;
        }
        f.v[12] = (int32_t)cf, g.v[12] = (int32_t)cg, d.v[12] = (int32_t)cd, e.v[12] = (int32_t)ce;
        if ((any | g.v[12]) == 0) break;
    }
    // f = +-1 (or a = 0: f = +-p, d = 0 mod p): the inverse is f d, brought into [0, p)
    int32_t neg = f.v[12] >> 31;
#pragma unroll 1
    for (int k = 0; k < 96; k++) {
        int64_t c = 0;
        Limbs30 s;
#pragma unroll
        for (int i = 0; i < 13; i++) {
            // first -d where f < 0, then d + p while negative, d - p while that is not negative
            c += k == 0 ? (neg ? -(int64_t)d.v[i] : (int64_t)d.v[i]) : (int64_t)d.v[i] + (d.v[12] < 0 ? p.v[i] : -p.v[i]);
            s.v[i] = i < 12 ? (int32_t)c & M : (int32_t)c;
            c >>= 30;
        }
        const bool done = k > 0 && d.v[12] >= 0 && s.v[12] < 0;  // 0 <= d < p
        if (done) break;
        d = s;
    }
#pragma unroll
    for (int i = 0; i < 12; i++) {
        const int bit = 32 * i, k = bit / 30, sft = bit % 30;
        uint64_t x = (uint64_t)(uint32_t)d.v[k] >> sft;
        x |= (uint64_t)(uint32_t)d.v[k + 1] << (30 - sft);
        if (k + 2 < 13) x |= (uint64_t)(uint32_t)d.v[k + 2] << (60 - sft);
        res.w[i] = (uint32_t)x;
    }
}
template <class F>
FK_HD void f_inv(Elem<F> &r, const Elem<F> &a) {
    if constexpr (F::N == 12) fp_inv_steps(r, a);
    else f_inv_pow<F>(r, a);
}

}  // namespace fk
