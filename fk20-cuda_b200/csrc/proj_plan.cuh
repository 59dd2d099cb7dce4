// proj_plan.cuh -- h_fft = P hext_fft as additions and one layer of
// fixed-scalar products (host side; kernels_proj.cu runs the plans).
//
// The pipeline's last half -- inverse G1 FFT of size m, upper half set to
// infinity, forward FFT (fk20_hext_fft2h_fft.cu:27-60) -- is one linear map,
// y_k = sum_c x_c p(k - c) with p(d) = (1/m) sum_{j < m/2} w^(j d):
// p(0) = 1/2, p(d) = 0 for even d != 0, p(d) = (2/m) / (1 - w^d) for odd d.
// With H = m/2, x'_t = x[-2t - 1] for the even outputs and x'_t = x[-2t] for
// the odd ones (indices mod m), both are the same Hankel map,
//   y[2k + inst] = x[2k + inst] / 2 + sum_t h_(k + t) x'_t,   h_t = p(2t + 1),
// of length H and cyclic in t, so every row is two instances of one map.
//
// A fixed-scalar product of a point costs about 1,300 Fp products and an
// addition 12, so the map is done as a bilinear algorithm with few products:
// E^T diag(beta) E, E made of additions, negations, the endomorphism phi
// ([lambda], one Fp product) and a few doublings, beta constants mod r.
// X^H - 1 splits into X - 1, X + 1, X^2 + 1, X^4 + 1, ... by additions; a
// negacyclic product of length n = m q is a polynomial product in X over
// R_q = Z[z]/(z^q + 1) with X^m = z (Nussbaumer), taken at points that cost no
// product: 0, infinity, powers of z (rotations of the q coefficients), their
// phi images (z has order 2q; with the cube roots of unity 1, lambda,
// lambda^2 there are 6q such points) and, for the length-8 leaf over the
// scalars, the sixth roots of unity +-lambda^j, twice those, and 1/2 (Toom-Cook).
// The transposed map E^T is the same additions run backwards.  For a fixed
// kernel the interpolation falls on the constants: beta solves the dual
// Vandermonde system of the points.
//
// Scalar products per instance: 865 for m = 512, 400 for 256, 175 for 128 --
// 1,730 / 800 / 350 a row, against 3,586 / 1,538 / 642 twiddle products in the
// two FFTs -- and they are independent of each other: one product deep instead
// of 2 log m - 2, which is what bounds a small batch.
#pragma once
#include <algorithm>
#include <array>
#include <map>
#include <tuple>
#include <vector>

#include "proj_task.cuh"
#include "scalar_prog.cuh"

namespace fk {

// a run of consecutive tasks with no dependency among them
struct ProjLevel {
    int first, count, phase;  // phase 0: before the products, 1: products, 2: after
};

struct ProjPlan {
    int slots = 0, muls = 0;
    std::vector<ProjTask> tasks;
    std::vector<ProjLevel> levels;
    std::vector<uint32_t> out;                                // output k: slot | neg << 16 | phi << 17
    std::vector<std::array<uint64_t, 4>> scalars;             // the products' constants (standard form)
    double lin_products[3] = {0, 0, 0};                       // Fp products of a phase's additions and doublings
};

namespace host {

// ---------------------------------------------------------------- Fr on the host
// The Montgomery product in 64-bit words.  A plan of 512 points takes some 550,000
// products, and the 32-bit form, written for the GPU, 0.3 us each on a host core: the
// first hext_fft -> h_fft of a process waited 0.29 s for its plan, now 0.06, its first
// transform of 512 points 0.16 and 0.09 s.
inline Fr operator*(const Fr &a, const Fr &b) {
    using u128 = unsigned __int128;
    const auto word = [](const uint32_t *w, int i) { return (uint64_t)w[2 * i] | (uint64_t)w[2 * i + 1] << 32; };
    constexpr auto mod = [](int i) { return (uint64_t)FrDesc::mod(2 * i) | (uint64_t)FrDesc::mod(2 * i + 1) << 32; };
    constexpr uint64_t m[4] = {mod(0), mod(1), mod(2), mod(3)};
    constexpr uint64_t inv = [](uint64_t m0) {  // 1 / m mod 2^64, by Newton's iteration: 1, 2, 4, .. 64 bits
        uint64_t v = 1;
        for (int k = 0; k < 6; k++) v *= 2 - m0 * v;
        return v;
    }(m[0]);
    uint64_t t[5] = {0, 0, 0, 0, 0};
    for (int i = 0; i < 4; i++) {
        const uint64_t bi = word(b.w, i);
        u128 c = 0;
        for (int j = 0; j < 4; j++) {
            c += (u128)word(a.w, j) * bi + t[j];
            t[j] = (uint64_t)c;
            c >>= 64;
        }
        c += t[4];
        t[4] = (uint64_t)c;  // t < 2^256 + 2^319 (a, m < 2^255): five words hold it, and q m too
        const uint64_t q = 0 - t[0] * inv;
        c = (u128)q * m[0] + t[0];
        c >>= 64;
        for (int j = 1; j < 4; j++) {
            c += (u128)q * m[j] + t[j];
            t[j - 1] = (uint64_t)c;
            c >>= 64;
        }
        c += t[4];
        t[3] = (uint64_t)c;
        t[4] = (uint64_t)(c >> 64);
    }
    Fr s, r;
    for (int i = 0; i < 4; i++) s.w[2 * i] = (uint32_t)t[i], s.w[2 * i + 1] = (uint32_t)(t[i] >> 32);
    f_reduce_once<FrDesc>(r.w, s.w);  // t < 2 m < 2^256
    return r;
}
inline Fr fr_mont(const Fr &a) {  // standard form -> Montgomery form
    Fr r2;
    for (int i = 0; i < 8; i++) r2.w[i] = FrDesc::r2(i);
    return a * r2;
}
inline Fr fr_from_u64(uint64_t v) {
    Fr t;
    f_set_zero(t);
    t.w[0] = (uint32_t)v;
    t.w[1] = (uint32_t)(v >> 32);
    return v ? fr_mont(t) : t;
}
inline Fr operator+(const Fr &a, const Fr &b) { Fr r; f_add(r, a, b); return r; }
inline Fr operator-(const Fr &a, const Fr &b) { Fr r; f_sub(r, a, b); return r; }
inline Fr fr_pow(const Fr &a, unsigned e) {
    Fr r;
    f_set_one(r);
    Fr q = a;
    for (; e; e >>= 1) {
        if (e & 1) r = r * q;
        if (e > 1) q = q * q;
    }
    return r;
}
inline Fr fr_pow(const Fr &a, const uint32_t e[8]) {
    Fr v;
    f_set_one(v);
    for (int i = 254; i >= 0; i--) {
        v = v * v;
        if ((e[i >> 5] >> (i & 31)) & 1) v = v * a;
    }
    return v;
}
inline Fr fr_inv(const Fr &a) {  // a^(r - 2)
    uint32_t e[8];
    for (int i = 0; i < 8; i++) e[i] = FrDesc::mod(i);
    e[0] -= 2, e[1] -= 1;  // r's low word is 1
    return fr_pow(a, e);
}
inline int log2_of(int v) {
    int l = 0;
    while ((1 << l) < v) l++;
    return l;
}
inline Fr fr_lambda() {  // z^2 - 1
    Fr t;
    f_set_zero(t);
    t.w[0] = 0xffffffffu, t.w[1] = 0, t.w[2] = 0x0001a402u, t.w[3] = 0xac45a401u;
    return fr_mont(t);
}
inline Fr fr_root(int log_order) {  // 5^((r-1) / 2^log_order)
    uint32_t e[8];
    for (int i = 0; i < 8; i++) e[i] = FrDesc::mod(i);
    e[0] -= 1;
    for (int k = 0; k < log_order; k++)
        for (int i = 0; i < 8; i++) e[i] = (e[i] >> 1) | (i < 7 ? e[i + 1] << 31 : 0);
    return fr_pow(fr_from_u64(5), e);
}

// ---------------------------------------------------------------- evaluation points
// num / den with num = +-z^e lambda^j 2^k or 0, den = 1, 2 or 0
struct ProjPoint {
    int zero = 0, neg = 0, e = 0, j = 0, k = 0;  // num
    int den_k = 0, inf = 0;                      // den = 2^den_k, or 0
    Fr num(const Fr &rho) const {
        if (zero) return fr_from_u64(0);
        Fr v = fr_pow(rho, (unsigned)e) * fr_pow(fr_lambda(), (unsigned)j) * fr_from_u64(1ull << k);
        return neg ? fr_from_u64(0) - v : v;
    }
    Fr den() const { return inf ? fr_from_u64(0) : fr_from_u64(1ull << den_k); }
};

// rows s, columns l: num_s^l den_s^(L - l), inverted (square)
inline std::vector<Fr> dual_vandermonde_inverse(const std::vector<ProjPoint> &pts, const Fr &rho) {
    const int n = (int)pts.size();
    // M[l][s] g[s] = h[l]
    std::vector<Fr> M((size_t)n * 2 * n, fr_from_u64(0));
    for (int s = 0; s < n; s++) {
        const Fr num = pts[s].num(rho), den = pts[s].den();
        Fr a = fr_from_u64(1), b = a;
        for (int l = 0; l < n; l++) M[(size_t)l * 2 * n + s] = a, a = a * num;
        for (int l = n - 1; l >= 0; l--) M[(size_t)l * 2 * n + s] = M[(size_t)l * 2 * n + s] * b, b = b * den;
    }
    const Fr one = fr_from_u64(1);
    for (int l = 0; l < n; l++) M[(size_t)l * 2 * n + n + l] = one;
    for (int c = 0; c < n; c++) {
        int p = c;
        while (f_is_zero(M[(size_t)p * 2 * n + c])) p++;  // invertible: distinct points
        if (p != c)
            for (int k = 0; k < 2 * n; k++) std::swap(M[(size_t)p * 2 * n + k], M[(size_t)c * 2 * n + k]);
        const Fr iv = fr_inv(M[(size_t)c * 2 * n + c]);
        for (int k = 0; k < 2 * n; k++) M[(size_t)c * 2 * n + k] = M[(size_t)c * 2 * n + k] * iv;
        for (int l = 0; l < n; l++) {
            if (l == c || f_is_zero(M[(size_t)l * 2 * n + c])) continue;
            const Fr f = M[(size_t)l * 2 * n + c];
            for (int k = c; k < 2 * n; k++) M[(size_t)l * 2 * n + k] = M[(size_t)l * 2 * n + k] - f * M[(size_t)c * 2 * n + k];
        }
    }
    std::vector<Fr> inv((size_t)n * n);
    for (int s = 0; s < n; s++)
        for (int l = 0; l < n; l++) inv[(size_t)s * n + l] = M[(size_t)s * 2 * n + n + l];
    return inv;
}

// ---------------------------------------------------------------- the graph
struct ProjRef {  // (-1)^neg phi^phi times a node (v < 0: zero)
    int v = -1;
    int neg = 0, phi = 0;
};

class ProjBuilder {
public:
    struct Node {
        int op;      // ProjOp, or -1: input
        ProjRef a, b;
        int sh = 0, c = 0;  // SHL: doublings; MUL: constant index
        int cross0 = -1, cross1 = -1;  // OUT: nodes read from the other instance
    };
    std::vector<Node> nodes;
    std::vector<Fr> consts;

    int input() { nodes.push_back(Node{-1, {}, {}}); return (int)nodes.size() - 1; }
    static ProjRef times(ProjRef r, int neg, int phi) {
        r.neg ^= neg & 1;
        r.phi = (r.phi + phi) % 3;
        return r;
    }
    ProjRef add(ProjRef a, ProjRef b) {
        if (a.v < 0) return b;
        if (b.v < 0) return a;
        if (a.v > b.v) std::swap(a, b);
        const ProjRef rel = times(b, a.neg, 3 - a.phi);
        const auto key = std::make_tuple(a.v, rel.v, rel.neg, rel.phi);
        auto it = adds_.find(key);
        int id;
        if (it == adds_.end()) {
            Node n{PROJ_LIN, ProjRef{a.v, 0, 0}, rel};
            nodes.push_back(n);
            id = (int)nodes.size() - 1;
            adds_[key] = id;
        } else {
            id = it->second;
        }
        return ProjRef{id, a.neg, a.phi};
    }
    ProjRef sub(ProjRef a, ProjRef b) { return add(a, times(b, 1, 0)); }
    ProjRef shl(ProjRef a, int k) {
        if (a.v < 0 || k == 0) return a;
        const auto key = std::make_pair(a.v, k);
        auto it = shls_.find(key);
        int id;
        if (it == shls_.end()) {
            Node n{PROJ_SHL, ProjRef{a.v, 0, 0}, {}};
            n.sh = k;
            nodes.push_back(n);
            id = (int)nodes.size() - 1;
            shls_[key] = id;
        } else {
            id = it->second;
        }
        return ProjRef{id, a.neg, a.phi};
    }

    ProjRef mul(int v, const Fr &c) {
        Node n{PROJ_MUL, ProjRef{v, 0, 0}, {}};
        n.c = (int)consts.size();
        consts.push_back(c);
        nodes.push_back(n);
        return ProjRef{(int)nodes.size() - 1, 0, 0};
    }
    ProjRef mul(const ProjRef &a, const Fr &c) {
        const ProjRef r = mul(a.v, c);
        return ProjRef{r.v, a.neg, a.phi};
    }

    // the negacyclic product of length n: evaluation of x (n refs) appended to
    // `out`, and the constants of the functional h (n values, h_(t+n) = -h_t)
    // appended to `beta`, product by product in the same order
    void negacyclic(int n, const std::vector<ProjRef> &x, const std::vector<Fr> &h, std::vector<ProjRef> &out,
                    std::vector<Fr> &beta) {
        if (n == 1) {
            out.push_back(x[0]);
            beta.push_back(h[0]);
            return;
        }
        const int q = n <= 8 ? 1 : 8, m = n / q;  // X^m = z, z^q = -1
        std::vector<ProjPoint> pts;
        std::vector<std::vector<ProjRef>> val;  // the polynomial's values: q refs each
        std::vector<std::vector<ProjRef>> poly(m);
        for (int i = 0; i < m; i++)
            for (int j = 0; j < q; j++) poly[i].push_back(x[i + m * j]);
        evaluate(m, q, poly, pts, val);
        const int np = (int)pts.size();  // >= 2m - 1
        // h_l on R_q: h_l[j] = h at index l + m j, extended by h_(t+n) = -h_t; in the basis of
        // the q embeddings z -> rho (rho^q = -1), then the dual Vandermonde system per embedding
        const int lq = q == 8 ? 3 : 0;
        const Fr z0 = fr_root(lq + 1);  // order 2q
        std::vector<std::vector<Fr>> g(np, std::vector<Fr>(q, fr_from_u64(0)));
        const Fr iq = fr_inv(fr_from_u64((uint64_t)q));
        for (int e = 0; e < q; e++) {
            const Fr rho = fr_pow(z0, (unsigned)(2 * e + 1)), irho = fr_inv(rho);
            std::vector<Fr> &inv = inverses_[std::make_tuple(m, q, e)];
            if (inv.empty()) inv = dual_vandermonde_inverse(pts, rho);
            std::vector<Fr> hl(np, fr_from_u64(0));
            for (int l = 0; l < 2 * m - 1; l++) {
                for (int j = 0; j < q; j++) {
                    const int t = l + m * j;
                    const Fr v = t < n ? h[t] : fr_from_u64(0) - h[t - n];
                    hl[l] = hl[l] + fr_pow(irho, (unsigned)j) * v;
                }
                hl[l] = hl[l] * iq;
            }
            for (int s = 0; s < np; s++) {
                Fr gs = fr_from_u64(0);
                for (int l = 0; l < np; l++) gs = gs + inv[(size_t)s * np + l] * hl[l];
                Fr rj = fr_from_u64(1);
                for (int j = 0; j < q; j++) {
                    g[s][j] = g[s][j] + gs * rj;
                    rj = rj * rho;
                }
            }
        }
        for (int s = 0; s < np; s++) {
            if (q == 1) {
                out.push_back(val[s][0]);
                beta.push_back(g[s][0]);
            } else {
                negacyclic(q, val[s], g[s], out, beta);
            }
        }
    }

private:
    std::map<std::tuple<int, int, int, int>, int> adds_;
    std::map<std::pair<int, int>, int> shls_;
    std::map<std::tuple<int, int, int>, std::vector<Fr>> inverses_;  // of (m, q, embedding)

    using Vec = std::vector<ProjRef>;
    Vec vadd(const Vec &a, const Vec &b) {
        Vec r;
        for (size_t i = 0; i < a.size(); i++) r.push_back(add(a[i], b[i]));
        return r;
    }
    static Vec vtimes(const Vec &a, int neg, int phi) {
        Vec r;
        for (const ProjRef &x : a) r.push_back(times(x, neg, phi));
        return r;
    }
    Vec vsub(const Vec &a, const Vec &b) { return vadd(a, vtimes(b, 1, 0)); }
    // times z^e in R_q
    static Vec rotate(const Vec &a, int e) {
        const int q = (int)a.size();
        e %= 2 * q;
        Vec r(q);
        for (int j = 0; j < q; j++) {
            const int t = j + e;
            r[t % q] = times(a[j], (t / q) & 1, 0);
        }
        return r;
    }
    // F_j = a + phi^j b + phi^(2j) c, j = 0, 1, 2
    void dft3(Vec F[3], const Vec &a, const Vec &b, const Vec &c, bool has_b, bool has_c) {
        if (!has_b || !has_c) {
            for (int j = 0; j < 3; j++)
                F[j] = has_b ? vadd(a, vtimes(b, 0, j)) : has_c ? vadd(a, vtimes(c, 0, 2 * j % 3)) : a;
            return;
        }
        const Vec s = vadd(b, c), v = vsub(b, c), u = vsub(a, c);
        F[0] = vadd(a, s);
        F[1] = vadd(u, vtimes(v, 0, 1));
        F[2] = vadd(u, vtimes(v, 0, 2));
    }
    // values at +-lambda^j of the polynomial folded to six coefficients (missing ones empty)
    void six(const Vec A[6], std::vector<Vec> &val) {
        const auto has = [&](int r) { return !A[r].empty(); };
        Vec ev[3], od[3];
        dft3(ev, A[0], A[4], A[2], has(4), has(2));
        dft3(od, A[3], A[1], A[5], has(1), has(5));
        for (int j = 0; j < 3; j++) {
            val.push_back(vadd(ev[j], od[j]));
            val.push_back(vsub(ev[j], od[j]));
        }
    }
    void point(std::vector<ProjPoint> &pts, int neg, int e, int j, int k = 0) {
        ProjPoint p;
        p.neg = neg, p.e = e, p.j = j, p.k = k;
        pts.push_back(p);
    }
    // sixteen values at lambda^tau z^k (q = 8: z has order 16) of up to 16 coefficients, k in natural order
    std::vector<Vec> fft16(const std::vector<Vec> &poly, int tau) {
        std::vector<Vec> a(16);
        for (size_t i = 0; i < poly.size(); i++) a[i] = vtimes(poly[i], 0, (int)(tau * i % 3));
        // decimation in frequency: block of size len at base b, twiddles (z^(16/len))^i
        for (int len = 16; len > 1; len /= 2)
            for (int b = 0; b < 16; b += len)
                for (int i = 0; i < len / 2; i++) {
                    Vec &u = a[b + i], &v = a[b + i + len / 2];
                    Vec s, d;
                    if (v.empty()) s = u, d = u;
                    else s = vadd(u, v), d = vsub(u, v);
                    u = s;
                    v = rotate(d, i * (16 / len));
                }
        std::vector<Vec> out(16);
        for (int k = 0; k < 16; k++) {
            int r = 0;
            for (int b = 0; b < 4; b++) r |= ((k >> b) & 1) << (3 - b);
            out[k] = a[r];
        }
        return out;
    }
    // points and values of a polynomial of m coefficients over R_q, at least 2m - 1 points
    void evaluate(int m, int q, const std::vector<Vec> &c, std::vector<ProjPoint> &pts, std::vector<Vec> &val) {
        ProjPoint zero, inf;
        zero.zero = 1;
        inf.inf = 1;
        pts.push_back(zero);
        val.push_back(c[0]);
        if (m == 4 && q == 1) {  // 0 and the six units
            Vec A[6] = {c[0], c[1], c[2], c[3], {}, {}};
            six(A, val);
            for (int j = 0; j < 3; j++) point(pts, 0, 0, j), point(pts, 1, 0, j);
            return;
        }
        pts.push_back(inf);
        val.push_back(c[m - 1]);
        if (m == 2) {  // 0, infinity, 1
            point(pts, 0, 0, 0);
            val.push_back(vadd(c[0], c[1]));
        } else if (m == 4) {  // and +-1, +-z^4 (square roots of -1), lambda
            const Vec e0 = vadd(c[0], c[2]), e1 = vsub(c[0], c[2]), o0 = vadd(c[1], c[3]), o1 = vsub(c[1], c[3]);
            const Vec t = rotate(o1, 4);
            point(pts, 0, 0, 0), val.push_back(vadd(e0, o0));
            point(pts, 1, 0, 0), val.push_back(vsub(e0, o0));
            point(pts, 0, 4, 0), val.push_back(vadd(e1, t));
            point(pts, 1, 4, 0), val.push_back(vsub(e1, t));
            point(pts, 0, 0, 1);
            val.push_back(vadd(vadd(c[0], c[3]), vadd(vtimes(c[1], 0, 1), vtimes(c[2], 0, 2))));
        } else if (m == 8 && q == 1) {  // and the units, twice the units, 1/2
            Vec A[6] = {vadd(c[0], c[6]), vadd(c[1], c[7]), c[2], c[3], c[4], c[5]};
            six(A, val);
            for (int j = 0; j < 3; j++) point(pts, 0, 0, j), point(pts, 1, 0, j);
            const auto sh = [&](const Vec &v, int k) { return Vec{shl(v[0], k)}; };
            Vec B[6] = {vadd(c[0], sh(c[6], 6)), sh(vadd(c[1], sh(c[7], 6)), 1), sh(c[2], 2), sh(c[3], 3), sh(c[4], 4),
                        sh(c[5], 5)};
            six(B, val);
            for (int j = 0; j < 3; j++) point(pts, 0, 0, j, 1), point(pts, 1, 0, j, 1);
            // sum of 2^(7-i) c_i, as a tree: 7 doublings and 3 additions deep instead of 7 and 7
            const auto up = [&](const Vec &a, const Vec &b, int k) { return vadd(b, sh(a, k)); };
            const Vec t = up(up(up(c[0], c[1], 1), up(c[2], c[3], 1), 2), up(up(c[4], c[5], 1), up(c[6], c[7], 1), 2), 4);
            ProjPoint half;
            half.den_k = 1;
            pts.push_back(half);
            val.push_back(t);
        } else {  // m = 8 or 16 over R_8: powers of z and, for 16, their phi images
            std::vector<Vec> f = fft16(c, 0);
            const int k0 = m == 8 ? 13 : 16;
            for (int k = 0; k < k0; k++) point(pts, 0, k, 0), val.push_back(f[k]);
            if (m == 16) {
                f = fft16(c, 1);
                for (int k = 0; k < 13; k++) point(pts, 0, k, 1), val.push_back(f[k]);
            }
        }
    }
};

// Tasks, levels and slots of the graph's nodes that the outputs need; nodes 0 ..
// inputs - 1 are the inputs, in slots of the same number.
inline ProjPlan finish_plan(const ProjBuilder &g, int inputs, const std::vector<ProjRef> &outs) {
    // ---- live nodes, pairs (a + b, a - b), doublings folded into their only user
    const int N = (int)g.nodes.size();
    std::vector<char> live(N, 0);
    for (const ProjRef &k : outs) live[k.v] = 1;
    for (int v = N - 1; v >= 0; v--) {
        if (!live[v]) continue;
        const auto &n = g.nodes[v];
        for (int r : {n.a.v, n.b.v, n.cross0, n.cross1})
            if (r >= 0) live[r] = 1;
    }
    std::vector<int> uses(N, 0);
    for (int v = 0; v < N; v++)
        if (live[v])
            for (int r : {g.nodes[v].a.v, g.nodes[v].b.v, g.nodes[v].cross0, g.nodes[v].cross1})
                if (r >= 0) uses[r]++;
    std::map<std::tuple<int, int, int>, std::array<int, 2>> pairs;
    for (int v = 0; v < N; v++)
        if (live[v] && g.nodes[v].op == PROJ_LIN) {
            const auto &n = g.nodes[v];
            auto &p = pairs.emplace(std::make_tuple(n.a.v, n.b.v, n.b.phi), std::array<int, 2>{-1, -1}).first->second;
            p[n.b.neg] = v;
        }
    std::vector<char> folded(N, 0);
    for (auto &q : pairs) {
        const int b = std::get<1>(q.first), own = (q.second[0] >= 0 ? 1 : 0) + (q.second[1] >= 0 ? 1 : 0);
        folded[b] |= g.nodes[b].op == PROJ_SHL && uses[b] == own;
    }
    struct Task {
        ProjOp op;
        int a = -1, b = -1, b2 = -1, sh = 0, phi = 0, neg = 0, d0 = -1, d1 = -1, c = 0, level = 0;
    };
    std::vector<Task> tasks;
    std::vector<int> owner(N, -1);  // the task that writes a node
    for (int v = 0; v < N; v++) {
        if (!live[v]) continue;
        const auto &n = g.nodes[v];
        Task t;
        if (n.op < 0) continue;
        t.op = (ProjOp)n.op;
        t.a = n.a.v;
        t.d0 = v;
        if (n.op == PROJ_LIN) {
            const auto &p = pairs[std::make_tuple(n.a.v, n.b.v, n.b.phi)];
            t.b = n.b.v, t.phi = n.b.phi, t.neg = n.b.neg;
            if (p[0] >= 0 && p[1] >= 0) {
                if (owner[p[0]] >= 0 || owner[p[1]] >= 0) continue;  // written by the pair's first node
                t.neg = 0, t.d0 = p[0], t.d1 = p[1];
            }
            // a doubled second operand that nothing else reads: doubled here
            // (a pair's two nodes count as its two uses)
            if (folded[t.b]) t.sh = g.nodes[t.b].sh, t.b = g.nodes[t.b].a.v;
        } else if (n.op == PROJ_SHL) {
            t.sh = n.sh;
            if (folded[v]) continue;  // into its only user
        } else if (n.op == PROJ_MUL) {
            t.c = n.c;
        } else {
            t.b = n.cross0, t.b2 = n.cross1, t.neg = n.a.neg, t.phi = n.a.phi;
        }
        owner[t.d0] = (int)tasks.size();
        if (t.d1 >= 0) owner[t.d1] = (int)tasks.size();
        tasks.push_back(t);
    }
    // ---- levels: before the products, the products, after them.  A task with
    // no product above it and no other use for it than the output (the diagonal
    // term) still belongs to the first phase.
    std::vector<int> phase(tasks.size(), 0);
    const int NT = (int)tasks.size();
    std::vector<int> order;
    {   // nodes were created in dependency order except that a pair is written by its first node:
        // process by repeated relaxation (levels only grow)
        bool again = true;
        while (again) {
            again = false;
            for (int i = 0; i < NT; i++) {
                int lv = 0, ph = tasks[i].op == PROJ_MUL ? 1 : 0;
                for (int r : {tasks[i].a, tasks[i].b, tasks[i].b2}) {
                    if (r < 0 || owner[r] < 0) continue;
                    const int o = owner[r];
                    const int po = phase[o] == 1 ? 2 : phase[o];
                    if (po > ph) ph = po;
                    lv = std::max(lv, tasks[o].level + 1);
                }
                if (lv != tasks[i].level || ph != phase[i]) tasks[i].level = lv, phase[i] = ph, again = true;
            }
        }
        for (int i = 0; i < NT; i++) order.push_back(i);
        std::stable_sort(order.begin(), order.end(), [&](int i, int j) {
            return std::make_tuple(phase[i], phase[i] == 1 ? 0 : tasks[i].level) <
                   std::make_tuple(phase[j], phase[j] == 1 ? 0 : tasks[j].level);
        });
    }
    // ---- slots.  A task may write over a value all of whose readers are above
    // it in the dependency graph (or are the task itself): they have finished
    // when it runs.  Tasks of the last phase wait until every product of their
    // group is done, so the products and all that is above one of them count too;
    // a task of the first phase that feeds no product (a diagonal term's doublings)
    // does not.
    ProjPlan P;
    std::vector<int> slot(N, -1), ver(N, 0), pos(NT, 0);
    std::vector<std::vector<int>> readers(N);
    for (int k = 0; k < NT; k++) pos[order[k]] = k;
    for (int i : order)
        for (int r : {tasks[i].a, tasks[i].b, tasks[i].b2})
            if (r >= 0) readers[r].push_back(i);
    const size_t words = (size_t)(NT + 63) / 64;
    std::vector<std::vector<uint64_t>> above(NT);
    const auto under = [&](int i, int o) {  // task i runs after task o
        for (size_t k = 0; k < words; k++) above[i][k] |= above[o][k];
        above[i][(size_t)o / 64] |= 1ull << (o % 64);
    };
    std::vector<uint64_t> produced(words, 0);  // the products and the tasks above them (complete before the last phase)
    const auto finished = [&](int r, int i) {  // reader r has finished when task i runs
        const auto has = [&](const std::vector<uint64_t> &set) { return ((set[(size_t)r / 64] >> (r % 64)) & 1) != 0; };
        return r == i || has(above[i]) || (phase[i] == 2 && has(produced));
    };
    struct Dead { int slot, ver; std::vector<int> readers; };
    std::vector<Dead> dead;
    std::vector<std::pair<uint16_t, uint8_t>> wrote(NT);  // slot and version of each task's d0
    std::vector<int> left(N);  // readers not yet placed
    for (int v = 0; v < N; v++) left[v] = (int)readers[v].size();
    for (const ProjRef &k : outs) left[k.v]++;  // outputs are never written over
    for (int t = 0; t < inputs; t++) slot[t] = t;
    int next = inputs;
    int last_level = -1, last_phase = -1;
    for (int i : order) {
        const Task &t = tasks[i];
        ProjTask o{};
        above[i].assign(words, 0);
        for (int r : {t.a, t.b, t.b2})
            if (r >= 0 && owner[r] >= 0) under(i, owner[r]);
        o.op = t.op, o.sh = (uint8_t)t.sh, o.phi = (uint8_t)t.phi, o.neg = (uint8_t)t.neg;
        o.a = (uint16_t)slot[t.a], o.va = (uint8_t)ver[t.a];
        o.b = o.b2 = o.d1 = PROJ_NONE;
        if (t.b >= 0) o.b = (uint16_t)slot[t.b], o.vb = (uint8_t)ver[t.b];
        if (t.b2 >= 0) o.b2 = (uint16_t)slot[t.b2], o.vb2 = (uint8_t)ver[t.b2];
        // the other instance's values (OUT) are never written over
        for (int r : {t.a, t.op == PROJ_OUT ? -1 : t.b})
            if (r >= 0 && --left[r] == 0) dead.push_back(Dead{slot[r], ver[r], readers[r]});
        const auto place = [&](int v, uint16_t &d, uint8_t &wv) {
            int pick = -1;
            for (int k = (int)dead.size() - 1; k >= 0 && pick < 0; k--) {
                bool ok = true;
                for (int r : dead[k].readers) ok &= finished(r, i);
                if (ok) pick = k;
            }
            // or one whose only other reader is a task of an earlier level: this
            // task then waits for that reader's result as well (b2)
            for (int k = (int)dead.size() - 1; k >= 0 && pick < 0 && t.op != PROJ_OUT && o.b2 == PROJ_NONE; k--) {
                int other = -1, n = 0;
                for (int r : dead[k].readers)
                    if (!finished(r, i)) other = r, n++;
                if (n != 1 || phase[i] == 1 || phase[other] != phase[i] || tasks[other].level >= t.level) continue;
                pick = k;
                o.b2 = wrote[other].first, o.vb2 = wrote[other].second;
                under(i, other);
            }
            if (pick >= 0) {
                slot[v] = dead[pick].slot, ver[v] = dead[pick].ver + 1;
                dead.erase(dead.begin() + pick);
            } else {
                slot[v] = next++, ver[v] = 1;
            }
            d = (uint16_t)slot[v], wv = (uint8_t)ver[v];
        };
        place(t.d0, o.d0, o.w0);
        wrote[i] = {o.d0, o.w0};
        if (t.d1 >= 0) place(t.d1, o.d1, o.w1);
        if (phase[i] == 1) {
            for (size_t k = 0; k < words; k++) produced[k] |= above[i][k];
            produced[(size_t)i / 64] |= 1ull << (i % 64);
        }
        if (t.op == PROJ_MUL) {
            o.prog = (uint16_t)P.scalars.size();
            Fr s;
            f_from_mont(s, g.consts[t.c]);
            std::array<uint64_t, 4> k;
            for (int q = 0; q < 4; q++) k[q] = (uint64_t)s.w[2 * q] | ((uint64_t)s.w[2 * q + 1] << 32);
            P.scalars.push_back(k);
        } else {
            P.lin_products[phase[i]] += 8.0 * t.sh + (t.phi ? 1 : 0) + (t.op == PROJ_SHL ? 0 : t.d1 >= 0 ? 18 : 12);
        }
        const int ph = phase[i], lv = ph == 1 ? 0 : t.level;
        o.phase = (uint8_t)ph;
        if (ph != last_phase || lv != last_level) P.levels.push_back(ProjLevel{(int)P.tasks.size(), 0, ph});
        last_phase = ph, last_level = lv;
        P.levels.back().count++;
        P.tasks.push_back(o);
    }
    P.slots = next;
    P.muls = (int)P.scalars.size();
    for (const ProjRef &k : outs) P.out.push_back((uint32_t)slot[k.v] | (uint32_t)k.neg << 16 | (uint32_t)k.phi << 17);
    return P;
}

// the sum of v, as a tree
inline ProjRef total(ProjBuilder &g, std::vector<ProjRef> v) {
    while (v.size() > 1) {
        std::vector<ProjRef> nx;
        for (size_t i = 0; i + 1 < v.size(); i += 2) nx.push_back(g.add(v[i], v[i + 1]));
        if (v.size() & 1) nx.push_back(v.back());
        v = nx;
    }
    return v.empty() ? ProjRef{} : v[0];
}

// The projection of FFT size 2^log_m.  The inputs are hext_fft / 2^log_m (the bases of
// the pipeline's tables carry the inverse FFT's factor) or, `half`, hext_fft itself.
inline ProjPlan build_proj_plan(int log_m, bool half) {
    const int m = 1 << log_m, H = m / 2;
    ProjBuilder g;
    std::vector<ProjRef> x(H);
    for (int t = 0; t < H; t++) x[t] = ProjRef{g.input(), 0, 0};
    // h_t = p(2t + 1), times m when the inputs are divided by m
    std::vector<Fr> h(H);
    const Fr w = fr_root(log_m), one = fr_from_u64(1);
    for (int t = 0; t < H; t++) {
        h[t] = fr_from_u64(2) * fr_inv(one - fr_pow(w, (unsigned)(2 * t + 1)));
        if (half) h[t] = h[t] * fr_inv(fr_from_u64((uint64_t)m));
    }
    const Fr ihalf = fr_inv(fr_from_u64(2));
    std::vector<ProjRef> ev;
    std::vector<Fr> beta;
    for (int n = H / 2; n >= 1; n /= 2) {  // X^(2n) - 1 = (X^n + 1)(X^n - 1)
        std::vector<ProjRef> xn(n), xc(n);
        std::vector<Fr> hn(n), hc(n);
        for (int t = 0; t < n; t++) {
            xc[t] = g.add(x[t], x[t + n]);
            xn[t] = g.sub(x[t], x[t + n]);
            hc[t] = ihalf * (h[t] + h[t + n]);
            hn[t] = ihalf * (h[t] - h[t + n]);
        }
        g.negacyclic(n, xn, hn, ev, beta);
        x = xc;
        h = hc;
    }
    ev.push_back(x[0]);
    beta.push_back(h[0]);
    const int npre = (int)g.nodes.size();

    // products: [beta coef^2] of the node itself, so that the transposed map starts at the node
    std::map<int, Fr> prod;
    const Fr lam = fr_lambda();
    for (size_t s = 0; s < ev.size(); s++) {
        const Fr c = beta[s] * fr_pow(lam, (unsigned)(2 * ev[s].phi % 3));
        auto it = prod.find(ev[s].v);
        if (it == prod.end()) prod[ev[s].v] = c;
        else it->second = it->second + c;
    }
    std::vector<std::vector<ProjRef>> adj(npre);
    std::vector<int> diag(H);
    if (half)  // the diagonal term's x / 2: products too
        for (int t = 0; t < H; t++)
            diag[t] = g.mul(t, ihalf).v;
    else
        for (int t = 0; t < H; t++) diag[t] = g.shl(ProjRef{t, 0, 0}, log_m - 1).v;
    for (auto &p : prod) {
        if (f_is_zero(p.second)) continue;
        adj[p.first].push_back(g.mul(p.first, p.second));
    }
    // the transposed additions, in reverse order
    for (int v = npre - 1; v >= H; v--) {
        const ProjRef s = total(g, adj[v]);
        if (s.v < 0) continue;
        const ProjBuilder::Node n = g.nodes[v];
        if (n.op == PROJ_LIN) {
            adj[n.a.v].push_back(s);
            adj[n.b.v].push_back(ProjBuilder::times(s, n.b.neg, n.b.phi));
        } else {  // SHL
            adj[n.a.v].push_back(g.shl(s, n.sh));
        }
    }
    std::vector<ProjRef> outs(H);
    for (int k = 0; k < H; k++) {
        const ProjRef c = total(g, adj[k]);
        ProjBuilder::Node n{PROJ_OUT, c, {}};
        n.cross0 = diag[(H - k) & (H - 1)];   // instance 0 reads x[2k] from instance 1
        n.cross1 = diag[H - 1 - k];           // instance 1 reads x[2k + 1] from instance 0
        g.nodes.push_back(n);
        outs[k] = ProjRef{(int)g.nodes.size() - 1, 0, 0};
    }
    return finish_plan(g, H, outs);
}


// ---------------------------------------------------------------- whole transforms
// The negacyclic Hankel map of length n with functional h on x: its graph is
// built apart, copied in, and run backwards to the n outputs.
inline std::vector<ProjRef> hankel(ProjBuilder &g, const std::vector<ProjRef> &x, const std::vector<Fr> &h) {
    const int n = (int)x.size();
    ProjBuilder e;
    std::vector<ProjRef> in(n), out;
    std::vector<Fr> beta;
    for (int t = 0; t < n; t++) in[t] = ProjRef{e.input(), 0, 0};
    e.negacyclic(n, in, h, out, beta);
    const auto coef = [](ProjRef r, ProjRef by) { return ProjBuilder::times(r, by.neg, by.phi); };
    std::vector<ProjRef> at(e.nodes.size());
    for (size_t v = 0; v < e.nodes.size(); v++) {
        const auto &nd = e.nodes[v];
        if (nd.op < 0) at[v] = x[v];
        else if (nd.op == PROJ_LIN) at[v] = g.add(at[nd.a.v], coef(at[nd.b.v], nd.b));
        else at[v] = g.shl(at[nd.a.v], nd.sh);
    }
    std::vector<std::vector<ProjRef>> adj(e.nodes.size());
    const Fr lam = fr_lambda();
    for (size_t s = 0; s < out.size(); s++) {
        if (f_is_zero(beta[s])) continue;
        const ProjRef v = at[out[s].v];  // the node's place in g, with its own coefficient
        Fr c = beta[s] * fr_pow(lam, (unsigned)((2 * out[s].phi + v.phi) % 3));
        if (v.neg) c = fr_from_u64(0) - c;
        adj[out[s].v].push_back(g.mul(v.v, c));
    }
    for (int v = (int)e.nodes.size() - 1; v >= n; v--) {
        const ProjRef s = total(g, adj[v]);
        if (s.v < 0) continue;
        const auto &nd = e.nodes[v];
        if (nd.op == PROJ_LIN) {
            adj[nd.a.v].push_back(s);
            adj[nd.b.v].push_back(coef(s, nd.b));
        } else {
            adj[nd.a.v].push_back(g.shl(s, nd.sh));
        }
    }
    std::vector<ProjRef> y(n);
    for (int t = 0; t < n; t++) y[t] = total(g, adj[t]);
    return y;
}

// sum_{j < d/2} u_j w_d^(sign j k) times `scale` at the odd k < d, in order
// (d = 2 u.size()).  Even j give the same sums of half the length.  Odd j and
// odd k are +-5^b mod d, and 5^(d/8) = 1 + d/2 turns the sign: with the sums
// and differences over +-, two negacyclic Hankel maps of length d/8.
inline std::vector<ProjRef> odd_sums(ProjBuilder &g, const std::vector<ProjRef> &u, const Fr &w, const Fr &scale,
                                     bool scaled) {
    const int half = (int)u.size(), d = 2 * half;
    if (d == 2) return {scaled ? g.mul(u[0], scale) : u[0]};
    std::vector<ProjRef> ue;
    for (int j = 0; j < half; j += 2) ue.push_back(u[j]);
    const std::vector<ProjRef> E = odd_sums(g, ue, w * w, scale, scaled);
    std::vector<ProjRef> O(half / 2);  // odd k < d/2
    if (d == 4) {
        O[0] = g.mul(u[1], w * scale);
    } else {
        const int n = d / 8;
        std::vector<ProjRef> v[2], p(n), q(n);
        std::vector<Fr> hp(n), hm(n);
        std::vector<int> res(n);
        const Fr ih = fr_inv(fr_from_u64(2)) * scale, iw = fr_inv(w);
        const auto pick = [&](int r) { return r < half ? u[r] : ProjBuilder::times(u[r - half], 1, 0); };
        for (int b = 0, r = 1; b < n; b++, r = r * 5 % d) {
            res[b] = r;
            const ProjRef x = pick(r), y = pick(d - r);
            p[b] = g.add(x, y), q[b] = g.sub(x, y);
            const Fr c0 = fr_pow(w, (unsigned)r), c1 = fr_pow(iw, (unsigned)r);
            hp[b] = ih * (c0 + c1), hm[b] = ih * (c0 - c1);
        }
        const std::vector<ProjRef> A = hankel(g, p, hp), B = hankel(g, q, hm);
        for (int b = 0; b < n; b++) {
            const ProjRef y[2] = {g.add(A[b], B[b]), g.sub(A[b], B[b])};
            const int k[2] = {res[b], d - res[b]};
            for (int a = 0; a < 2; a++) {  // k + d/2 has the opposite sign
                if (k[a] < half) O[k[a] / 2] = y[a];
                else O[(k[a] - half) / 2] = ProjBuilder::times(y[a], 1, 0);
            }
        }
    }
    std::vector<ProjRef> out(half);
    for (int i = 0; i < half / 2; i++) out[i] = g.add(E[i], O[i]), out[i + half / 2] = g.sub(E[i], O[i]);
    return out;
}

// The transform of 2^log_m points, or its inverse with the factor 1/m: input j
// in slot j, output k in out[k].  1,388 products at m = 512 (the inverse 1,398,
// its factor on every product and on the few values that meet none), one deep;
// radix 2 takes 1,793 (2,305), nine (ten) deep.  B200: 32 inverse transforms of
// 512 points by stages 12.6 ms, by plan 4.3.
inline ProjPlan build_dft_plan(int log_m, bool inverse) {
    const int m = 1 << log_m;
    ProjBuilder g;
    std::vector<ProjRef> x(m), out(m);
    for (int t = 0; t < m; t++) x[t] = ProjRef{g.input(), 0, 0};
    const Fr scale = inverse ? fr_inv(fr_from_u64((uint64_t)m)) : fr_from_u64(1);
    for (int d = m, step = 1; d > 1; d /= 2, step *= 2) {  // outputs k = step * odd
        const Fr w = inverse ? fr_inv(fr_root(log2_of(d))) : fr_root(log2_of(d));
        std::vector<ProjRef> s, t;
        for (int j = 0; j < d / 2; j++) s.push_back(g.add(x[j], x[j + d / 2])), t.push_back(g.sub(x[j], x[j + d / 2]));
        const std::vector<ProjRef> y = odd_sums(g, t, w, scale, inverse);
        for (int i = 0; i < d / 2; i++) out[step * (2 * i + 1)] = y[i];
        x = s;
    }
    out[0] = inverse ? g.mul(x[0], scale) : x[0];
    return finish_plan(g, m, out);
}

// The launch order over segments of plans p[k] with G[k] groups: phase by
// phase; within the first and the last phase chunks of groups, level by level
// (the levels of a chunk are wide enough to fill the chip, and a chunk's first
// level of the last phase finds its products long done); false if the runs do
// not fit.
inline bool build_proj_runs(ProjRuns &r, const ProjPlan *const *p, const int *G, int nseg) {
    for (int chunk = 8; chunk <= 1 << 16; chunk *= 2) {
        r.n = 0;
        unsigned at = 0;
        bool fits = true;
        const auto put = [&](int k, int first, int count, int g0, int gn) {
            if (r.n == MAX_PROJ_RUNS) { fits = false; return; }
            r.run[r.n++] = ProjRun{at, (unsigned short)first, (unsigned short)k, (unsigned short)g0, (unsigned short)gn};
            at += (unsigned)count * (unsigned)gn;
        };
        int gmax = 0;
        size_t lmax = 0;
        for (int k = 0; k < nseg; k++) gmax = std::max(gmax, G[k]), lmax = std::max(lmax, p[k]->levels.size());
        for (int phase = 0; phase < 3; phase++)
            for (int c = 0; c * chunk < gmax; c++)
                for (size_t l = 0; l < lmax; l++)
                    for (int k = 0; k < nseg; k++) {
                        if (l >= p[k]->levels.size() || p[k]->levels[l].phase != phase) continue;
                        const int g0 = c * chunk, gn = std::min(chunk, G[k] - g0);
                        if (gn > 0) put(k, p[k]->levels[l].first, p[k]->levels[l].count, g0, gn);
                    }
        r.total = at;
        if (fits) return true;
    }
    return false;
}

}  // namespace host
}  // namespace fk
