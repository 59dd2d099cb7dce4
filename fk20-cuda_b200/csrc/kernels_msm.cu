// kernels_msm.cu -- fixed-base MSM of the FK20 pipeline.
//
// hext_fft[row][c] = sum_{i<16} tc_fft[row][i][c] * X_i[c]  (fk20_msm.cu:23-66;
// FK20Py/fk20_single.py:73-76).  The bases X_i[c] are fixed per setup, so each
// has a table of its signed-digit multiples: entry (w, e) = (e+1) 2^(cb w) X,
// e < 2^(cb-1), affine Montgomery (built by kernels_tables.cu).  A 255-bit
// scalar is recoded on the fly into ceil(255/cb) signed digits in
// [-2^(cb-1), 2^(cb-1)] and each nonzero digit costs one mixed addition of a
// gathered 96-byte entry: no doublings at all, against ~255 doublings + ~128
// additions per term in the reference's g1p_mul loop.  The accumulator is in
// XYZZ coordinates (x = X/ZZ, y = Y/ZZZ), whose mixed addition takes 8 M + 2 S
// (the complete projective one 11 M); its exceptional cases -- accumulator at
// infinity, equal or opposite points -- are tested and handled, so every sum
// is exact.  The result goes back to homogeneous projective coordinates.
// The Fp product and square out of line (one shared copy each): the mixed
// addition's ten inlined products overflowed the instruction cache.
#ifndef FK_MSM_OUTLINE
#define FK_MSM_OUTLINE 1
#endif
#if FK_MSM_OUTLINE
#define FK_FP_MUL_OUTLINE 1
#endif
#include <algorithm>
#include <cmath>

#include "../../include/fk20_b200.h"
#include "check.cuh"
#include "consts.cuh"
#include "launch.h"
#include "layout.cuh"

#ifndef FK_MSM_MINB
#define FK_MSM_MINB 1
#endif
// largest block size the launcher may use; the launch bounds cap registers
// at 65536 / (FK_MSM_MAX_THREADS * FK_MSM_MINB): 384 gives 168 registers, so
// three 128-thread blocks (12 warps) fit an SM (64-, 128- and 256-thread
// blocks launch as they are)
#ifndef FK_MSM_MAX_THREADS
#define FK_MSM_MAX_THREADS 384
#endif
constexpr int MSM_MAX_THREADS = FK_MSM_MAX_THREADS;

namespace fk {

cudaError_t upload_consts_msm() { return upload_module_consts(); }

FK_CHECK_WORD(msm)

// XYZZ point: x = X / ZZ, y = Y / ZZZ (ZZ^3 = ZZZ^2); ZZ = 0 is infinity
struct G1Z {
    Fp x, y, zz, zzz;
};
FK_D void g1z_set_inf(G1Z &a) {
    f_set_one(a.x);
    f_set_one(a.y);
    f_set_zero(a.zz);
    f_set_zero(a.zzz);
}
// a = 2 (qx, qy), affine q not infinity (y != 0 in the prime-order group):
// U = 2y, V = U^2, W = U V, S = x V, M = 3 x^2, X = M^2 - 2S,
// Y = M (S - X) - W y, ZZ = V, ZZZ = W
FK_D void g1z_dbl_affine(G1Z &a, const Fp &qx, const Fp &qy) {
    Fp u, v, w, sv, m, t;
    f_add(u, qy, qy);
    fp_sqr(v, u);
    fp_mul(w, u, v);
    fp_mul(sv, qx, v);
    fp_sqr(m, qx);
    f_add(t, m, m);
    f_add(m, t, m);
    fp_sqr(t, m);
    f_sub(t, t, sv);
    f_sub(a.x, t, sv);
    f_sub(t, sv, a.x);
    fp_mul(t, m, t);
    fp_mul(u, w, qy);
    f_sub(a.y, t, u);
    a.zz = v;
    a.zzz = w;
}
// a += (qx, qy), affine q not infinity (madd-2008-s: U2 = qx ZZ, S2 = qy ZZZ,
// P = U2 - X, R = S2 - Y, X3 = R^2 - P^3 - 2 X P^2, Y3 = R (X P^2 - X3) - Y P^3,
// ZZ3 = ZZ P^2, ZZZ3 = ZZZ P^3)
FK_D void g1z_madd(G1Z &a, const Fp &qx, const Fp &qy) {
    if (f_is_zero(a.zz)) {
        a.x = qx;
        a.y = qy;
        f_set_one(a.zz);
        f_set_one(a.zzz);
        return;
    }
    Fp u2, s2, p, r, pp, ppp, q, t;
    fp_mul(u2, qx, a.zz);
    fp_mul(s2, qy, a.zzz);
    f_sub(p, u2, a.x);
    f_sub(r, s2, a.y);
    if (f_is_zero(p)) {
        if (f_is_zero(r)) g1z_dbl_affine(a, qx, qy);  // a = q
        else g1z_set_inf(a);                          // a = -q
        return;
    }
    fp_sqr(pp, p);
    fp_mul(ppp, p, pp);
    fp_mul(q, a.x, pp);
    fp_sqr(t, r);
    f_sub(t, t, ppp);
    f_sub(t, t, q);
    f_sub(a.x, t, q);
    f_sub(t, q, a.x);
    fp_mul(t, r, t);
    fp_mul(s2, a.y, ppp);
    f_sub(a.y, t, s2);
    fp_mul(a.zz, a.zz, pp);
    fp_mul(a.zzz, a.zzz, ppp);
}
// homogeneous projective (X ZZZ, Y ZZ, ZZ ZZZ); infinity as (0, 1, 0)
FK_D void g1z_to_proj(G1P &r, const G1Z &a) {
    if (f_is_zero(a.zz)) {
        g1_set_inf(r);
        return;
    }
    fp_mul(r.x, a.x, a.zzz);
    fp_mul(r.y, a.y, a.zz);
    fp_mul(r.z, a.zz, a.zzz);
}

// acc += the table entry at ent (96 bytes, affine Montgomery), or its negative;
// an entry (0, 0) encodes a base at infinity (not on the curve)
FK_D void msm_add_entry(G1Z &acc, const uint4 *__restrict__ ent, bool neg) {
    Fp x, y;
    const uint4 q0 = ent[0], q1 = ent[1], q2 = ent[2], q3 = ent[3], q4 = ent[4], q5 = ent[5];
    x.w[0] = q0.x; x.w[1] = q0.y; x.w[2] = q0.z; x.w[3] = q0.w;
    x.w[4] = q1.x; x.w[5] = q1.y; x.w[6] = q1.z; x.w[7] = q1.w;
    x.w[8] = q2.x; x.w[9] = q2.y; x.w[10] = q2.z; x.w[11] = q2.w;
    y.w[0] = q3.x; y.w[1] = q3.y; y.w[2] = q3.z; y.w[3] = q3.w;
    y.w[4] = q4.x; y.w[5] = q4.y; y.w[6] = q4.z; y.w[7] = q4.w;
    y.w[8] = q5.x; y.w[9] = q5.y; y.w[10] = q5.z; y.w[11] = q5.w;
    if (f_is_zero(x) && f_is_zero(y)) return;
    if (neg) f_neg(y, y);
    g1z_madd(acc, x, y);
}

// acc += s * X for one base X, whose table `tb` holds (e+1) 2^(cb w) X for
// window w and e < 2^(cb-1): the 255-bit scalar s (9 words, s[8] = 0) is
// recoded into W signed digits in [-2^(cb-1), 2^(cb-1)] on the fly and every
// nonzero digit costs one mixed addition of a gathered 96-byte entry.
// Returns the recoding's final carry: nonzero when s needs more than W
// windows (the tables do not cover it).
FK_D int msm_add_scalar(G1Z &acc, const uint32_t s[9], const uint4 *__restrict__ tb, int W, int cb) {
    const int E = 1 << (cb - 1);
    const uint32_t mask = (1u << cb) - 1u;
    int carry = 0;
    for (int w = 0; w < W; w++) {
        const int bit = w * cb;
        const int wd = bit >> 5, sh = bit & 31;
        uint32_t raw = s[wd] >> sh;
        if (sh + cb > 32) raw |= s[wd + 1] << (32 - sh);
        int d = (int)(raw & mask) + carry;
        carry = d > E;
        if (carry) d -= (1 << cb);
        if (d != 0) {
            const int e = (d < 0 ? -d : d) - 1;
            msm_add_entry(acc, tb + ((size_t)w * E + e) * 6, d < 0);
        }
    }
    return carry;
}

// sum of the lanes that differ in the lane bits off, 2 off, .. 16 (every lane
// gets it)
FK_D void g1_sum_lanes(G1P &p, int off) {
#pragma unroll 1
    for (; off < 32; off <<= 1) {
        G1P q;
#pragma unroll
        for (int k = 0; k < 12; k++) {
            q.x.w[k] = __shfl_xor_sync(0xffffffffu, p.x.w[k], off);
            q.y.w[k] = __shfl_xor_sync(0xffffffffu, p.y.w[k], off);
            q.z.w[k] = __shfl_xor_sync(0xffffffffu, p.z.w[k], off);
        }
        g1_add(p, p, q);
    }
}

// sum of n warps' points (warps w0 .. w0 + n - 1 of the block), in warp w0;
// part holds 36 x 32 words per warp.  Every thread of the block calls it.
FK_D void g1_sum_warps(G1P &p, uint32_t *part, int w0, int n) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const StridedPoint mine{part + w * 36 * 32 + lane, 32};
    if (w != w0) mine.put(p);
    __syncthreads();
    if (w == w0)
        for (int k = 1; k < n; k++) {
            const StridedPoint other{part + (w0 + k) * 36 * 32 + lane, 32};
            g1_add_q(p, p, other, false);
        }
}

// Unit (segment, column c, group g of rows): 2^rl rows on the low lane bits,
// the 32 (base, GLV half) terms of a column shared by the 32 >> rl lane groups
// and args.split warps of the unit; their sums are added by shuffles and
// through shared memory.  Large batches have one warp per unit and a row per
// lane.  Units are numbered segment by segment, g fastest, so the warps of a
// block read the same table column.
__global__ void __launch_bounds__(MSM_MAX_THREADS, FK_MSM_MINB) k_msm(const __grid_constant__ MsmArgs args) {
    extern __shared__ uint32_t part[];
    const unsigned warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    bool on = warp < args.warps;  // uniform over a unit's warps
    int k = 0;
    while (k + 1 < args.nseg && warp >= args.seg[k + 1].warp_start) k++;
    const MsmSeg &a = args.seg[k];
    const int m = 1 << a.log_m;
    const int lane = threadIdx.x & 31;
    const unsigned wl = on ? warp - a.warp_start : 0;
    const unsigned unit = wl / (unsigned)args.split;
    const int sub = (int)(wl % (unsigned)args.split);
    const int g = (int)(unit % (unsigned)a.G), c = (int)(unit / (unsigned)a.G);
    on = on && FK_CHECK(g_check_msm, k < args.nseg && c < m && args.split * (32 >> a.rl) <= 32, FK20_CHECK_MSM_TILE);
    if (!on && args.split == 1) return;
    if (args.test_check && warp == 0 && lane == 0) (void)FK_CHECK(g_check_msm, false, FK20_CHECK_MSM_PLANTED);
    const int row = a.row0 + g * 32 + (lane & ((1 << a.rl) - 1));
    const bool live = on && row < a.rows;
    const int E = 1 << (a.cb - 1);
    // sum_i [s_i] X_i = phi(sum_i [s2_i] X_i) + sum_i [s1_i] X_i with
    // s_i = s1_i + s2_i lambda (the scalar tile holds s1 at uint4 0 and s2 at
    // uint4 1): terms 0..15 are the s2 halves, 16..31 the s1 halves; phi goes on
    // the accumulator ((X, Y, ZZ, ZZZ) -> (beta X, Y, ZZ, ZZZ)) after the last
    // s2 half.
    const int per = 32 / ((32 >> a.rl) * args.split);
    const int q0 = ((lane >> a.rl) * args.split + sub) * per;
    G1Z accz;
    g1z_set_inf(accz);
#pragma unroll 1
    for (int j = 0; j < per && on; j++) {
        const int q = q0 + j, half = q < L_COLS, i = q & (L_COLS - 1);
        uint32_t s[9];
        uint4 v = make_uint4(0, 0, 0, 0);
        if (live) v = a.S[(row >> 5) * a.s_stride + (((size_t)c * L_COLS + i) * SCAL_Q + half) * 32 + (row & 31)];
        s[0] = v.x; s[1] = v.y; s[2] = v.z; s[3] = v.w;
#pragma unroll
        for (int k = 4; k < 9; k++) s[k] = 0;
        const uint4 *tb = a.table + ((size_t)(i * m + c) * a.W) * E * 6;
        const int carry = msm_add_scalar(accz, s, tb, a.W, a.cb);
        (void)FK_CHECK(g_check_msm, carry == 0, FK20_CHECK_MSM_CARRY);
        if (q == L_COLS - 1 || (half && j == per - 1)) {
            Fp beta;
#pragma unroll
            for (int k = 0; k < 12; k++) beta.w[k] = beta_mont(k);
            fp_mul(accz.x, accz.x, beta);
        }
    }
    G1P acc;
    g1z_to_proj(acc, accz);
    g1_sum_lanes(acc, 1 << a.rl);
    if (args.split > 1) g1_sum_warps(acc, part, (threadIdx.x >> 5) - sub, args.split);
    if (!on || sub != 0) return;
    if (args.times_m) {
        for (int t = 0; t < a.log_m; t++) g1_dbl(acc, acc);
    }
    // lanes beyond the rows of the segment get copies of its rows' points
    if (!a.fill && (lane >> a.rl) != 0) return;
    const int to = a.row0 + g * 32 + lane;
    if ((a.row0 & 31) + lane > 31) return;
    if (a.arena.slots == 0) {
        tile_store(a.D + tile_index(to >> 5, m, c), to & 31, acc);
    } else {
        int ga, la;
        if (!proj_lane(a.arena, to, proj_in_inst(c), ga, la)) return;
        tile_store(a.D + proj_tile(a.arena, ga, proj_in_slot(c, a.log_m)), la, acc);
    }
}

// ---------------------------------------------------------------- KZG commitments
// commitment[row] = sum_i poly[row][i] * s_i over fixed-base tables of the
// setup points s_i (commit_to_poly, FK20Py/kzg_proofs.py:159-163).  Pass 1: the
// n W digits (base i, window w) of a row are cut into equal runs; warp c of
// group g sums its run, or with the packed rows of the last group each of its
// 32 >> rl lane groups one, into a partial-sum tile.  A run that starts inside
// a scalar scans the windows below for the recoding's carry.  Pass 2: one block
// per row adds its partials, as a tree.
__global__ void __launch_bounds__(128, 3) k_commit_partial(uint4 *__restrict__ part, const uint64_t *__restrict__ poly,
                                                           const uint4 *__restrict__ table, int rows, int n, int W,
                                                           int cb, const CommitCut cut) {
    const unsigned warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (warp >= (unsigned)cut.tiles()) return;
    const int lane = threadIdx.x & 31;
    const bool last = warp >= (unsigned)(cut.full * cut.P);
    const int g = last ? cut.full : (int)(warp / (unsigned)cut.P);
    const int c = (int)warp - g * cut.P, rl = last ? cut.rl : 5;
    const int row = g * 32 + (lane & ((1 << rl) - 1));
    const bool live = row < rows;
    const int E = 1 << (cb - 1);
    const uint32_t mask = (1u << cb) - 1u;
    const long long ways = (long long)(last ? cut.Pr : cut.P) * (32 >> rl), way = (long long)c * (32 >> rl) + (lane >> rl);
    const long long units = (long long)n * W;
    const int u0 = (int)(way * units / ways), u1 = (int)((way + 1) * units / ways);
    G1Z accz;
    g1z_set_inf(accz);
    uint32_t s[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    int i = u0 / W - 1, w = W, carry = 0;  // the first unit loads its scalar
    int start = u0 - (i + 1) * W;
    for (int u = u0; u < u1; u++) {
        const auto digit = [&](int v) {  // window v's signed digit; the carry moves on
            const int bit = v * cb, wd = bit >> 5, sh = bit & 31;
            uint32_t raw = s[wd] >> sh;
            if (sh + cb > 32) raw |= s[wd + 1] << (32 - sh);
            int d = (int)(raw & mask) + carry;
            carry = d > E;
            return carry ? d - (1 << cb) : d;
        };
        if (w == W) {
            i++;
            w = start;
            start = 0;
            if (live) {
                Fr f;
                fr_from_ref(f, poly + 4 * ((size_t)row * n + i));
#pragma unroll
                for (int k = 0; k < 8; k++) s[k] = f.w[k];
            }
            carry = 0;
            for (int v = 0; v < w; v++) (void)digit(v);
        }
        const int d = digit(w);
        if (d != 0) {
            const int e = (d < 0 ? -d : d) - 1;
            msm_add_entry(accz, table + (((size_t)i * W + w) * E + e) * 6, d < 0);
        }
        w++;
    }
    __syncwarp();
    G1P acc;
    g1z_to_proj(acc, accz);
    g1_sum_lanes(acc, 1 << rl);
    if ((lane >> rl) == 0) tile_store(part + tile_index(0, 0, (int)warp), row & 31, acc);
}

constexpr int REDUCE_THREADS = 128;
__global__ void __launch_bounds__(REDUCE_THREADS) k_commit_reduce(uint64_t *__restrict__ out, const uint4 *__restrict__ part,
                                                                  const CommitCut cut) {
    __shared__ uint32_t sm[(REDUCE_THREADS / 32) * 36 * 32];
    const int row = blockIdx.x, g = row >> 5, lane = row & 31;
    const int P = g < cut.full ? cut.P : cut.Pr;
    G1P acc, q;
    g1_set_inf(acc);
    for (int c = threadIdx.x; c < P; c += REDUCE_THREADS) {
        tile_load(q, part + tile_index(0, 0, g * cut.P + c), lane);
        g1_add(acc, acc, q);
    }
    __syncwarp();
    g1_sum_lanes(acc, 1);
    constexpr int WARPS = REDUCE_THREADS / 32;
    const int warps = (P + 31) / 32;
    g1_sum_warps(acc, sm, 0, warps < WARPS ? warps : WARPS);
    if (threadIdx.x == 0) g1p_to_ref(out + 18 * (size_t)row, acc);
}

// The same for many rows: 2^ll lanes a row, rows on the low lane bits.
__global__ void __launch_bounds__(REDUCE_THREADS) k_commit_reduce_rows(uint64_t *__restrict__ out, const uint4 *__restrict__ part,
                                                                       int rows, const CommitCut cut, int ll) {
    const int lane = threadIdx.x & 31, per = 32 >> ll;
    const unsigned warp = blockIdx.x * (REDUCE_THREADS / 32) + (threadIdx.x >> 5);
    const int row = (int)(warp * (unsigned)per) + (lane & (per - 1)), sub = lane >> (5 - ll), g = row >> 5;
    const int P = row >= rows ? 0 : g < cut.full ? cut.P : cut.Pr;
    G1P acc, q;
    g1_set_inf(acc);
    if (sub < P) tile_load(acc, part + tile_index(0, 0, g * cut.P + sub), row & 31);
    for (int c = sub + (1 << ll); c < P; c += 1 << ll) {
        tile_load(q, part + tile_index(0, 0, g * cut.P + c), row & 31);
        g1_add(acc, acc, q);
    }
    __syncwarp();
    g1_sum_lanes(acc, per);
    if (P > 0 && sub == 0) g1p_to_ref(out + 18 * (size_t)row, acc);
}

int commit_blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_commit_partial, 128, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// Pass 1 as one wave of the warps the device holds at once, every lane group
// with a run of the same length (at least 4 digits): the last group's rows,
// packed, take a share of the warps like their share of the lanes.  B200, 48
// commitments of 4096 at window 10: 2.47 ms; with whole bases and whole groups 2.96.
// Where a group's share is few warps, rounding it down would leave much of the chip
// idle: several waves, by the least count of waves times digits of a run (a run's
// own sum and conversion taken as 4).
CommitCut commit_cut(int rows, int n, int W, int resident, int sms) {
    CommitCut c{};
    c.lanes = sms * 256;
    const int rest = rows & 31, lanes = rest ? 32 >> msm_row_lanes(rest) : 32;
    const double groups = (rows >> 5) + (rest ? 1.0 / lanes : 0.0);
    c.full = rows >> 5;
    c.rl = rest ? msm_row_lanes(rest) : 5;
    const int most = std::max(1, n * W / 4);
    const double share = resident / groups;
    // the last group's runs are no longer than the others'
    const auto part = [&](int p) { return rest ? (p + lanes - 1) / lanes : 0; };
    const auto warps = [&](int p) { return (double)c.full * p + part(p); };
    int P = std::max(1, (int)std::min<double>(most, share));
    while (P > 1 && warps(P) > resident) P--;
    if (share < 16) {
        double least = 0;
        for (int p = 1; p <= std::min(most, std::max(8, (int)(4 * share))); p++) {
            const double cost = std::ceil(warps(p) / resident) * ((double)n * W / p + 4);
            if (p == 1 || cost < least) least = cost, P = p;
        }
    }
    c.P = c.full ? P : 0;
    c.Pr = part(P);
    return c;
}

void launch_commit(uint64_t *out, uint4 *part, const uint64_t *poly, const uint4 *table, int rows, int n, int W,
                   int cb, const CommitCut &cut, cudaStream_t st) {
    k_commit_partial<<<blocks_for((size_t)cut.tiles(), 4), 128, 0, st>>>(part, poly, table, rows, n, W, cb, cut);
    // as many lanes a row as two warps a scheduler give, at most one a partial sum: a
    // block, or a part of a warp.  A block for each of many rows would add mostly
    // points at infinity: 10,000 commitments of 32 7.6 ms with blocks, 3.35 with lanes.
    const int lanes = cut.lanes / rows;
    if (lanes >= REDUCE_THREADS) {
        k_commit_reduce<<<(unsigned)rows, REDUCE_THREADS, 0, st>>>(out, part, cut);
        return;
    }
    int ll = 0;
    while (ll < 5 && (2 << ll) <= lanes && (2 << ll) <= std::max(cut.P, cut.Pr)) ll++;
    k_commit_reduce_rows<<<blocks_for((size_t)rows << ll, REDUCE_THREADS), REDUCE_THREADS, 0, st>>>(out, part, rows, cut, ll);
}

// How a launch is cut.  A segment's last rows % 32 rows form one or two segments
// of their own whose lanes are packed (msm_row_lanes); and while whole units leave the
// chip's last wave of warps a large share of the time, four warps (two in
// 64-thread blocks) share a unit.  Resident: three 128-thread blocks per SM.
// A batch of one or two rows has 16 or 32 lane groups already, and more warps
// would only add sums.  B200, window 10, MSM alone, before (a row per lane, a
// warp per unit) and after: 1 row of 4096 4.41 -> 0.21 ms, 19 of 2048 4.64 ->
// 1.33, 160 of 4096 15.1 -> 13.5; at 512 rows of 4096 (4.6 waves) splitting
// costs 1 %, 40.7 -> 41.1, hence the line at 4 waves.
void launch_msm(const MsmArgs &in, int threads, int sms, cudaStream_t st) {
    if (threads != 64 && threads != 128 && threads != 256) threads = 128;
    if (threads > MSM_MAX_THREADS) threads = MSM_MAX_THREADS;
    MsmArgs a = in;
    a.nseg = 0;
    unsigned units = 0;
    for (int k = 0; k < in.nseg; k++) {
        // whole groups; then 16 rows when the rest is 17 to 24 (at most half of
        // the packed lanes of the last part idle); then the rest
        const int rows = in.seg[k].rows, full = rows & ~31, rest = rows & 31;
        const int cut[4] = {0, full, full + (rest > 16 && rest <= 24 ? 16 : 0), rows};
        for (int part = 0; part < 3; part++) {
            const int n = cut[part + 1] - cut[part];
            if (n <= 0) continue;
            MsmSeg s = in.seg[k];
            s.row0 = cut[part];
            s.rows = cut[part + 1];
            s.rl = part ? msm_row_lanes(n) : 5;
            s.G = part ? 1 : n / 32;
            s.fill = cut[part + 1] == rows;
            s.warp_start = units;
            units += (unsigned)s.G << s.log_m;
            a.seg[a.nseg++] = s;
        }
    }
    const unsigned resident = (unsigned)sms * 12;
    int rl_max = 0;
    for (int k = 0; k < a.nseg; k++) rl_max = std::max(rl_max, a.seg[k].rl);
    a.split = 1;
    if (rl_max > 1 && units < 4 * resident) a.split = threads == 64 ? 2 : 4;
    for (int k = 0; k < a.nseg; k++) {
        // at most 32 terms: lane groups and warps together
        a.seg[k].rl = std::max(a.seg[k].rl, a.split == 4 ? 2 : a.split == 2 ? 1 : 0);
        a.seg[k].warp_start *= (unsigned)a.split;
    }
    a.warps = units * (unsigned)a.split;
    const size_t smem = a.split > 1 ? (size_t)threads * 36 * sizeof(uint32_t) : 0;
    k_msm<<<blocks_for(a.warps, (unsigned)threads / 32), threads, smem, st>>>(a);
}

}  // namespace fk
