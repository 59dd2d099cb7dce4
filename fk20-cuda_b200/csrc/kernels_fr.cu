// kernels_fr.cu -- Fr side of the pipeline: toeplitz gather fused with the
// 16 Fr FFTs of each row (fk20_poly2toeplitz_coefficients.cu:25-58 followed
// by fr_fft.cu:28-158), plus the reference-layout Fr FFT and toeplitz entry
// points.  Fr data stays in standard form; twiddles are Montgomery constants,
// so Montgomery products of data by twiddles return standard form.
#include "consts.cuh"
#include "glv.cuh"
#include "launch.h"
#include "layout.cuh"

namespace fk {

cudaError_t upload_consts_fr() { return upload_module_consts(); }

// Decimation-in-time transform of m = 2^log_m >= 8 values by m / 8 threads, 8
// values a thread: up to three stages at a time in registers, exchanged
// between through shared memory (word-major, position p at p + p / 8: no bank
// conflicts in the first two passes, at most two-way in the last).
//
// The multiply pipe's share at m = 512 is 1,793 products a transform (0.13 ms
// for 4,000); one stage at a time through sm[m][8] took 0.35 ms, its eight-word
// stride an eight-way bank conflict on every access; this takes 0.20 ms
// (128-thread blocks at 134 registers 0.22; for 4,000 transforms of 128 values
// 0.055 against 0.072).
//
// Load: fn(natural index) -> value, store: fn(index, value).
constexpr int FR_THREADS = 64;  // threads of a block: 64 / (m / 8) transforms
constexpr int FR_STRIDE = FR_THREADS * 9;
constexpr int FR_SMEM_WORDS = 8 * FR_STRIDE;

FK_D int fr_slot(int p) { return p + (p >> 3); }

// stages s0 .. s0 + NB - 1 of the 8 >> NB sets of 2^NB values each that thread t holds
template <int NB>
__device__ __forceinline__ void fr_pass(int t, int log_m, int s0, bool inverse, Fr v[8]) {
    const int m8 = 1 << (log_m - 3);
#pragma unroll
    for (int u = 0; u < (8 >> NB); u++) {
        const int r = t + u * m8, low = r & ((1 << s0) - 1);
#pragma unroll
        for (int b = 0; b < NB; b++) {
#pragma unroll
            for (int h = 0; h < (1 << NB) / 2; h++) {
                const int q = ((h >> b) << (b + 1)) | (h & ((1 << b) - 1));
                Fr &x = v[(u << NB) + q], &y = v[(u << NB) + (q | (1 << b))];
                // power of w_m, then of w_512
                const int j = ((q & ((1 << b) - 1)) << s0) | low;
                int tix = j << (MAX_LOG_M - 1 - s0 - b);
                if (tix != 0) {
                    if (inverse) tix = 512 - tix;
                    const uint4 *w = reinterpret_cast<const uint4 *>(g_fr_tw[tix]);
                    const uint4 w0 = w[0], w1 = w[1];
                    Fr tw;
                    tw.w[0] = w0.x; tw.w[1] = w0.y; tw.w[2] = w0.z; tw.w[3] = w0.w;
                    tw.w[4] = w1.x; tw.w[5] = w1.y; tw.w[6] = w1.z; tw.w[7] = w1.w;
                    f_mul(y, y, tw);
                }
                Fr d;
                f_sub(d, x, y);
                f_add(x, x, y);
                y = d;
            }
        }
    }
}

// position of value k of thread t in the pass of NB stages from s0
template <int NB>
FK_D int fr_pos(int t, int log_m, int s0, int k) {
    const int r = t + (k >> NB) * (1 << (log_m - 3)), q = k & ((1 << NB) - 1);
    return ((r >> s0) << (s0 + NB)) | (q << s0) | (r & ((1 << s0) - 1));
}

template <class LD, class ST>
__device__ __forceinline__ void fr_fft_block(uint32_t *sm, int t, int log_m, bool inverse, const LD &ld, const ST &st) {
    Fr v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) ld(v[k], (int)bitrev((unsigned)(8 * t + k), log_m));
    fr_pass<3>(t, log_m, 0, inverse, v);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (log_m == 3) { st(8 * t + k, v[k]); continue; }
        const int at = fr_slot(8 * t + k);
#pragma unroll
        for (int w = 0; w < 8; w++) sm[w * FR_STRIDE + at] = v[k].w[w];
    }
    for (int s0 = 3; s0 < log_m; s0 += 3) {
        const int nb = log_m - s0 < 3 ? log_m - s0 : 3;
        const bool last = s0 + 3 >= log_m;
        __syncthreads();
        int pos[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            pos[k] = nb == 3 ? fr_pos<3>(t, log_m, s0, k) : nb == 2 ? fr_pos<2>(t, log_m, s0, k) : fr_pos<1>(t, log_m, s0, k);
            const int at = fr_slot(pos[k]);
#pragma unroll
            for (int w = 0; w < 8; w++) v[k].w[w] = sm[w * FR_STRIDE + at];
        }
        if (nb == 3) fr_pass<3>(t, log_m, s0, inverse, v);
        else if (nb == 2) fr_pass<2>(t, log_m, s0, inverse, v);
        else fr_pass<1>(t, log_m, s0, inverse, v);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (last) { st(pos[k], v[k]); continue; }
            const int at = fr_slot(pos[k]);  // the same positions: no other thread reads them before the barrier
#pragma unroll
            for (int w = 0; w < 8; w++) sm[w * FR_STRIDE + at] = v[k].w[w];
        }
    }
}

// toeplitz coefficient p of column i for a row of n = 16 k coefficients
// (FK20Py/fk20_multi_cuda.py:145-146; fk20_poly2toeplitz_coefficients.cu:40-56):
//   p = 0: poly[n-1-i];  1 <= p <= k+1: 0;  p = k+2+t: poly[2l-1-i + l t]
__device__ void toeplitz_coef(Fr &v, const uint64_t *__restrict__ poly, int n, int i, int p) {
    const int k = n / L_COLS;
    if (p == 0) {
        fr_from_ref(v, poly + 4 * (size_t)(n - 1 - i));
    } else if (p <= k + 1) {
        f_set_zero(v);
    } else {
        fr_from_ref(v, poly + 4 * (size_t)(2 * L_COLS - 1 - i + L_COLS * (p - k - 2)));
    }
}

// A scalar tile entry holds the GLV halves of the canonical scalar v:
// uint4 0 = v mod lambda, uint4 1 (32 entries on) = v div lambda
// (glv.cuh); the MSM's tables cover 128-bit scalars.
__device__ __forceinline__ void store_scalar(uint4 *dst, const uint32_t v[8]) {
    uint32_t s1[4], s2[4];
    glv_split(s1, s2, v);
    dst[0] = make_uint4(s1[0], s1[1], s1[2], s1[3]);
    dst[32] = make_uint4(s2[0], s2[1], s2[2], s2[3]);
}

// transform (row, i) = 16 row + i of the launch: toeplitz -> FFT -> scalar
// tiles S[g][c][i][q][lane], group g at S + g * stride
__global__ void __launch_bounds__(FR_THREADS, 8) k_tc_fft(uint4 *__restrict__ S, size_t stride, const uint64_t *__restrict__ poly,
                                                      const size_t *__restrict__ row_off, int n, int log_m, unsigned rows) {
    __shared__ uint32_t sm[FR_SMEM_WORDS];
    const int m8 = 1 << (log_m - 3), sub = threadIdx.x / m8, t = threadIdx.x % m8;
    const unsigned tr = blockIdx.x * (FR_THREADS / m8) + sub;
    const int row = (int)(tr / L_COLS), i = (int)(tr % L_COLS);
    const bool on = row < (int)rows;
    const uint64_t *pr = poly + 4 * (!on ? 0 : row_off ? row_off[row] : (size_t)row * n);
    uint4 *dst = S + (row >> 5) * stride + (size_t)i * SCAL_Q * 32 + (row & 31);
    fr_fft_block(
        sm + 9 * m8 * sub, t, log_m, false,
        [&](Fr &v, int p) {
            if (on) toeplitz_coef(v, pr, n, i, p);
            else f_set_zero(v);
        },
        [&](int c, const Fr &v) {
            if (on) store_scalar(dst + (size_t)c * L_COLS * SCAL_Q * 32, v.w);
        });
}

// batched Fr FFT on reference arrays, natural order in and out (fr_fft_wrapper /
// fr_ift_wrapper, fr_fft.cu:318-363); the inverse includes 1/m.  Each block
// reads its whole transforms before writing, so in-place calls are safe.
__global__ void __launch_bounds__(FR_THREADS, 8) k_fr_fft_ref(uint64_t *out, const uint64_t *in, int log_m, unsigned count,
                                                          int inverse) {
    __shared__ uint32_t sm[FR_SMEM_WORDS];
    const int m8 = 1 << (log_m - 3), sub = threadIdx.x / m8, t = threadIdx.x % m8;
    const unsigned tr = blockIdx.x * (FR_THREADS / m8) + sub;
    const bool on = tr < count;
    const size_t at = on ? (size_t)tr << log_m : 0;
    fr_fft_block(
        sm + 9 * m8 * sub, t, log_m, inverse != 0,
        [&](Fr &v, int p) {
            if (on) fr_from_ref(v, in + 4 * (at + p));
            else f_set_zero(v);
        },
        [&](int c, const Fr &x) {
            if (!on) return;
            Fr v = x;
            if (inverse) {
                Fr s;
#pragma unroll
                for (int k = 0; k < 8; k++) s.w[k] = g_fr_inv2[log_m][k];
                f_mul(v, v, s);
            }
            fr_to_ref(out + 4 * (at + c), v);
        });
}

// Few transforms: a butterfly a thread and a barrier a stage, grid (count),
// block m / 2.  A call that leaves the chip idle costs its chain of products: one
// a stage here, up to twelve a pass in registers above.
__global__ void __launch_bounds__(256) k_fr_fft_few(uint64_t *out, const uint64_t *in, int log_m, int inverse) {
    __shared__ uint32_t sm[512][8];
    const int m = 1 << log_m, tid = threadIdx.x;
    const uint64_t *src = in + 4 * (size_t)blockIdx.x * m;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int p = tid + h * (m >> 1);
        Fr v;
        fr_from_ref(v, src + 4 * (size_t)p);
        const int d = (int)bitrev((unsigned)p, log_m);
#pragma unroll
        for (int k = 0; k < 8; k++) sm[d][k] = v.w[k];
    }
    __syncthreads();
    for (int s = 0; s < log_m; s++) {
        const int half = 1 << s, j = tid & (half - 1), i0 = ((tid >> s) << (s + 1)) | j, i1 = i0 + half;
        Fr u, v, t;
#pragma unroll
        for (int k = 0; k < 8; k++) { u.w[k] = sm[i0][k]; v.w[k] = sm[i1][k]; }
        const int texp = j << (log_m - 1 - s);  // power of w_m
        if (texp != 0) {
            int tix = (texp << (MAX_LOG_M - log_m)) & 511;  // power of w_512
            if (inverse) tix = (512 - tix) & 511;
#pragma unroll
            for (int k = 0; k < 8; k++) t.w[k] = g_fr_tw[tix][k];
            f_mul(v, v, t);
        }
        Fr x, y;
        f_add(x, u, v);
        f_sub(y, u, v);
#pragma unroll
        for (int k = 0; k < 8; k++) { sm[i0][k] = x.w[k]; sm[i1][k] = y.w[k]; }
        __syncthreads();
    }
    uint64_t *dst = out + 4 * (size_t)blockIdx.x * m;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = tid + h * (m >> 1);
        Fr v;
#pragma unroll
        for (int k = 0; k < 8; k++) v.w[k] = sm[c][k];
        if (inverse) {
            Fr s;
#pragma unroll
            for (int k = 0; k < 8; k++) s.w[k] = g_fr_inv2[log_m][k];
            f_mul(v, v, s);
        }
        fr_to_ref(dst + 4 * (size_t)c, v);
    }
}

// many transforms of 2 and 4 values, one thread each
__global__ void k_fr_fft_tiny(uint64_t *out, const uint64_t *in, int log_m, unsigned count, int inverse) {
    const unsigned tr = blockIdx.x * blockDim.x + threadIdx.x;
    if (tr >= count) return;
    const int m = 1 << log_m;
    const size_t at = (size_t)tr << log_m;
    Fr v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (k < m) fr_from_ref(v[(int)bitrev((unsigned)k, log_m)], in + 4 * (at + k));
    for (int s = 0; s < log_m; s++)
        for (int h = 0; h < m / 2; h++) {
            const int half = 1 << s, j = h & (half - 1), q = ((h >> s) << (s + 1)) | j;
            Fr x = v[q], y = v[q + half];
            if (j) {  // w_4
                Fr tw;
                for (int k = 0; k < 8; k++) tw.w[k] = g_fr_tw[inverse ? 384 : 128][k];
                f_mul(y, y, tw);
            }
            f_add(v[q], x, y);
            f_sub(v[q + half], x, y);
        }
    for (int k = 0; k < m; k++) {
        if (inverse) {
            Fr s;
            for (int w = 0; w < 8; w++) s.w[w] = g_fr_inv2[log_m][w];
            f_mul(v[k], v[k], s);
        }
        fr_to_ref(out + 4 * (at + k), v[k]);
    }
}

// grid (rows), block 256: reference toeplitz output tc[row][16][m], canonical
__global__ void k_toeplitz_ref(uint64_t *__restrict__ tc, const uint64_t *__restrict__ poly, int n, int log_m) {
    const int m = 1 << log_m;
    const int row = blockIdx.x;
    const uint64_t *pr = poly + 4 * (size_t)row * n;
    uint64_t *dst = tc + 4 * (size_t)row * L_COLS * m;
    for (int e = threadIdx.x; e < L_COLS * m; e += blockDim.x) {
        Fr v;
        toeplitz_coef(v, pr, n, e / m, e % m);
        fr_to_ref(dst + 4 * (size_t)e, v);
    }
}

// grid-stride: reference tc_fft[row][16][m] -> scalar tiles (canonicalised)
__global__ void k_ref_to_scalars(uint4 *__restrict__ S, const uint64_t *__restrict__ tcf, int rows, int log_m) {
    const int m = 1 << log_m;
    const size_t total = (size_t)rows * L_COLS * m;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int row = (int)(e / ((size_t)L_COLS * m));
        const int rem = (int)(e % ((size_t)L_COLS * m));
        const int i = rem / m, c = rem % m;
        Fr v;
        fr_from_ref(v, tcf + 4 * e);
        const int g = row >> 5, lane = row & 31;
        store_scalar(S + ((((size_t)g * m + c) * L_COLS + i) * SCAL_Q) * 32 + lane, v.w);
    }
}

void launch_tc_fft(uint4 *S, size_t stride, const uint64_t *poly, const size_t *row_off, int n, int log_m, unsigned rows,
                   cudaStream_t st) {
    const unsigned per = FR_THREADS >> (log_m - 3);
    k_tc_fft<<<blocks_for((size_t)rows * L_COLS, per), FR_THREADS, 0, st>>>(S, stride, poly, row_off, n, log_m, rows);
}
// Values an SM up to which k_fr_fft_few is the faster one, for forward and inverse
// transforms (of which k_fr_fft_ref pays more for the factor 1/m) of 2^1 .. 2^9
// values.  Its time is that of one transform and then grows with every block that
// an SM gets: the others' is flat up to about 2,000 values an SM.  B200, us, few and
// other, at the line and at twice it: 2 values inverse 4.6 and 6.3, 6.3 and 6.2; 4:
// 6.6 and 6.8, 10.5 and 7.2; 8: 10.5 and 10.6, 14.6 and 10.6; 16: 14.6 and 14.7, 23.0
// and 15.6; 32: 16.9 and 17.1, 28.0 and 18.9; 64: 22.9 and 22.9, 37.5 and 26.0; 128:
// 31.1 and 31.0, 58.0 and 39.0; 256: 34.0 and 35.2, 62.0 and 45.5; 512: 29.0 and 33.2,
// 47.6 and 40.9.
constexpr unsigned short FR_FEW[2][MAX_LOG_M + 1] = {{0, 8, 80, 176, 400, 672, 944, 1472, 1536, 1024},
                                                     {0, 8, 64, 176, 400, 816, 1312, 1648, 1600, 1536}};
void launch_fr_fft_ref(uint64_t *out, const uint64_t *in, int log_m, unsigned count, int inverse, int sms, cudaStream_t st) {
    if (((size_t)count << log_m) <= (size_t)sms * FR_FEW[inverse != 0][log_m]) {
        k_fr_fft_few<<<count, 1u << (log_m - 1), 0, st>>>(out, in, log_m, inverse);
        return;
    }
    if (log_m < 3) {
        k_fr_fft_tiny<<<blocks_for(count, 64), 64, 0, st>>>(out, in, log_m, count, inverse);
        return;
    }
    const unsigned per = FR_THREADS >> (log_m - 3);
    k_fr_fft_ref<<<blocks_for(count, per), FR_THREADS, 0, st>>>(out, in, log_m, count, inverse);
}
void launch_toeplitz_ref(uint64_t *tc, const uint64_t *poly, int n, int log_m, unsigned rows, cudaStream_t st) {
    k_toeplitz_ref<<<rows, 256, 0, st>>>(tc, poly, n, log_m);
}
void launch_ref_to_scalars(uint4 *S, const uint64_t *tcf, int rows, int log_m, cudaStream_t st) {
    k_ref_to_scalars<<<grid_stride_blocks((size_t)rows * L_COLS * (1u << log_m)), 256, 0, st>>>(S, tcf, rows, log_m);
}

}  // namespace fk
