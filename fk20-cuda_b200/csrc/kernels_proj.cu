// kernels_proj.cu -- the map hext_fft -> h_fft as a persistent launch over the
// tasks of a projection plan (proj_plan.cuh).
//
// One warp per (task, group of 32 lanes): a task is an addition (usually
// a + b and a - b together), a few doublings, one fixed-scalar product
// (scalar_prog.cuh, warp-uniform) or an output.  Warps take (task, group)
// pairs in dependency order from a global counter and wait for the versions
// of the slots they read (ready[g][slot], published with release semantics
// after the stores) and, in the last phase, for all products of the group
// (ready[g][slots] counts them), which lets the additions after the products
// reuse every slot of the phases before.  Tasks go only to running warps and
// only wait on tasks of lower index, so the lowest unfinished task never
// waits and every wait ends, with any number of resident blocks.  Each wait is
// still bounded (spin_limit polls); on expiry the kernel records an error code
// and returns.  Points written by other SMs are read through L2 (ld.cg).
//
// Bound by the integer multiply pipe, as the butterflies it replaces, with
// about half their products; a small batch is bound by the depth, one product
// (~1,300 dependent Fp products) and ~35 additions instead of 14-16 products.
// Whole calls (MSM included, whose own cuts and products became faster too) with
// the persistent radix-2 FFT and now: one blob of 4096 34.8 and 3.2 ms, 160 blobs
// 68.6 and 31.5, 512 blobs at window 13 172.8 and 86.0.
#define FK_FP_MUL_OUTLINE 1
#include "../../include/fk20_b200.h"
#include "check.cuh"
#include "launch.h"
#include "layout.cuh"
#include "scalar_prog.cuh"
#include <string.h>

namespace fk {

FK_CHECK_WORD(proj)

namespace {

FK_D unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
FK_D void st_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

FK_D void load_cg(G1P &p, const uint4 *base, int lane) {
    uint32_t w[36];
#pragma unroll
    for (int q = 0; q < TILE_Q; q++) {
        const uint4 v = __ldcg(base + q * 32 + lane);
        w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < 12; k++) { p.x.w[k] = w[k]; p.y.w[k] = w[12 + k]; p.z.w[k] = w[24 + k]; }
}
FK_D void slot_cg(const StridedPoint &slot, const uint4 *base, int lane) {
#pragma unroll
    for (int q = 0; q < TILE_Q; q++) {
        const uint4 v = __ldcg(base + q * 32 + lane);
        slot.base[(4 * q) * slot.stride] = v.x;
        slot.base[(4 * q + 1) * slot.stride] = v.y;
        slot.base[(4 * q + 2) * slot.stride] = v.z;
        slot.base[(4 * q + 3) * slot.stride] = v.w;
    }
}
FK_D void store_coord_cg(uint4 *base, int lane, int c, const Fp &f) {
#pragma unroll
    for (int q = 0; q < 3; q++)
        __stcg(base + (3 * c + q) * 32 + lane, make_uint4(f.w[4 * q], f.w[4 * q + 1], f.w[4 * q + 2], f.w[4 * q + 3]));
}
FK_D void store_cg(uint4 *base, int lane, const G1P &p) {
    store_coord_cg(base, lane, 0, p.x);
    store_coord_cg(base, lane, 1, p.y);
    store_coord_cg(base, lane, 2, p.z);
}

// A product keeps its scale u in the tile it will write: 144 words of scratch a
// thread instead of 156 let a sixth block fit an SM.
struct TileU {
    uint4 *d0;
    int lane;
    FK_D void put(const Fp &f) const { store_coord_cg(d0, lane, 0, f); }
    FK_D void get(Fp &f) const {
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const uint4 v = __ldcg(d0 + q * 32 + lane);
            f.w[4 * q] = v.x; f.w[4 * q + 1] = v.y; f.w[4 * q + 2] = v.z; f.w[4 * q + 3] = v.w;
        }
    }
};

// The launch gives up: the other warps stop at their next task, and the host
// learns of it from a word of its own.  That word is written only here, so a
// later launch that succeeds does not take the report away.
FK_D void proj_stop(const ProjArgs &P, int code) {
    if (atomicCAS(P.err, 0, code) == 0) {
        *(volatile int *)P.report = code;
        __threadfence_system();
    }
}

}  // namespace

// Six blocks (12 warps) an SM, 168 registers: with three warps a scheduler the
// pipe stays busier than with two (512 blobs of 4096: 54.7 ms at 228 registers
// and four blocks, 52.6 here); small launches use fewer of them (proj_grid).  What
// 168 registers spill (524 bytes stored, 800 loaded a thread) is 0.14 % of the
// instructions.
__global__ void __launch_bounds__(FFT_THREADS, 6) k_proj(const __grid_constant__ ProjArgs P) {
    __shared__ uint32_t slots[PROG_POINT_WORDS][FFT_THREADS];
    const int lane = threadIdx.x & 31;
    const ProgSlots slot{&slots[0][threadIdx.x], FFT_THREADS};
    for (;;) {
        unsigned index = 0;
        if (lane == 0) index = P.first + atomicAdd(P.next, 1u);
        index = __shfl_sync(0xffffffffu, index, 0);
        if (index >= P.last) return;
        if (*(volatile int *)P.err) return;
        int sk, tk, g;
        proj_decode(P.runs, index, sk, tk, g);
        const ProjSeg &S = P.seg[sk];
        const ProjArena A = S.arena;
        ProjTask t;
        {
            const uint2 *src = reinterpret_cast<const uint2 *>(S.tasks + tk);
            uint2 w[3] = {src[0], src[1], src[2]};
            memcpy(&t, w, sizeof t);
        }
        // checked build: the decoded task lies in its segment and names slots
        // and a program that exist; else stop the launch (no access, no
        // publication)
        if (!FK_CHECK(g_check_proj, sk < P.nseg && tk < S.ntasks && g < A.G && t.a < A.slots && t.d0 < A.slots &&
                                        (t.b == PROJ_NONE || t.b < A.slots) && (t.b2 == PROJ_NONE || t.b2 < A.slots) &&
                                        (t.d1 == PROJ_NONE || t.d1 < A.slots),
                      FK20_CHECK_FFT_TASK) ||
            !FK_CHECK(g_check_proj, t.op != PROJ_MUL || t.prog < S.nprog, FK20_CHECK_FFT_PROGRAM)) {
            if (lane == 0) proj_stop(P, 2000);
            return;
        }
        unsigned *rg = S.ready + (size_t)g * (A.slots + 1);
        // an output reads the other instance's slot: b for instance 0, b2 for
        // instance 1 (both, in the same group, when instances share a group)
        const bool pair = g >= 2 * A.F;
        const int inst = pair ? lane >> 4 : g >= A.F;
        const int gx = pair ? g : inst ? g - A.F : g + A.F;
        const int sx = inst ? t.b2 : t.b;
        int ok = 1;
        if (lane < 4) {  // lane 0: a, 1: b, 2: b2, 3: the group's products
            const unsigned *r = rg;
            unsigned need = 0;
            const bool out = t.op == PROJ_OUT;
            if (lane == 0) r = rg + t.a, need = t.va;
            if (lane == 1 && t.b != PROJ_NONE && !(out && !pair && inst)) {
                r = (out ? S.ready + (size_t)gx * (A.slots + 1) : rg) + t.b, need = t.vb;
            }
            if (lane == 2 && t.b2 != PROJ_NONE && !(out && !pair && !inst)) {
                r = (out ? S.ready + (size_t)gx * (A.slots + 1) : rg) + t.b2, need = t.vb2;
            }
            if (lane == 3 && t.phase == 2) r = rg + A.slots, need = (unsigned)S.nprod;
            unsigned spins = 0;
            while (need && ld_acquire(r) < need) {
                if (++spins >= P.spin_limit) { ok = 0; break; }
                __nanosleep(64);
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        __threadfence();
        if (!ok) {
            if (lane == 0) proj_stop(P, 1000 + t.phase);
            return;
        }
        const uint4 *pa = S.D + proj_tile(A, g, t.a);
        uint4 *d0 = S.D + proj_tile(A, g, t.d0);
        G1P acc;
        if (t.op == PROJ_MUL) {
            slot_cg(slot[0], pa, lane);
            g1_mul_prog(acc, slot, S.progs + (size_t)t.prog * PROG_WORDS, TileU{d0, lane});
            store_cg(d0, lane, acc);
        } else if (t.op == PROJ_SHL) {
            load_cg(acc, pa, lane);
            for (int k = 0; k < t.sh; k++) g1_dbl(acc, acc);
            store_cg(d0, lane, acc);
        } else {
            const uint4 *pb = t.op == PROJ_OUT ? S.D + proj_tile(A, gx, sx) : S.D + proj_tile(A, g, t.b);
            const int lb = t.op == PROJ_OUT && pair ? lane ^ 16 : lane;
            // the operand with the coefficient goes to the scratch point: b, or a for an output
            const bool out = t.op == PROJ_OUT;
            slot_cg(slot[1], out ? pa : pb, out ? lane : lb);
            if (t.phi) {
                Fp x;
                slot_get(x, slot.word(36), slot.stride);
                fp_mul_beta(x, x, t.phi);
                slot_put(slot.word(36), slot.stride, x);
            }
            if (t.sh) {
                slot[1].load(acc);
                for (int k = 0; k < t.sh; k++) g1_dbl(acc, acc);
                slot[1].put(acc);
            }
            load_cg(acc, out ? pb : pa, out ? lb : lane);
            if (t.d1 != PROJ_NONE) {
                uint4 *d1 = S.D + proj_tile(A, g, t.d1);
                g1_addsub_q(acc, slot[1], [&](int which, int c, const Fp &f) { store_coord_cg(which ? d1 : d0, lane, c, f); });
            } else {
                g1_add_q(acc, acc, slot[1], t.neg != 0);
                store_cg(d0, lane, acc);
            }
        }
        __threadfence();
        __syncwarp();
        if (lane == 0 && index != P.unpublished) {  // see ProjArgs::unpublished (tests of the bounded wait)
            if (t.op == PROJ_MUL) atomicAdd(rg + A.slots, 1u);
            st_release(rg + t.d0, t.w0);
            if (t.d1 != PROJ_NONE) st_release(rg + t.d1, t.w1);
        }
    }
}

int proj_blocks_per_sm() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_proj, FFT_THREADS, 0) != cudaSuccess) return 0;
    return n;
}

void launch_proj(const ProjArgs &p, int blocks, cudaStream_t st) { k_proj<<<blocks, FFT_THREADS, 0, st>>>(p); }

// reference rows [rows][m] -> arena inputs: of the two instances of a
// projection, or of a transform (position c in slot c)
__global__ void k_ref_to_arena(uint4 *__restrict__ D, ProjArena A, const uint64_t *__restrict__ src, int rows, int log_m,
                               int two) {
    const int m = 1 << log_m;
    const size_t total = (size_t)(32 * A.F + 16 * A.paired) * m;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int row = (int)(e >> log_m), c = (int)(e & (size_t)(m - 1));
        G1P p;
        if (row < rows) g1p_from_ref(p, src + 18 * e);
        else g1_set_inf(p);
        int g, lane;
        (void)proj_lane(A, row, two ? proj_in_inst(c) : 0, g, lane);
        tile_store(D + proj_tile(A, g, two ? proj_in_slot(c, log_m) : c), lane, p);
    }
}

void launch_ref_to_arena(uint4 *D, const ProjArena &A, const uint64_t *src, int rows, int log_m, int two, cudaStream_t st) {
    const size_t lanes = (size_t)(32 * A.F + 16 * A.paired) << log_m;
    k_ref_to_arena<<<grid_stride_blocks(lanes), 256, 0, st>>>(D, A, src, rows, log_m, two);
}

}  // namespace fk
