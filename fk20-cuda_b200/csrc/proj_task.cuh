// proj_task.cuh -- tasks, arenas and launch order of the projection plans
// (proj_plan.cuh builds them, kernels_proj.cu runs them).
#pragma once
#include "limbs.cuh"

namespace fk {

// ---------------------------------------------------------------- task format
enum ProjOp : uint8_t {
    PROJ_LIN = 0,   // d0 = a + s phi^k 2^sh b; d1 (if any) = a - s phi^k 2^sh b
    PROJ_SHL = 1,   // d0 = 2^sh a
    PROJ_MUL = 2,   // d0 = [program] a
    PROJ_OUT = 3    // d0 = s phi^k a + (slot b of instance 1 for instance 0, slot b2 of instance 0 for instance 1)
};
constexpr uint16_t PROJ_NONE = 0xffff;

struct alignas(8) ProjTask {
    uint8_t op, sh, phi, neg;
    uint16_t d0, d1;         // slots written (d1 PROJ_NONE: none)
    uint16_t a, b, b2;       // slots read (PROJ_NONE: none); b2 of a task that is no output: waited for, not read
    uint8_t va, vb, vb2;     // versions the reads need (0: the input itself)
    uint8_t w0, w1, phase;   // versions the writes publish; the task's phase
    uint16_t prog;           // PROJ_MUL: program index
    uint16_t pad;
};
static_assert(sizeof(ProjTask) == 24, "three 8-byte loads");

// ---------------------------------------------------------------- arena and launch
// A segment's points live in an arena of G groups of `slots` point tiles
// (layout.cuh: 9 x 32 uint4 each).  Lanes of a group are (row, instance)
// pairs: groups [0, F) are instance 0 of 32 rows each and groups [F, 2 F)
// instance 1; the last rows of a segment, when 16 or fewer, share one more
// group (`paired`): lane 16 inst + row.
struct ProjArena {
    int slots, G, F, paired;
};
FK_HD ProjArena proj_arena(int slots, unsigned rows) {
    const int rest = (int)(rows & 31u), paired = rest > 0 && rest <= 16;
    const int F = (int)(rows >> 5) + (rest > 16);
    return ProjArena{slots, 2 * F + paired, F, paired};
}
// false: a lane beyond the rows that the paired group holds
FK_HD bool proj_lane(const ProjArena &a, int row, int inst, int &g, int &lane) {
    const bool pair = row >= 32 * a.F;
    const int r = pair ? row - 32 * a.F : row & 31;
    g = pair ? 2 * a.F : inst * a.F + (row >> 5);
    lane = pair ? 16 * inst + r : r;
    return !pair || (a.paired && r < 16);
}
FK_HD size_t proj_tile(const ProjArena &a, int g, int slot) { return ((size_t)g * a.slots + slot) * 9 * 32; }

// Task order of a launch: runs of tasks (first .. first + count) over groups
// [g0, g0 + gn) of one segment, groups fastest.
constexpr int MAX_PROJ_RUNS = 1024;
constexpr int MAX_PROJ_SEGS = 8;
struct ProjRun {
    unsigned start;  // launch index of its first (task, group)
    unsigned short first, seg, g0, gn;
};
struct ProjRuns {
    ProjRun run[MAX_PROJ_RUNS];
    int n;
    unsigned total;
};
FK_HD void proj_decode(const ProjRuns &r, unsigned t, int &seg, int &task, int &g) {
    int lo = 0, hi = r.n - 1;  // the last run with start <= t
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (r.run[mid].start <= t) lo = mid;
        else hi = mid - 1;
    }
    const unsigned k = t - r.run[lo].start, gn = r.run[lo].gn;
    seg = r.run[lo].seg;
    task = r.run[lo].first + (int)(k / gn);
    g = r.run[lo].g0 + (int)(k % gn);
}

// input slot and instance of hext position c; output k, instance of position j
FK_HD int proj_in_slot(int c, int log_m) {
    const int H = 1 << (log_m - 1), i = c >> 1;
    return (c & 1) ? H - 1 - i : (H - i) & (H - 1);
}
FK_HD int proj_in_inst(int c) { return (c & 1) ^ 1; }

}  // namespace fk
