// dfs_kernel.cuh -- persistent iterative-DFS kernel for sm_100a.
//
// Replaces the reference kernel n_queens() of src/n_queens_cuda.cu:9-82 and
// its ticket counter global_counter (:8).  Same per-task arithmetic
// (n_queens() of src/n_queens.cpp:8-21); different machine organisation:
//
//  * One lane runs one DFS.  The current level lives in registers
//    (cols, ld, rd, avail); only levels that still have untried columns are
//    pushed to the lane's shared-memory stack, so a pop always resumes a level
//    with work and every DFS step places exactly one queen.
//  * The count kernels' step (VAR 6) lists only a level's alive columns --
//    those whose child still has a free column in the next row -- skips
//    children whose row two below has none, and counts the completions of a
//    row N-2 level from its alive columns instead of stepping rows N-2 and N-1
//    (44 % fewer steps at N=18).
//  * cols carries the off-board bits (~last) pre-set.  Then the free mask is
//    one LOP3 (~(cols|ld|rd)) with no `& last`, a completed board is
//    cols == 0xffffffff, and no depth counter is kept at all.
//  * Stack layout: slot s of lane l in warp w is the 16-byte entry at
//    w*levels*512 + s*512 + l*16.  Every stack access is a 128-bit LDS/STS and
//    the eight lanes of a quarter-warp always cover the 32 banks once,
//    whatever the per-lane depths are, so no access needs more wavefronts
//    than a dense 16-byte access of the warp (the reference mixes in a
//    32-bit store, src/n_queens_cuda.cu:47, which is 4-way conflicted).
//  * Tasks come from a device queue: one atomicAdd per warp refill hands a
//    block of consecutive queue positions to the idle lanes (the reference
//    takes one atomic per task per thread, :10,80).  An optional permutation
//    maps queue positions to tasks (longest-first schedules).
//  * Once the queue is empty, idle lanes take the bottom (shallowest, hence
//    largest) stacked level of a busy lane in the same warp: __ballot_sync
//    finds donors and receivers, __shfl_sync moves the donor's slot address,
//    and the receiver loads the entry straight from the donor's stack.
//  * A warp with nothing left takes levels from other warps through a mailbox
//    in global memory (see "Mailbox").
//  * Counts are uint32 per lane inside a bounded inner loop, folded into
//    uint64 per lane, reduced per warp (shuffles) and per CTA, and the last
//    CTA to finish sums the per-CTA partials in a fixed order.
//
// Only warps that have no work wait (for mail, with a time and a poll limit);
// nothing else in the kernel depends on another CTA's progress.  An optional
// %globaltimer deadline bounds its run.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nqb {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kSlotBytes = 512;  // one stack level of one warp: 32 lanes x 16 B
constexpr uint32_t kNoOwner = 0xffffffffu;

enum CtlWord : int {
    kCtlHead = 0,      // next queue position
    kCtlDone = 1,      // CTAs finished
    kCtlError = 2,     // error bits (kErr*)
    kCtlTimeout = 3,   // set when the deadline stopped the kernel
    kCtlCont = 4,      // continuation entries written at a deadline stop
    kCtlMail = 5,      // mailbox tickets: low half requested, high half supplied
    kCtlWork = 6,      // signed: mail posted and not taken, minus warps out of work
    kCtlWords = 7,
};
enum : unsigned long long { kErrDepth = 1ull, kErrContOverflow = 2ull };
// Bits of *status_out: a task needed more stack levels than the launch had
// (it was skipped), and/or the run-time limit stopped the kernel early.
enum : unsigned long long { kStatDepth = 1ull, kStatTimeout = 2ull, kStatContOverflow = 4ull, kStatMail = 8ull };

// One slot of the mailbox through which busy warps hand stacked levels to warps
// that ran out of work (see "Mailbox" below).
constexpr int kMailLevels = 8;  // most levels of one slot
struct alignas(256) MailSlot {
    uint4 level[kMailLevels];      // (cols, ld, rd, avail) in the kernel's lane form
    uint32_t owner[kMailLevels];   // per-owner output slots (PER_OWNER kernels)
    uint32_t cls[kMailLevels];     // class indices (DIH kernels)
    uint32_t count;
    uint32_t state;                // use of the slot << 2 | kMail*
    uint32_t pad[14];
};
static_assert(sizeof(MailSlot) == 256, "slot layout");
enum : uint32_t { kMailEmpty = 0u, kMailFull = 1u, kMailGone = 2u, kMailDone = 3u };

struct DfsParams {
    const uint32_t *cols;      // task column masks (reference `cur`)
    const uint32_t *ld;        // task left-diagonal masks (reference `left`)
    const uint32_t *rd;        // task right-diagonal masks (reference `right`)
    const uint8_t *task_n;     // per-task board size, or nullptr (use N)
    const uint32_t *owner_of;  // per-task output slot, or nullptr (slot = task index)
    const uint32_t *order;     // queue position -> task index, or nullptr (identity)
    long long ntasks;
    long long nqueue;          // queue positions to run (<= ntasks; 0 = ntasks)
    int N;                     // board size when task_n is nullptr
    long long coarse;          // the first `coarse` tasks are queued as 2^lg_coarse shares of their
    uint32_t lg_coarse;        // columns each, the others as 2^lg_fine (see set_shares in launch.h)
    uint32_t lg_fine;
    int levels;                // stack slots per lane
    int inner;                 // DFS steps per outer trip (multiple of 4)
    int steal;                 // in-warp donation on/off
    unsigned long long limit_ns;     // run-time limit from the CTA's start, 0 = none
    unsigned long long *ctl;         // kCtlWords control words (zeroed before launch)
    unsigned long long *block_cnt;   // [gridDim.x] per-CTA count partials
    unsigned long long *block_nodes; // [gridDim.x] per-CTA node partials (NODES)
    unsigned long long *out_cnt;     // per-owner counts (PER_OWNER), zeroed by the host
    unsigned long long *out_nodes;   // per-owner nodes (PER_OWNER && NODES), zeroed by the host
    unsigned long long *sum_out;     // total count (device word)
    unsigned long long *nodes_out;   // total nodes (device word, NODES)
    unsigned long long *status_out;  // kStat* bits of this launch (device word)
    uint32_t k_one, k_two, k_mone;   // 1, 2, -1 (see dfs_step)
    unsigned long long *cta_times;   // optional [2*gridDim.x]: %globaltimer at CTA start and end
    int layout;                      // stack layout: 0 interleaved (default), 1 lane-major
    // Resumable runs.  Queue positions [0, n_cont_in) are continuation entries
    // (a lane's saved level: cols with the off-board bits set, ld, rd, untried
    // columns); position n_cont_in + j is task list position task_base + j.
    const uint4 *cont_in;
    const uint32_t *cont_in_owner;   // optional owners of the continuation entries
    long long n_cont_in;
    long long task_base;
    // At a deadline stop every lane writes its unfinished levels here (if not
    // null): the current level and each stacked level, in kCtlCont order.
    uint4 *cont_out;
    uint32_t *cont_out_owner;        // optional
    long long cont_cap;
    // Dihedral decomposition (DIH kernels only): class index per task and the
    // class table {popc threshold, row N-1 mask, tie column bit,
    // weight | tie weight << 16}; a child whose column mask (off-board bits
    // set) has more bits than the threshold may not use column 0 or N-1.
    const uint8_t *task_cls;
    const uint4 *cls_tab;
    uint32_t noside;                 // ~(column 0 | column N-1)
    // Resumable dihedral runs: the class index of each continuation entry
    // (in) and of each saved level (out).
    const uint8_t *cont_in_cls;
    uint8_t *cont_out_cls;
    // Mailbox (kernels without RESUME; nullptr switches it off).  Every slot is
    // kMailEmpty at the start of a launch and again at its end.
    MailSlot *mail;
    uint32_t mail_cap;
    uint32_t mail_patience_ns;  // how long a warp waits for mail, at most kMailPatienceNs
    // Where the host does not know the tasks' depth: the rows left in the deepest
    // task; the mailbox is used only if they are kMailRootRows or more.  The word is
    // not written during the launch and shares no cache line with the control words,
    // whose atomics would hold up its load.  nullptr: used.
    const uint32_t *mail_gate;
    // With cta_times: per-CTA sum over warps of the time spent waiting for mail.
    unsigned long long *cta_wait;
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ void lds128(uint32_t a, uint32_t &x, uint32_t &y, uint32_t &z, uint32_t &w) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a) : "memory");
}

// One DFS step of one lane, branch-free.  State: (cols, ld, rd, avail) of the
// level being enumerated; sp/bot are the lane's stack top/bottom addresses.
//   bit   = lowest free column;  avail -= bit
//   child = (cols|bit, (ld|bit)<<1, (rd|bit)>>1),  free = ~(c|l|r)
//   child cols == ~0            -> one completed board: cnt += 1
//   free != 0 (and bit != 0)    -> descend; the parent is pushed only if
//                                  it still has untried columns
//   otherwise, level exhausted  -> pop a stacked level if there is one
// An idle lane (avail == 0, empty stack) passes through with no effect.
// Right shift is arithmetic, as in the reference's `int` arithmetic.
//
// Operands: %0 cols, %1 ld, %2 rd, %3 avail, %4 sp, %5 cnt, %6 placements
// (node statistics), %7 bot, %8 = 1, %9 = 2, %10 = -1, %11 the slot stride
// (512 B interleaved, 16 B lane-major).  The constants arrive as kernel
// parameters, so the compiler cannot fold the multiply-adds below back into
// ALU adds/moves: adds, left shifts and register moves are issued in multiply-add
// form (the FMA pipe), which leaves LOP3, right shifts and compares to the ALU
// pipe (an all-ALU form was 20 % slower).  Predicates come from LOP3's predicate
// output (p = (result != 0) op q); four or sixteen steps share one asm block, whose
// head sets the constant predicate `pt1` (true) once.
//
// The forms: 4 and its in-place successors 6 and 7 for counts, 6 with a node counter
// for node counts, 5 and DIH4 for the dihedral kernels.  (Steps 1 to 3, which
// stepped every row, are gone.)
//
// VAR 4 ("filtered") enumerates only children that have a future.  A child C
// of the level (placed at column `bit`) lists the columns of the next row it
// may try (free = ~(c|l|r)); such a column b is dead when the row after it
// would have no free column at all.  With F0 = the free columns of that row
// before b is placed (~(c | l<<1 | r>>1)), b is dead exactly when F0 lies
// inside {b-1, b, b+1}, i.e. when no column of F0 is two or more away from
// b.  The alive columns are therefore
//   (columns >= lowest(F0) + 2) | (columns <= highest(F0) - 2)
//   = -(lo << 2) | (0x3fffffff >> bfind.shiftamt(F0))       (empty when F0 = 0)
// (bfind.shiftamt is 31 - the highest set bit's position, all ones for 0, and a
// shift by 32 or more gives 0).
// and the child's list becomes free & that mask.  A child on row N-2 (its
// column mask has 30 bits set, off-board bits included) is not entered: every
// alive column of it completes the board on row N-1, so the step adds the
// popcount of its filtered list.  Rows N-2 and N-1 are never stepped and dead
// children never cost a step or a stack push: at N=18, k=6 the steps fall from
// 29.7e9 to 18.6e9 and the pushes from 7.8e9 to 5.0e9.  Tasks and saved levels
// on rows N-2 and N-1 are counted when they are loaded.
//
// Look-ahead: a child above row N-2 whose row two below (F1 = ~(c | l<<2 |
// r>>2)) has no free column even before anything is placed under it is not
// entered either.  That takes a multiply, a shift and a LOP3 whose predicate
// output replaces pg, and removes 9 % of the steps at N=14, 11 % at N=18 and
// 12.6 % at N=21 (CPU model of the step); looking one row further would remove
// 5 % more for another three operations, which is even.
//
// Lane registers: ld holds the left mask pre-shifted for the children (left << 1),
// so a child's left mask is one multiply-add, ld + 2*bit (bit is free, so | equals
// +); rd too is kept pre-shifted (right >> 1), so a child's right mask is (bit >> 1) + rd, which the compiler
// issues as one operation (shift-and-add) where `|` and the shift took two, and
// the shift for the grandchildren rides on the descend move.  (A multiply-high
// in its place loads the FMA pipe more than it saves: 5-7 % slower.)
// Operands as above plus %12 = 0x3fffffff, %13 = -4, %14 = 30.
//
// What bounds it: integer issue (84 % of the issue slots, ALU pipe 72 %, FMA
// 69 %, XU 55 %, shared-memory wavefronts 62 % at N=18).  Measured without and
// with both changes: 1.1e6 prefixes of N=18, k=6 19.47 -> 18.34 ms (pre-shifted
// rd alone: 4 %), N=19 153.2 -> 147.8 ms, 8 % of N=21's prefixes 952 -> 911 ms.
// Pipe balance: taking the highest bit's mask from bfind's shift amount instead
// of a multiply-add saved 4.2 % at N=21, negating F0 on the ALU instead of the
// FMA pipe 0.3 %.  Slower at N=18: moving avail as a float on the light half of
// the FMA pipe (+1.5 %), moving registers in pairs by mad.wide (+30 %), one
// compare with two outputs for pg and p2 (+12 %: the compiler adds operations).
#define NQB_STEP4_HEAD                                                                \
    "{\n\t"                                                                           \
    ".reg .pred pt1, pb, pg, p2, pd, pk, pp, pq;\n\t"                                 \
    ".reg .b32 t, bit, nc, nl, nr, na, xl, xr, f0, lo, ma, mb, pos, pc, naf;\n\t"     \
    "setp.ne.u32 pt1, %8, 0;\n\t"

#define NQB_STEP4_CHILD                                                               \
    "mul.lo.s32 t, %3, %10;\n\t"                                                      \
    "lop3.and.b32 bit|pb, t, %3, 0, 0xC0, pt1;\n\t"                                   \
    "mad.lo.s32 nc, bit, %8, %0;\n\t"                                                 \
    "mad.lo.s32 nl, bit, %9, %1;\n\t"                                                 \
    "shr.u32 nr, bit, 1;\n\t"                                                         \
    "add.u32 nr, nr, %2;\n\t"                                                         \
    "lop3.b32 na, nc, nl, nr, 0x01;\n\t"                                              \
    "mul.lo.s32 xl, nl, %9;\n\t"                                                      \
    "shr.s32 xr, nr, 1;\n\t"                                                          \
    "lop3.b32 f0, nc, xl, xr, 0x01;\n\t"                                              \
    "neg.s32 t, f0;\n\t"                                                              \
    "and.b32 lo, t, f0;\n\t"                                                          \
    "mul.lo.s32 ma, lo, %13;\n\t"                                                     \
    "bfind.shiftamt.u32 pos, f0;\n\t"                                                 \
    "shr.b32 mb, %12, pos;\n\t"                                                       \
    "popc.b32 pc, nc;\n\t"                                                            \
    "setp.ne.and.u32 pg, pc, %14, pb;\n\t"                                            \
    "setp.eq.and.u32 p2, pc, %14, pb;\n\t"

#define NQB_STEP4_LOOK                                                                \
    "mul.lo.s32 t, xl, %9;\n\t"                                                       \
    "shr.s32 pos, xr, 1;\n\t"                                                         \
    "lop3.and.b32 t|pg, nc, t, pos, 0x01, pg;\n\t"

#define NQB_STEP4_TAIL                                                                \
    "lop3.and.b32 naf|pd, na, ma, mb, 0xE0, pg;\n\t"                                  \
    "popc.b32 t, naf;\n\t"                                                            \
    "@p2 mad.lo.s32 %5, t, %8, %5;\n\t"                                               \
    "lop3.or.b32 %3|pk, %3, bit, 0, 0x3C, pd;\n\t"                                    \
    "setp.ne.and.u32 pp, %3, 0, pd;\n\t"                                              \
    "@pp st.shared.v4.u32 [%4], {%0, %1, %2, %3};\n\t"                                \
    "@pp mad.lo.s32 %4, %8, %11, %4;\n\t"                                             \
    "@pd mul.lo.s32 %0, nc, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %1, xl, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %2, xr, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %3, naf, %8;\n\t"                                                 \
    "setp.ne.and.u32 pq, %4, %7, !pk;\n\t"                                            \
    "@pq mad.lo.s32 %4, %10, %11, %4;\n\t"                                            \
    "@pq ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t"

#define NQB_STEP4 NQB_STEP4_CHILD NQB_STEP4_LOOK NQB_STEP4_TAIL
#define NQB_STEP4_X4 NQB_STEP4 NQB_STEP4 NQB_STEP4 NQB_STEP4

// VAR 6: VAR 4 in place, the default.  VAR 4 computes a child beside its parent
// and moves it over (four predicated moves) if it is entered.  Here the parent's
// remaining columns are pushed first, whether the child lives or not, the child
// is computed in the level's own registers, and a child that is not entered
// (dead, or counted on row N-2) is undone by the pop that a finished level needs
// anyway.  30 operations instead of 34, for more stack traffic: a step pushes
// whenever columns remain (38 % of the steps, VAR 4 27 %), and one more slot, for
// the push on row N-3.  A lane without work must stay without: a step that enters
// nothing clears avail before the pop, which only a lane with a stacked level
// does.  Bound by issue (82 %; ALU 77 %, FMA 58 %, shared-memory wavefronts 74 %
// at N=18).  N=19, k=6 145.2 -> 132.1 ms, 1.1e6
// prefixes of N=18 18.5 -> 17.5 ms, 8 % of N=21's 839 -> 757 ms.
// Launches whose stated CTA size and stack depth leave no room for that slot run
// VAR 4, and so do the resumable kernels.
#define NQB_STEP6_HEAD                                                                \
    "{\n\t"                                                                           \
    ".reg .pred pt1, pb, pg, p2, pd, pp, pq;\n\t"                                     \
    ".reg .b32 t, bit, na, f0, lo, ma, mb, pos, pc;\n\t"                              \
    "setp.ne.u32 pt1, %8, 0;\n\t"

#define NQB_STEP6_PUSH                                                                \
    "mul.lo.s32 t, %3, %10;\n\t"                                                      \
    "lop3.and.b32 bit|pb, t, %3, 0, 0xC0, pt1;\n\t"                                   \
    "lop3.and.b32 %3|pp, %3, bit, 0, 0x3C, pt1;\n\t"                                  \
    "@pp st.shared.v4.u32 [%4], {%0, %1, %2, %3};\n\t"                                \
    "@pp mad.lo.s32 %4, %8, %11, %4;\n\t"                                             \
    "mad.lo.s32 %0, bit, %8, %0;\n\t"                                                 \
    "mad.lo.s32 %1, bit, %9, %1;\n\t"                                                 \
    "shr.u32 t, bit, 1;\n\t"                                                          \
    "add.u32 %2, t, %2;\n\t"                                                          \
    "lop3.b32 na, %0, %1, %2, 0x01;\n\t"                                              \
    "mul.lo.s32 %1, %1, %9;\n\t"                                                      \
    "shr.s32 %2, %2, 1;\n\t"                                                          \
    "lop3.b32 f0, %0, %1, %2, 0x01;\n\t"                                              \
    "popc.b32 pc, %0;\n\t"                                                            \
    "setp.eq.and.u32 p2, pc, 30, pb;\n\t"

// a child on row N-2 is counted and not entered
#define NQB_STEP6_GATE "setp.ne.and.u32 pg, pc, 30, pb;\n\t"

// the masks of the alive columns, from F0
#define NQB_STEP6_ALIVE                                                               \
    "neg.s32 t, f0;\n\t"                                                              \
    "and.b32 lo, t, f0;\n\t"                                                          \
    "mul.lo.s32 ma, lo, -4;\n\t"                                                      \
    "bfind.shiftamt.u32 pos, f0;\n\t"                                                 \
    "shr.b32 mb, 0x3fffffff, pos;\n\t"

#define NQB_STEP6_LOOK                                                                \
    "mul.lo.s32 t, %1, %9;\n\t"                                                       \
    "shr.s32 pos, %2, 1;\n\t"                                                         \
    "lop3.and.b32 t|pg, %0, t, pos, 0x01, pg;\n\t"

// VAR 7, the count kernels with per-owner outputs: VAR 6 without the gate.  A
// counted child on row N-2 is entered too when its row two below (there is none)
// looks free; its level finds no alive column and ends.  One ALU operation fewer
// on every step for about 1 % more steps, and a second extra slot (for the push on
// row N-2).  1.1e6 prefixes of N=18 with per-task counts 17.24 -> 16.69 ms, 1.8e6 of N=19
// 128.2 -> 125.6 ms; in the kernel without per-owner outputs the same step issues
// 80.9 instead of 84.4 % of the slots and is slower (126.8 -> 129.8 ms), so that
// one keeps the gate.
#define NQB_STEP7_LOOK                                                                \
    "mul.lo.s32 t, %1, %9;\n\t"                                                       \
    "shr.s32 pos, %2, 1;\n\t"                                                         \
    "lop3.and.b32 t|pg, %0, t, pos, 0x01, pb;\n\t"

// Node counts (%6): a level's placements are its free columns, dead ones
// included, so a step adds the size of its child's unfiltered list (the root
// level's is added when a task is loaded), and rows N-2 and N-1 and dead
// children need no steps of their own.  No look-ahead: a child whose row two
// below is full still has placements on the row between.  29 operations on 0.63
// steps per node where a step per placement took 21 on one, and fewer stack
// accesses, which bound that form (shared-memory wavefronts 65 %).  300,007 prefixes
// of N=17, k=6: the whole call 3.39 ms so, 3.01 with VAR 4's form, 2.78 in place.
#define NQB_STEP6_NODES                                                               \
    "popc.b32 t, na;\n\t"                                                             \
    "@pb mad.lo.s32 %6, t, %8, %6;\n\t"

#define NQB_STEP6_CHILD                                                               \
    "lop3.and.b32 %3|pd, na, ma, mb, 0xE0, pg;\n\t"                                   \
    "popc.b32 t, %3;\n\t"

#define NQB_STEP6_POP                                                                 \
    "@!pd mov.b32 %3, 0;\n\t"                                                         \
    "setp.ne.and.u32 pq, %4, %7, !pd;\n\t"                                            \
    "@pq mad.lo.s32 %4, %10, %11, %4;\n\t"                                            \
    "@pq ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t"

#define NQB_STEP6_COUNT "@p2 mad.lo.s32 %5, t, %8, %5;\n\t"
#define NQB_STEP6 \
    NQB_STEP6_PUSH NQB_STEP6_GATE NQB_STEP6_ALIVE NQB_STEP6_LOOK NQB_STEP6_CHILD NQB_STEP6_COUNT NQB_STEP6_POP
#define NQB_STEP6N \
    NQB_STEP6_PUSH NQB_STEP6_GATE NQB_STEP6_ALIVE NQB_STEP6_NODES NQB_STEP6_CHILD NQB_STEP6_COUNT NQB_STEP6_POP
#define NQB_STEP7 \
    NQB_STEP6_PUSH NQB_STEP6_ALIVE NQB_STEP7_LOOK NQB_STEP6_CHILD NQB_STEP6_COUNT NQB_STEP6_POP
#define NQB_STEP6_X4 NQB_STEP6 NQB_STEP6 NQB_STEP6 NQB_STEP6
#define NQB_STEP6_X16 NQB_STEP6_X4 NQB_STEP6_X4 NQB_STEP6_X4 NQB_STEP6_X4
#define NQB_STEP7_X4 NQB_STEP7 NQB_STEP7 NQB_STEP7 NQB_STEP7
#define NQB_STEP7_X16 NQB_STEP7_X4 NQB_STEP7_X4 NQB_STEP7_X4 NQB_STEP7_X4
#define NQB_STEP6N_X4 NQB_STEP6N NQB_STEP6N NQB_STEP6N NQB_STEP6N

// DIH4, the resumable dihedral kernel's step: the class rules of the lane's task,
//   pc = popc(child cols) = 32 - N + child row
//   pc > %12            -> the child row may not use the side columns, and
//                          when it is row N-1 (pc == 31) only %13's columns
//   child cols == ~0    -> one completion of weight %16 if the row N-1 queen
//                          is at %14, else %15
// with the left diagonal pre-shifted and each child's list cut to its alive
// columns (those whose next row keeps a free column, ignoring the class rules --
// the rules only remove columns, so this drops dead children only) except on row
// N-1, whose columns complete the board.  Rows N-2 and N-1 are stepped, because the
// class rules and the tie weight decide what their completions count, and because
// checkpoints hold levels on those rows.
// Operands %0-%11 as in the plain step; %12 popc threshold, %13 row N-1 mask, %14
// tie column bit, %15 weight, %16 tie weight, %17 ~side columns.
#define NQB_STEP_HEAD_DIH4                                                            \
    "{\n\t"                                                                           \
    ".reg .pred pb, pd, pp, pe, pq, pq0, ps, pl, px;\n\t"                              \
    ".reg .b32 t, bit, nc, nl, nr, na, pc, msk, w, xl, xr, f0, lo, ma, mb, pos;\n\t"  \

#define NQB_STEP_DIH4                                                                 \
    "mul.lo.s32 t, %3, %10;\n\t"                                                      \
    "and.b32 bit, t, %3;\n\t"                                                         \
    "setp.ne.u32 pb, bit, 0;\n\t"                                                     \
    "mad.lo.s32 %3, bit, %10, %3;\n\t"                                                \
    "mad.lo.s32 nc, bit, %8, %0;\n\t"                                                 \
    "mad.lo.s32 nl, bit, %9, %1;\n\t"                                                 \
    "or.b32 nr, %2, bit;\n\t"                                                         \
    "shr.s32 nr, nr, 1;\n\t"                                                          \
    "lop3.b32 na, nc, nl, nr, 0x01;\n\t"                                              \
    "popc.b32 pc, nc;\n\t"                                                            \
    "setp.gt.u32 ps, pc, %12;\n\t"                                                    \
    "setp.eq.u32 pl, pc, 31;\n\t"                                                     \
    "selp.b32 msk, %13, %17, pl;\n\t"                                                 \
    "@ps and.b32 na, na, msk;\n\t"                                                    \
    "mul.lo.s32 xl, nl, %9;\n\t"                                                      \
    "shr.s32 xr, nr, 1;\n\t"                                                          \
    "lop3.b32 f0, nc, xl, xr, 0x01;\n\t"                                              \
    "mul.lo.s32 t, f0, %10;\n\t"                                                      \
    "and.b32 lo, t, f0;\n\t"                                                          \
    "mul.lo.s32 ma, lo, -4;\n\t"                                                      \
    "bfind.u32 pos, f0;\n\t"                                                          \
    "mad.lo.s32 pos, pos, %10, 33;\n\t"                                               \
    "shr.b32 mb, %10, pos;\n\t"                                                       \
    "@!pl lop3.b32 na, na, ma, mb, 0xE0;\n\t"                                         \
    "setp.ne.and.u32 pd, na, 0, pb;\n\t"                                              \
    "setp.eq.u32 pe, nc, 0xffffffff;\n\t"                                             \
    "setp.eq.u32 px, bit, %14;\n\t"                                                   \
    "selp.b32 w, %16, %15, px;\n\t"                                                   \
    "@pe mad.lo.s32 %5, w, %8, %5;\n\t"                                               \
    "setp.ne.and.u32 pp, %3, 0, pd;\n\t"                                              \
    "setp.eq.and.u32 pq0, %3, 0, !pd;\n\t"                                            \
    "@pp st.shared.v4.u32 [%4], {%0, %1, %2, %3};\n\t"                                \
    "@pp mad.lo.s32 %4, %8, %11, %4;\n\t"                                             \
    "@pd mul.lo.s32 %0, nc, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %1, xl, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %2, nr, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %3, na, %8;\n\t"                                                  \
    "setp.ne.and.u32 pq, %4, %7, pq0;\n\t"                                            \
    "@pq mad.lo.s32 %4, %10, %11, %4;\n\t"                                            \
    "@pq ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t"                                \
    "}\n\t"

// VAR 5, the dihedral kernels' default: VAR 4's step (both diagonals
// pre-shifted, alive columns, row N-2 counted, look-ahead) under the class rules.
//  * Side columns barred past side_row: whoever enters such a row with a side
//    column still unused can never complete the board (every column needs a
//    queen), so the child's list becomes empty; with both used no list holds
//    them.  One compare, one LOP3 with a predicate, one predicated move, as many
//    as masking the list took, and 8 % fewer nodes (N=16..17, k=6).
//  * Row N-1's columns: a child on row N-2 masks the free columns of row N-1
//    (F0) with them before its alive columns are taken; its completions are then
//    its alive columns, as in VAR 4 (the mask is all ones in the classes that do
//    not bar row N-1).
//  * Weights: each completion weighs w, and the one whose row N-1 queen stands
//    at the tie column weighs w + dw; there is one when the tie column is unused
//    and a column other than it is alive.
// A counted child on row N-2 may be entered too (see VAR 7); its level finds no
// alive column and ends.  40 operations, as the form above, on fewer steps (0.85 at N=11, CPU
// model).  Bound by issue (84 %, was 79 %) and the ALU pipe.  N=19, k=6, a whole
// call: 132.1 ms with the form above, 108.7 with the compare that keeps row N-2
// out, 106.2 without it (in place, as VAR 6, it is no faster).  Operands as above,
// with %16 the tie's extra weight dw.
#define NQB_STEP5_HEAD                                                                \
    "{\n\t"                                                                           \
    ".reg .pred pt1, pb, pg, p2, pd, pk, pp, pq, ps;\n\t"                             \
    ".reg .b32 t, bit, nc, nl, nr, na, xl, xr, f0, lo, ma, mb, pos, pc, naf;\n\t"     \
    "setp.ne.u32 pt1, %8, 0;\n\t"

#define NQB_STEP5                                                                     \
    "mul.lo.s32 t, %3, %10;\n\t"                                                      \
    "lop3.and.b32 bit|pb, t, %3, 0, 0xC0, pt1;\n\t"                                   \
    "mad.lo.s32 nc, bit, %8, %0;\n\t"                                                 \
    "mad.lo.s32 nl, bit, %9, %1;\n\t"                                                 \
    "shr.u32 nr, bit, 1;\n\t"                                                         \
    "add.u32 nr, nr, %2;\n\t"                                                         \
    "lop3.b32 na, nc, nl, nr, 0x01;\n\t"                                              \
    "mul.lo.s32 xl, nl, %9;\n\t"                                                      \
    "shr.s32 xr, nr, 1;\n\t"                                                          \
    "lop3.b32 f0, nc, xl, xr, 0x01;\n\t"                                              \
    "popc.b32 pc, nc;\n\t"                                                            \
    "setp.eq.and.u32 p2, pc, 30, pb;\n\t"                                             \
    "setp.gt.u32 ps, pc, %12;\n\t"                                                    \
    "lop3.and.b32 t|ps, nc, %17, 0, 0x03, ps;\n\t"                                    \
    "@ps mul.lo.s32 na, na, 0;\n\t"                                                   \
    "@p2 and.b32 f0, f0, %13;\n\t"                                                    \
    "neg.s32 t, f0;\n\t"                                                              \
    "and.b32 lo, t, f0;\n\t"                                                          \
    "mul.lo.s32 ma, lo, -4;\n\t"                                                      \
    "bfind.shiftamt.u32 pos, f0;\n\t"                                                 \
    "shr.b32 mb, 0x3fffffff, pos;\n\t"                                                \
    "mul.lo.s32 t, xl, %9;\n\t"                                                       \
    "shr.s32 pos, xr, 1;\n\t"                                                         \
    "lop3.and.b32 t|pg, nc, t, pos, 0x01, pb;\n\t"                                    \
    "lop3.and.b32 naf|pd, na, ma, mb, 0xE0, pg;\n\t"                                  \
    "popc.b32 t, naf;\n\t"                                                            \
    "@p2 mad.lo.s32 %5, t, %15, %5;\n\t"                                              \
    "lop3.and.b32 t|p2, %14, nc, 0, 0x30, p2;\n\t"                                    \
    "lop3.and.b32 t|p2, naf, %14, 0, 0x30, p2;\n\t"                                   \
    "@p2 mad.lo.s32 %5, %16, %8, %5;\n\t"                                             \
    "lop3.or.b32 %3|pk, %3, bit, 0, 0x3C, pd;\n\t"                                    \
    "setp.ne.and.u32 pp, %3, 0, pd;\n\t"                                              \
    "@pp st.shared.v4.u32 [%4], {%0, %1, %2, %3};\n\t"                                \
    "@pp mad.lo.s32 %4, %8, %11, %4;\n\t"                                             \
    "@pd mul.lo.s32 %0, nc, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %1, xl, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %2, xr, %8;\n\t"                                                  \
    "@pd mul.lo.s32 %3, naf, %8;\n\t"                                                 \
    "setp.ne.and.u32 pq, %4, %7, !pk;\n\t"                                            \
    "@pq mad.lo.s32 %4, %10, %11, %4;\n\t"                                            \
    "@pq ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t"

#define NQB_STEP5_X4 NQB_STEP5 NQB_STEP5 NQB_STEP5 NQB_STEP5

// Class registers of a lane in a DIH kernel (cls: the class index, kept for
// the deadline dump of resumable runs).
struct DihLane {
    uint32_t side_popc = 64u, last_mask = ~0u, tie_bit = 0u, w = 0u, w_tie = 0u, cls = 0u;
};

struct StepConsts {
    uint32_t one, two, mone, stride;  // stride: bytes between a lane's consecutive stack slots
};

// Step variants: of the count kernels ...
constexpr int kStepVar = 6;
// ... with per-owner outputs
constexpr int kOwnerStepVar = 7;
// ... that count DFS nodes
constexpr int kNodesStepVar = 6;
// ... of launches without room for the extra slots of 6 and 7, and of the resumable
// kernel, whose stated stack depth leaves none either;
constexpr int kTightStepVar = 4;
// of the dihedral kernels, and of the resumable one (DIH4)
constexpr int kDihStepVar = 5;
constexpr int kDihResumeStepVar = 4;

// Stack rows a step variant never pushes beyond the reference's N-1-rows: VAR 4
// enters no level on row N-2 or N-1 and pushes what it leaves for a child, so the
// deepest level it pushes is on row N-4; VAR 5 and 6 push on row N-3 too, VAR 7 on
// row N-2.
template <int VAR>
constexpr int kStackRowsSpared = VAR == 4 ? 2 : VAR == 5 || VAR == 6 ? 1 : 0;

// Lane registers (ld, rd) from the reference's (left, right) masks of the row
// a level enumerates, and back (for the checkpoint file, which stores the
// reference's form).  Going back loses left's bit 31 and right's bit 0, which
// no later row can see (left bits only move further left, right bits further
// right, and the level's own untried columns are stored beside them).  DIH4 keeps
// the right mask as it is (PRE_RD false).
__device__ __forceinline__ uint32_t lane_ld(uint32_t left) { return left << 1; }
__device__ __forceinline__ uint32_t ref_ld(uint32_t ld) { return ld >> 1; }
template <bool PRE_RD>
__device__ __forceinline__ uint32_t lane_rd(uint32_t right) {
    return PRE_RD ? (uint32_t)((int32_t)right >> 1) : right;
}
template <bool PRE_RD>
__device__ __forceinline__ uint32_t ref_rd(uint32_t rd) { return PRE_RD ? rd << 1 : rd; }

// The alive part of a level's untried columns (VAR 4): drops every column
// whose child would leave the next row without a free column.  ld and rd in
// VAR 4's lane form (pre-shifted).
__device__ __forceinline__ uint32_t alive_columns(uint32_t cols, uint32_t ld, uint32_t rd, uint32_t avail) {
    const uint32_t f0 = ~(cols | ld | rd);
    if (f0 == 0) return 0;
    const uint32_t lo = f0 & (0u - f0);
    const int hi = 31 - __clz(f0);
    const uint32_t above = 0u - (lo << 2);                              // columns >= lowest + 2
    const uint32_t below = hi >= 2 ? (0xffffffffu >> (33 - hi)) : 0u;  // columns <= highest - 2
    return avail & (above | below);
}

// One step of DIH4.
__device__ __forceinline__ void dfs_step_dih(uint32_t &cols, uint32_t &ld, uint32_t &rd, uint32_t &avail, uint32_t &sp,
                                             uint32_t &cnt, uint32_t &it, uint32_t bot, const StepConsts &k,
                                             const DihLane &d, uint32_t noside) {
    asm volatile(NQB_STEP_HEAD_DIH4 NQB_STEP_DIH4
                 : "+r"(cols), "+r"(ld), "+r"(rd), "+r"(avail), "+r"(sp), "+r"(cnt), "+r"(it)
                 : "r"(bot), "r"(k.one), "r"(k.two), "r"(k.mone), "r"(k.stride), "r"(d.side_popc),
                   "r"(d.last_mask), "r"(d.tie_bit), "r"(d.w), "r"(d.w_tie), "r"(noside)
                 : "memory");
}

// UNROLL steps of VAR 4 (no NODES form), four per asm block.  Operand %6 is
// unused (it stands where the node counter sits in the other forms).
template <int UNROLL>
__device__ __forceinline__ void dfs_steps4(uint32_t &cols, uint32_t &ld, uint32_t &rd, uint32_t &avail, uint32_t &sp,
                                           uint32_t &cnt, uint32_t bot, const StepConsts &k) {
    static_assert(UNROLL % 4 == 0, "VAR 4 unrolls in groups of 4");
#pragma unroll
    for (int g = 0; g < UNROLL / 4; ++g)
        asm volatile(NQB_STEP4_HEAD NQB_STEP4_X4 "}\n\t"
                     : "+r"(cols), "+r"(ld), "+r"(rd), "+r"(avail), "+r"(sp), "+r"(cnt)
                     : "r"(0u), "r"(bot), "r"(k.one), "r"(k.two), "r"(k.mone), "r"(k.stride), "r"(0x3fffffffu),
                       "r"(0xfffffffcu), "r"(30u)
                     : "memory");
}

// UNROLL steps of VAR 6 or 7, sixteen per asm block where UNROLL allows, else
// four.  Operand %6, the node counter, is used by the NODES form (VAR 6) only.
#define NQB_RUN_STEPS(TEXT)                                                                                     \
    asm volatile(NQB_STEP6_HEAD TEXT "}\n\t"                                                                    \
                 : "+r"(cols), "+r"(ld), "+r"(rd), "+r"(avail), "+r"(sp), "+r"(cnt)                             \
                 : "r"(0u), "r"(bot), "r"(k.one), "r"(k.two), "r"(k.mone), "r"(k.stride)                        \
                 : "memory")
template <int VAR, bool NODES, int UNROLL>
__device__ __forceinline__ void dfs_steps6(uint32_t &cols, uint32_t &ld, uint32_t &rd, uint32_t &avail, uint32_t &sp,
                                           uint32_t &cnt, uint32_t &it, uint32_t bot, const StepConsts &k) {
    static_assert(UNROLL % 4 == 0, "VAR 6 and 7 unroll in groups of 4 or 16");
    constexpr int kGroup = UNROLL % 16 == 0 && !NODES ? 16 : 4;
#pragma unroll
    for (int g = 0; g < UNROLL / kGroup; ++g) {
        if constexpr (NODES)
            asm volatile(NQB_STEP6_HEAD NQB_STEP6N_X4 "}\n\t"
                         : "+r"(cols), "+r"(ld), "+r"(rd), "+r"(avail), "+r"(sp), "+r"(cnt), "+r"(it)
                         : "r"(bot), "r"(k.one), "r"(k.two), "r"(k.mone), "r"(k.stride)
                         : "memory");
        else if constexpr (VAR == 7 && kGroup == 16)
            NQB_RUN_STEPS(NQB_STEP7_X16);
        else if constexpr (VAR == 7)
            NQB_RUN_STEPS(NQB_STEP7_X4);
        else if constexpr (kGroup == 16)
            NQB_RUN_STEPS(NQB_STEP6_X16);
        else
            NQB_RUN_STEPS(NQB_STEP6_X4);
    }
}
#undef NQB_RUN_STEPS

// UNROLL steps of VAR 5, four per asm block.
template <int UNROLL>
__device__ __forceinline__ void dfs_steps5(uint32_t &cols, uint32_t &ld, uint32_t &rd, uint32_t &avail, uint32_t &sp,
                                           uint32_t &cnt, uint32_t &it, uint32_t bot, const StepConsts &k,
                                           const DihLane &d, uint32_t noside) {
    static_assert(UNROLL % 4 == 0, "VAR 5 unrolls in groups of 4");
    const uint32_t dw = d.w_tie - d.w;
#pragma unroll
    for (int g = 0; g < UNROLL / 4; ++g)
        asm volatile(NQB_STEP5_HEAD NQB_STEP5_X4 "}\n\t"
                     : "+r"(cols), "+r"(ld), "+r"(rd), "+r"(avail), "+r"(sp), "+r"(cnt), "+r"(it)
                     : "r"(bot), "r"(k.one), "r"(k.two), "r"(k.mone), "r"(k.stride), "r"(d.side_popc),
                       "r"(d.last_mask), "r"(d.tie_bit), "r"(d.w), "r"(dw), "r"(noside)
                     : "memory");
}

// UNROLL steps of a kernel.
template <int VAR, bool NODES, bool DIH, int UNROLL>
__device__ __forceinline__ void dfs_steps(uint32_t &cols, uint32_t &ld, uint32_t &rd, uint32_t &avail, uint32_t &sp,
                                          uint32_t &cnt, uint32_t &it, uint32_t bot, const StepConsts &k,
                                          const DihLane &d, uint32_t noside) {
    if constexpr (VAR == 5) {
        dfs_steps5<UNROLL>(cols, ld, rd, avail, sp, cnt, it, bot, k, d, noside);
    } else if constexpr (DIH) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) dfs_step_dih(cols, ld, rd, avail, sp, cnt, it, bot, k, d, noside);
    } else if constexpr (VAR == 4) {
        dfs_steps4<UNROLL>(cols, ld, rd, avail, sp, cnt, bot, k);
    } else {
        dfs_steps6<VAR, NODES, UNROLL>(cols, ld, rd, avail, sp, cnt, it, bot, k);
    }
}

__device__ __forceinline__ void load_class_index(const DfsParams &p, uint32_t idx, DihLane &d) {
    const uint4 c = __ldg(p.cls_tab + idx);
    d.cls = idx;
    d.side_popc = c.x;
    d.last_mask = c.y;
    d.tie_bit = c.z;
    d.w = c.w & 0xffffu;
    d.w_tie = c.w >> 16;
}

__device__ __forceinline__ void load_class(const DfsParams &p, long long t, DihLane &d) {
    load_class_index(p, __ldg(p.task_cls + t), d);
}

// VAR 4 and 6 keep only levels on rows 0..N-3, with their alive columns.  A level
// on row N-1 (one column left) completes once per free column; on row N-2
// once per alive column.  Returns those completions and leaves avail = 0 for
// such levels; otherwise filters avail and returns 0.
__device__ __forceinline__ uint32_t settle_level(int n, uint32_t cols, uint32_t ld, uint32_t rd, uint32_t &avail) {
    const int row = __popc(cols) - (32 - n);
    if (row >= n - 1) {
        const uint32_t done = __popc(avail);
        avail = 0;
        return done;
    }
    avail = alive_columns(cols, ld, rd, avail);
    if (row == n - 2) {
        const uint32_t done = __popc(avail);
        avail = 0;
        return done;
    }
    return 0;
}

// The same for VAR 5: weighted completions of a level on rows N-2 and N-1, whose
// avail already follows the class rules of its own row.
__device__ __forceinline__ uint32_t settle_level_dih(int n, uint32_t cols, uint32_t ld, uint32_t rd, uint32_t &avail,
                                                     const DihLane &d) {
    const int row = __popc(cols) - (32 - n);
    if (row >= n - 1) {
        const uint32_t done = (avail & ~d.tie_bit) ? d.w : avail ? d.w_tie : 0u;  // one column at most
        avail = 0;
        return done;
    }
    const bool n2 = row == n - 2;
    // columns that row N-1 may not use count as taken there
    avail = alive_columns(cols, ld | (n2 ? ~d.last_mask : 0u), rd, avail);
    if (!n2) return 0;
    const uint32_t done = __popc(avail) * d.w + ((d.tie_bit & ~cols) && (avail & ~d.tie_bit) ? d.w_tie - d.w : 0u);
    avail = 0;
    return done;
}

// Loads task t into a lane.  Returns the completions credited immediately
// (1 for an already-complete board) and leaves avail == 0 when the task has
// no free column.  A column mask with off-board bits can never equal `last`,
// so such a task counts 0, exactly as the reference recursion does.
// VAR 4 and 6: `placed` receives the columns whose placements the nodes of the task's
// own row are (its free columns on rows before N-1).
// SPARED: the rows by which the launch's stack may fall short of N-1-popc(cols).
template <bool PRE_RD, bool SETTLE, int SPARED>
__device__ __forceinline__ uint32_t load_task(const DfsParams &p, long long t, uint32_t &cols, uint32_t &ld,
                                              uint32_t &rd, uint32_t &avail, uint32_t &placed) {
    const int n = p.task_n ? (int)p.task_n[t] : p.N;
    const uint32_t last = (n >= 32) ? kFull : ((1u << n) - 1u);
    const uint32_t c = __ldg(p.cols + t);
    const uint32_t l = __ldg(p.ld + t);
    const uint32_t r = __ldg(p.rd + t);
    avail = 0;
    if (c & ~last) return 0;
    if (c == last) return 1;
    const int need = n - 1 - __popc(c) - SPARED;
    if (need > p.levels) {
        atomicOr(p.ctl + kCtlError, kErrDepth);
        return 0;
    }
    cols = c | ~last;
    ld = lane_ld(l);
    rd = lane_rd<PRE_RD>(r);
    avail = ~(cols | l | r);
    if (SETTLE) {
        placed = __popc(c) < n - 1 ? avail : 0u;
        return settle_level(n, cols, ld, rd, avail);
    }
    return 0;
}

// The columns of share `way` when a level's untried columns are dealt out in
// 2^lg shares (by column number modulo 2^lg).
__device__ __forceinline__ uint32_t share_mask(uint32_t lg, uint32_t way) {
    uint32_t m = kFull;
    if (lg > 0) m = 0x55555555u;
    if (lg > 1) m = 0x11111111u;
    if (lg > 2) m = 0x01010101u;
    if (lg > 3) m = 0x00010001u;
    if (lg > 4) m = 0x00000001u;
    return m << way;
}

// ---------------------------------------------------------------------------
// Mailbox: work sharing between warps once the queue is empty.
//
// A warp that is wholly out of work takes a ticket (kCtlMail, low half) and
// watches the slot of that number.  A warp that has stacked levels and sees
// more tickets requested than supplied claims a supply number (high half) and
// posts up to kMailLevels of its lanes' bottom (shallowest, largest) levels
// into that slot.  Slot i thus belongs to ticket i, whoever comes first.
//
// The slots are a ring of mail_cap (a power of two) entries: ticket t lives in
// slot t % mail_cap as its (t / mail_cap)-th use, which the state word carries
// above the kMail* value; its taker readies the slot for the next use.  A warp
// holds one open ticket and claims one number at a time, so fewer than twice
// the grid's warps are live at once, which is below mail_cap.  Should a slot come
// round while its last taker still reads (a warp that stood still while the
// whole ring went by), its next waiter stays until that is over, so that no level is posted to
// a ticket that was given up unseen (tests/test_mailbox_model.py).
//
// kCtlWork counts, as a signed number, slots posted and not yet taken minus
// warps out of work; with the grid's warps added it is the number of parties
// that still hold work.  The warp that brings it to zero tells every waiting
// ticket (kMailDone).  A post is counted before it is made and its taker counts
// as working from then on, so the sum reaches zero only when nothing is left;
// the last CTA checks that (kStatMail).
//
// What it is worth beside the queue's shares (launch.h): 512 boards of N=12..17
// split three rows deep 7.7 ms, 24 without the mailbox (single subtrees of 4.5e6
// nodes sit in one warp); 8 % of N=21's prefixes (2.1 tasks per lane) 751 ms, 790
// without.  Levels with fewer than kMailMinRows rows left cost more to hand over (a
// ticket, a post and a poll, about 3 us, then a warp that starts with a few lanes)
// than they hold: with 10 instead of 12 the batch takes 7.9 ms.  For the same
// reason launches whose deepest task has fewer
// than kMailRootRows rows left run without (60,001 prefixes of N=16, k=5: 0.51 ms
// without, 0.65 with).  A list in device memory whose depth is not stated is looked
// through first (deepest_task_kernel, 2-3 us).  With the stack depth, an empty
// board's, in its place 8000 prefixes of N=13, k=5 took 99 us a call instead of 74,
// 300,007 of N=17, k=6 1.52 ms instead of 1.31.
//
// No count depends on the waiting: a waiter only watches its own slot, gives
// up after mail_patience_ns (it marks the slot kMailGone, so the supplier keeps
// its levels) and then just ends.  CTAs that have not started count as working
// and, when they start, find the queue as any other warp does.
constexpr uint32_t kMailPatienceNs = 20u * 1000 * 1000;
constexpr int kMailPolls = 1 << 16;   // second limit on a wait, in polls
constexpr int kMailRootRows = 13;      // rows left in the deepest task from which a launch uses the mailbox
constexpr uint32_t kMailMinRows = 12;  // rows left below which a level is not worth posting
constexpr uint32_t kGiveMinRows = 8;   // the same for a level given to a lane of the same warp
// Once the queue is empty a warp looks at its idle lanes after kTailTrip DFS
// steps, or as soon as kTailIdle lanes are idle: a look (donation, mailbox) costs
// about 290 instructions, ten steps, and with one at every newly idle lane they
// were a quarter of all instructions of a batch.  512 boards of N=12..17 9.1 ms
// with a look per idle lane, 8.2 at 8 lanes and 64 steps, 7.7 at 12 and 96; 60,001
// prefixes of N=16 500, 485, 484 us.  The loop of a
// live queue keeps its plain any-vote: counting the lanes there costs 6 % (N=19).
constexpr int kTailTrip = 96;
constexpr int kTailIdle = 12;

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *a) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ MailSlot *mail_slot(const DfsParams &p, uint32_t t) {
    return p.mail + (t & (p.mail_cap - 1u));
}
__device__ __forceinline__ uint32_t mail_tag(const DfsParams &p, uint32_t t, uint32_t st) {
    return (t / p.mail_cap) << 2 | st;
}

// Whether this launch uses the mailbox (the same answer in all of its warps).
__device__ __forceinline__ bool mail_on(const DfsParams &p) {
    return p.mail && p.steal && (!p.mail_gate || __ldg(p.mail_gate) >= (uint32_t)kMailRootRows);
}

// Counts this warp as out of work; the last one to be so ends every wait.
// Returns true for that one.
__device__ __forceinline__ bool out_of_work(const DfsParams &p, uint32_t lane) {
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    unsigned long long old = 0;
    if (lane == 0) {
        __threadfence();
        old = atomicAdd(p.ctl + kCtlWork, ~0ull);
        __threadfence();
    }
    old = __shfl_sync(kFull, old, 0);
    if ((long long)old - 1 + nwarps != 0) return false;
    const unsigned long long tk = *((volatile unsigned long long *)(p.ctl + kCtlMail));
    const uint32_t req = (uint32_t)tk;
    for (uint32_t i = (uint32_t)(tk >> 32) + lane; i < req; i += 32)
        atomicCAS(&mail_slot(p, i)->state, mail_tag(p, i, kMailEmpty), mail_tag(p, i, kMailDone));
    return true;
}

// For a warp that is out of work: takes a ticket and waits for its slot.  True:
// the lanes hold the posted levels, each dealt out over several lanes by its
// untried columns.  False: the warp is to end.
template <bool DIH>
__device__ __forceinline__ bool take_mail(const DfsParams &p, uint32_t lane, uint32_t &cols, uint32_t &ld,
                                          uint32_t &rd, uint32_t &avail, uint32_t &owner, DihLane &dih) {
    uint32_t t = 0, got = 0;
    unsigned long long t0 = 0;
    if (p.cta_times) t0 = globaltimer_ns();
    if (lane == 0) t = (uint32_t)atomicAdd(p.ctl + kCtlMail, 1ull);
    t = __shfl_sync(kFull, t, 0);
    if (out_of_work(p, lane)) return false;
    MailSlot *s = mail_slot(p, t);
    const uint32_t none = mail_tag(p, t, kMailEmpty);
    if (lane == 0) {
        const unsigned long long until = globaltimer_ns() + p.mail_patience_ns;
        uint32_t st = none;
        unsigned nap = 100;
        for (int i = 0; i < kMailPolls; ++i) {
            st = ld_acquire(&s->state);
            if (st > none || (st == none && globaltimer_ns() > until)) break;
            __nanosleep(nap);
            nap = min(nap * 2, 1000u);
        }
        if (st <= none) st = atomicCAS(&s->state, none, none | kMailGone);
        if (st == (none | kMailFull)) {
            __threadfence();
            got = __ldcg(&s->count);
        }
        if (p.cta_times) atomicAdd(p.cta_wait + blockIdx.x, globaltimer_ns() - t0);
    }
    got = __shfl_sync(kFull, got, 0);
    __syncwarp();
    if (got == 0) return false;
    // got levels over 32 lanes: 2^lg lanes for each
    const uint32_t lg = 31u - __clz(32u / got);
    const uint32_t e = lane >> lg;
    if (e < got) {
        const uint4 v = __ldcg(s->level + e);
        cols = v.x;
        ld = v.y;
        rd = v.z;
        avail = v.w & share_mask(lg, lane & ((1u << lg) - 1u));
        owner = avail ? __ldcg(s->owner + e) : kNoOwner;
        if (DIH) load_class_index(p, __ldcg(s->cls + e), dih);
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicExch(&s->state, none + 4u);  // ready for the slot's next use
    return true;
}

// Offers this warp's shallowest stacked levels to a waiting warp; returns 1 in
// the lanes whose bottom level is handed over (the caller then drops it).
template <bool DIH>
__device__ __forceinline__ uint32_t post_mail(const DfsParams &p, uint32_t lane, uint32_t sp, uint32_t bot,
                                              uint32_t owner, uint32_t cls, bool &queue_live) {
    const unsigned long long tk = *((volatile unsigned long long *)(p.ctl + kCtlMail));
    const uint32_t req = __shfl_sync(kFull, (uint32_t)tk, 0), sup = __shfl_sync(kFull, (uint32_t)(tk >> 32), 0);
    if (req) queue_live = false;  // a ticket is taken only when the queue is empty
    if (req <= sup) return 0;
    uint32_t x = kFull, y = 0, z = 0, w = 0;
    if (sp != bot) lds128(bot, x, y, z, w);
    const uint32_t rows = 32u - __popc(x);  // rows the level still has to place
    const uint32_t most = __reduce_max_sync(kFull, rows);
    if (most < kMailMinRows) return 0;
    const unsigned give = __ballot_sync(kFull, rows + 1u >= most && rows >= kMailMinRows);
    const uint32_t n = min((uint32_t)kMailLevels, ((uint32_t)__popc(give) + 1u) / 2u);
    uint32_t t = 0;
    if (lane == 0) {
        t = (uint32_t)(atomicAdd(p.ctl + kCtlMail, 1ull << 32) >> 32);
        atomicAdd(p.ctl + kCtlWork, 1ull);
        __threadfence();
    }
    t = __shfl_sync(kFull, t, 0);
    MailSlot *s = mail_slot(p, t);
    const uint32_t none = mail_tag(p, t, kMailEmpty);
    const uint32_t k = __popc(give & lanemask_lt());
    const bool mine = (give >> lane & 1u) && k < n;
    uint32_t posted = 0;
    const uint32_t ready = __shfl_sync(kFull, ld_acquire(&s->state), 0) == none;
    if (ready) {
        if (mine) {
            __stcg(s->level + k, make_uint4(x, y, z, w));
            __stcg(s->owner + k, owner);
            if (DIH) __stcg(s->cls + k, cls);
        }
        if (lane == 0) __stcg(&s->count, n);
        __threadfence();
        __syncwarp();
        if (lane == 0) posted = atomicCAS(&s->state, none, none | kMailFull) == none;
        posted = __shfl_sync(kFull, posted, 0);
    }
    if (!posted && lane == 0) {
        atomicCAS(&s->state, none | kMailGone, none + 4u);
        atomicAdd(p.ctl + kCtlWork, ~0ull);
    }
    return posted && mine ? 1u : 0u;
}

// RESUME adds the continuation queue and the deadline dump; it is a separate
// instantiation so that the plain count kernel carries none of that code
// (it measurably changed the code generated for the DFS loop).
// DIH runs the dihedral decomposition: every task carries a class (rules and
// weights, see DfsParams::cls_tab) and the step is VAR 5, with RESUME DIH4.
// The count kernels are held to 32 registers (2 x 1024 threads): left to itself
// the compiler takes 42 for one of them, and the loop's code is worse (N=19 133.6
// -> 136.2 ms); the others spill at 32.
template <bool PER_OWNER, bool NODES, int VAR, int UNROLL, bool RESUME = false, bool DIH = false>
__global__ void __launch_bounds__(1024, NODES || DIH || RESUME ? 0 : 2) dfs_kernel(DfsParams p) {
    static_assert(DIH ? (RESUME ? VAR == 4 : VAR == 5) : VAR == 4 || VAR == 6 || VAR == 7, "step variant");
    static_assert(!NODES || VAR == 6, "node counts run variant 6");
    constexpr bool kPreRd = !(DIH && VAR == 4);  // the lane form of rd, see lane_rd
    constexpr bool MAIL = !RESUME;
    // Node counts and the dihedral kernels take a stack of N-1-rows slots as
    // nq_stack_levels states it (one more than their step uses), and refuse less.
    constexpr int kSpared = NODES || DIH ? 0 : kStackRowsSpared<VAR>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned long long red_cnt[32];
    __shared__ unsigned long long red_nodes[32];
    __shared__ int s_is_last;

    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(smem_raw);
    // Stack layout 0 (interleaved): slot s of lane l at warp_base + s*512 + l*16,
    // conflict-free for every mix of depths.  Layout 1 (lane-major): each
    // lane's slots contiguous, lane_base + s*16 (kept for the autotuner).
    const uint32_t stride = p.layout == 1 ? 16u : kSlotBytes;
    const uint32_t my_base = p.layout == 1
                                 ? smem_base + (warp * 32u + lane) * (uint32_t)p.levels * 16u
                                 : smem_base + warp * (uint32_t)p.levels * kSlotBytes + lane * 16u;

    if (p.cta_times && threadIdx.x == 0) p.cta_times[2 * blockIdx.x] = globaltimer_ns();
    const StepConsts kc{p.k_one, p.k_two, p.k_mone, stride};
    uint32_t cols = 0, ld = 0, rd = 0, avail = 0;
    uint32_t sp = my_base, bot = my_base;
    uint32_t cnt = 0, it = 0;
    uint32_t owner = kNoOwner;
    DihLane dih;
    unsigned long long tot = 0, tot_nodes = 0;
    const long long qlen = RESUME ? p.n_cont_in + p.ntasks - p.task_base
                                  : (p.coarse << p.lg_coarse) +
                                        (((p.nqueue > 0 ? p.nqueue : p.ntasks) - p.coarse) << p.lg_fine);
    bool queue_live = qlen > 0;
    const bool gate = !DIH && mail_on(p);  // (a dihedral list's depth is always known)
    const auto mail = [&] { return MAIL && (DIH ? p.mail && p.steal : gate); };
    unsigned looks = 0;           // trips, for the looks at the mailbox
    bool timed_out = false;
    unsigned long long deadline = 0;
    if (p.limit_ns) {
        unsigned long long t0 = 0;
        if (lane == 0) t0 = globaltimer_ns();
        deadline = __shfl_sync(kFull, t0, 0) + p.limit_ns;
    }

    for (;;) {
        // ---- fold the per-lane 32-bit counters (bounded inner loop keeps them < 2^32)
        if (PER_OWNER) {
            if (owner != kNoOwner && (avail == 0 || ((cnt | it) >> 31))) {
                if (cnt) atomicAdd(p.out_cnt + owner, (unsigned long long)cnt);
                if (NODES && it) atomicAdd(p.out_nodes + owner, (unsigned long long)it);
                tot += cnt;
                if (NODES) tot_nodes += it;
                cnt = 0;
                it = 0;
                if (avail == 0) owner = kNoOwner;
            }
        } else {
            tot += cnt;
            if (NODES) tot_nodes += it;
            cnt = 0;
            it = 0;
        }

        // ---- deadline (lane 0 reads the timer; the decision is warp-uniform)
        if (deadline) {
            unsigned long long now = 0;
            if (lane == 0) now = globaltimer_ns();
            now = __shfl_sync(kFull, now, 0);
            if (now > deadline) {
                if (lane == 0) atomicExch(p.ctl + kCtlTimeout, 1ull);
                if (RESUME) timed_out = true;
                if (mail()) out_of_work(p, lane);
                break;
            }
        }

        unsigned idle = __ballot_sync(kFull, avail == 0);
        bool check_idle = true;
        if (idle) {
            if (queue_live) {
                // ---- refill from the queue: one atomic per warp
                const int nidle = __popc(idle);
                const int leader = __ffs(idle) - 1;
                unsigned long long b = 0;
                if ((int)lane == leader) b = atomicAdd(p.ctl + kCtlHead, (unsigned long long)nidle);
                b = __shfl_sync(kFull, b, leader);
                if (b + (unsigned long long)nidle >= (unsigned long long)qlen) queue_live = false;
                if (avail == 0) {
                    const unsigned long long q = b + (unsigned long long)__popc(idle & lanemask_lt());
                    if (RESUME && q < (unsigned long long)p.n_cont_in) {
                        // a level saved by an earlier, interrupted run
                        sp = bot = my_base;
                        const uint4 e = p.cont_in[q];
                        const int need = __popc(~e.x) - 1 - kSpared;
                        if (need > p.levels) {
                            atomicOr(p.ctl + kCtlError, kErrDepth);
                        } else {
                            cols = e.x;
                            ld = lane_ld(e.y);
                            rd = lane_rd<kPreRd>(e.z);
                            avail = e.w;
                            // a level saved on row N-2 or N-1 (by a kernel that steps those rows)
                            if (VAR == 4 && !DIH) tot += settle_level(p.N, cols, ld, rd, avail);
                            // a saved level already carries its class's rules in avail
                            if (DIH) load_class_index(p, p.cont_in_cls[q], dih);
                            if (PER_OWNER && avail) owner = p.cont_in_owner ? p.cont_in_owner[q] : 0u;
                        }
                    } else if (q < (unsigned long long)qlen) {
                        long long pos = (long long)q;
                        uint32_t way = 0, lg = 0;
                        if (RESUME) {
                            pos = p.task_base + (long long)(q - (unsigned long long)p.n_cont_in);
                        } else {
                            const long long fine = pos - (p.coarse << p.lg_coarse);
                            lg = fine < 0 ? p.lg_coarse : p.lg_fine;
                            if (fine >= 0) pos = fine;
                            way = (uint32_t)pos & ((1u << lg) - 1u);
                            pos = (pos >> lg) + (fine < 0 ? 0 : p.coarse);
                        }
                        const long long t = p.order ? (long long)__ldg(p.order + pos) : pos;
                        // A permutation entry out of range is skipped, never dereferenced.
                        if (t >= 0 && t < p.ntasks) {
                            sp = bot = my_base;
                            uint32_t placed = 0;
                            uint32_t done = load_task<kPreRd, !DIH, kSpared>(p, t, cols, ld, rd, avail, placed);
                            if (DIH) {
                                load_class(p, t, dih);
                                done *= dih.w;
                                // The task's own row follows the class rules too
                                // (the step applies them to children only).
                                const uint32_t pc = (uint32_t)__popc(cols);
                                if (avail && pc > dih.side_popc) avail &= pc == 31u ? dih.last_mask : p.noside;
                                if (VAR == 5 && avail) done += settle_level_dih(p.N, cols, ld, rd, avail, dih);
                            }
                            if (!RESUME) {
                                // this lane's share of the task's columns
                                avail &= share_mask(lg, way);
                                if (way) done = 0;
                            }
                            const uint32_t own = p.owner_of ? __ldg(p.owner_of + t) : (uint32_t)t;
                            if (PER_OWNER) {
                                if (done) atomicAdd(p.out_cnt + own, (unsigned long long)done);
                                if (avail) owner = own;
                            }
                            tot += done;
                            if (NODES) {
                                const uint32_t here = __popc(placed & share_mask(lg, way));
                                if (PER_OWNER && here) atomicAdd(p.out_nodes + own, (unsigned long long)here);
                                tot_nodes += here;
                            }
                        }
                    }
                }
                // Lanes whose task was empty are still idle: refill again.
                if (queue_live) continue;
                idle = __ballot_sync(kFull, avail == 0);
            }
            if (idle && !queue_live) {
                // ---- in-warp donation: k-th idle lane takes the bottom
                // stacked level of the k-th lane that has one worth it.
                uint32_t low = kFull;
                if (sp != bot) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(low) : "r"(bot) : "memory");
                const bool has = 32u - __popc(low) >= kGiveMinRows;
                const unsigned rich = p.steal ? __ballot_sync(kFull, has) : 0u;
                __syncwarp();  // order the donors' earlier stack stores before the reads below
                const int npair = min(__popc(idle), __popc(rich));
                if (npair > 0) {
                    int donor = -1;
                    if (avail == 0) {
                        const int k = __popc(idle & lanemask_lt());
                        if (k < npair) {
                            unsigned m = rich;
                            for (int i = 0; i < k; ++i) m &= m - 1;
                            donor = __ffs(m) - 1;
                        }
                    }
                    const uint32_t src_addr = __shfl_sync(kFull, bot, donor < 0 ? lane : donor);
                    const uint32_t src_owner = __shfl_sync(kFull, owner, donor < 0 ? lane : donor);
                    DihLane src_dih;
                    if (DIH) {
                        const int src = donor < 0 ? (int)lane : donor;
                        src_dih.side_popc = __shfl_sync(kFull, dih.side_popc, src);
                        src_dih.last_mask = __shfl_sync(kFull, dih.last_mask, src);
                        src_dih.tie_bit = __shfl_sync(kFull, dih.tie_bit, src);
                        src_dih.w = __shfl_sync(kFull, dih.w, src);
                        src_dih.w_tie = __shfl_sync(kFull, dih.w_tie, src);
                        src_dih.cls = __shfl_sync(kFull, dih.cls, src);
                    }
                    if (donor >= 0) {
                        lds128(src_addr, cols, ld, rd, avail);
                        sp = bot = my_base;
                        owner = src_owner;
                        if (DIH) dih = src_dih;
                    }
                    __syncwarp();
                    if (has && __popc(rich & lanemask_lt()) < npair) bot += stride;
                    __syncwarp();
                    check_idle = npair == __popc(idle);
                } else if (idle == kFull) {
                    // whole warp idle, queue empty
                    if (!mail()) break;
                    if (!take_mail<DIH>(p, lane, cols, ld, rd, avail, owner, dih)) break;
                    sp = bot = my_base;
                    check_idle = false;
                } else {
                    check_idle = false;
                }
            }
        }
        // Other warps may be out of work (and the queue empty): offer them
        // stacked levels.
        if (mail()) {
            looks += check_idle ? 4u : 1u;
            if (looks >= 4u) {
                looks = 0;
                bot += stride * post_mail<DIH>(p, lane, sp, bot, owner, dih.cls, queue_live);
            }
        }

        if (!RESUME) check_idle &= queue_live;

        // ---- DFS steps
        if (check_idle) {
            for (int s = 0; s < p.inner; s += UNROLL) {
                dfs_steps<VAR, NODES, DIH, UNROLL>(cols, ld, rd, avail, sp, cnt, it, bot, kc, dih, p.noside);
                if (__any_sync(kFull, avail == 0)) break;
            }
        } else {
            for (int s = 0; s < kTailTrip; s += UNROLL) {
                dfs_steps<VAR, NODES, DIH, UNROLL>(cols, ld, rd, avail, sp, cnt, it, bot, kc, dih, p.noside);
                const unsigned idle_now = __ballot_sync(kFull, avail == 0);
                if (RESUME ? idle_now == kFull : (p.steal && __popc(idle_now) >= kTailIdle)) break;
            }
        }
    }

    // Deadline stop: save every unfinished level so a later run can resume.
    // The current level keeps its untried columns; every stacked level does
    // too (only levels with untried columns are ever pushed).
    if (RESUME && timed_out && p.cont_out) {
        const uint32_t nstk = (sp - bot) / stride;
        const uint32_t mine = (avail != 0 ? 1u : 0u) + nstk;
        unsigned long long at = 0;
        if (mine) at = atomicAdd(p.ctl + kCtlCont, (unsigned long long)mine);
        if (mine && at + mine > (unsigned long long)p.cont_cap) {
            atomicOr(p.ctl + kCtlError, kErrContOverflow);
        } else if (mine) {
            if (avail) {
                p.cont_out[at] = make_uint4(cols, ref_ld(ld), ref_rd<kPreRd>(rd), avail);
                if (p.cont_out_owner) p.cont_out_owner[at] = owner;
                if (DIH) p.cont_out_cls[at] = (uint8_t)dih.cls;
                ++at;
            }
            for (uint32_t a = bot; a != sp; a += stride, ++at) {
                uint32_t x, y, z, w;
                lds128(a, x, y, z, w);
                p.cont_out[at] = make_uint4(x, ref_ld(y), ref_rd<kPreRd>(z), w);
                if (p.cont_out_owner) p.cont_out_owner[at] = owner;
                if (DIH) p.cont_out_cls[at] = (uint8_t)dih.cls;
            }
        }
    }

    // CTA finish time: the last warp of the CTA to leave the DFS loop.
    if (p.cta_times) atomicMax(p.cta_times + 2 * blockIdx.x + 1, globaltimer_ns());

    // Flush what the last trip left (deadline exit, or the final fold).
    if (PER_OWNER) {
        if (owner != kNoOwner) {
            if (cnt) atomicAdd(p.out_cnt + owner, (unsigned long long)cnt);
            if (NODES && it) atomicAdd(p.out_nodes + owner, (unsigned long long)it);
        }
    }
    tot += cnt;
    if (NODES) tot_nodes += it;

    // ---- per-warp, per-CTA reduction
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tot += __shfl_xor_sync(kFull, tot, o);
        if (NODES) tot_nodes += __shfl_xor_sync(kFull, tot_nodes, o);
    }
    if (lane == 0) {
        red_cnt[warp] = tot;
        red_nodes[warp] = tot_nodes;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long s = 0, sn = 0;
        for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) {
            s += red_cnt[w];
            sn += red_nodes[w];
        }
        p.block_cnt[blockIdx.x] = s;
        if (NODES) p.block_nodes[blockIdx.x] = sn;
        __threadfence();
        const unsigned long long ticket = atomicAdd(p.ctl + kCtlDone, 1ull);
        s_is_last = (ticket == (unsigned long long)gridDim.x - 1ull);
    }
    __syncthreads();
    // ---- the last CTA empties the mailbox for the next launch and sums the
    // per-CTA partials in CTA order
    if (s_is_last) {
        __threadfence();
        if (MAIL && p.mail) {
            const unsigned long long tk = *((volatile unsigned long long *)(p.ctl + kCtlMail));
            const uint32_t used = min(p.mail_cap, max((uint32_t)tk, (uint32_t)(tk >> 32)));
            for (uint32_t i = threadIdx.x; i < used; i += blockDim.x) p.mail[i].state = kMailEmpty;
        }
        unsigned long long s = 0, sn = 0;
        for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
            s += *((volatile unsigned long long *)(p.block_cnt + b));
            if (NODES) sn += *((volatile unsigned long long *)(p.block_nodes + b));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(kFull, s, o);
            if (NODES) sn += __shfl_xor_sync(kFull, sn, o);
        }
        __syncthreads();
        if (lane == 0) {
            red_cnt[warp] = s;
            red_nodes[warp] = sn;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long a = 0, an = 0;
            for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) {
                a += red_cnt[w];
                an += red_nodes[w];
            }
            *p.sum_out = a;
            if (NODES) *p.nodes_out = an;
            const unsigned long long err = *((volatile unsigned long long *)(p.ctl + kCtlError));
            const unsigned long long tmo = *((volatile unsigned long long *)(p.ctl + kCtlTimeout));
            // Every warp is out of work and no posted level was left behind.
            const bool mail_ok = !mail() || tmo ||
                                 (long long)*((volatile unsigned long long *)(p.ctl + kCtlWork)) +
                                         (long long)gridDim.x * (blockDim.x >> 5) == 0;
            *p.status_out = ((err & kErrDepth) ? kStatDepth : 0ull) | (tmo ? kStatTimeout : 0ull) |
                            ((err & kErrContOverflow) ? kStatContOverflow : 0ull) | (mail_ok ? 0ull : kStatMail);
        }
    }
}

}  // namespace nqb
