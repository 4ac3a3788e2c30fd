// launch.h -- launch-shape choices shared by every entry that starts the DFS
// kernel (capi.cu and the allocation-free entry in noalloc.cu).
//
// The reference fixes its CTA size and stack depth at compile time
// (CU1DBLOCK / STACKSIZE, src/macro.h:25-35).  Here both are chosen per launch
// from the stack depth the tasks need: a warp's stack takes levels x 512 B of
// shared memory, so the CTA size decides how much of the SM's shared memory
// can hold stacks, and with it how many warps stay resident.
#pragma once

#include <cuda_runtime.h>

#include "dfs_kernel.cuh"

namespace nqb {

// DFS steps per warp vote (the unroll of the kernel's inner loop), a
// compile-time choice.  The count steps run 16 between votes: fewer votes and loop
// branches per step, for lanes that wait up to 15 steps for a refill (1.1 % faster
// than 8 at N=21, k=6).  So does the node-count step (300,007 prefixes of N=17:
// kernel 1.88 ms with 8, 1.79 with 16); the dihedral steps keep 8.  A trip of the
// inner loop runs inner_steps rounded up to a multiple of the unroll.
#ifndef NQB_COUNT_UNROLL
#define NQB_COUNT_UNROLL 16
#endif
#ifndef NQB_NODES_UNROLL
#define NQB_NODES_UNROLL 16
#endif
#ifndef NQB_DIH_UNROLL
#define NQB_DIH_UNROLL 8
#endif
constexpr int kCountUnroll = NQB_COUNT_UNROLL;
constexpr int kNodesUnroll = NQB_NODES_UNROLL;
constexpr int kDihUnroll = NQB_DIH_UNROLL;
static_assert(kCountUnroll % 4 == 0 && kNodesUnroll % 4 == 0 && kDihUnroll % 4 == 0,
              "inner_steps are rounded to multiples of 4");

// DFS steps a warp runs between visits to the queue (the fold of its 32-bit
// counters happens at the same point).
constexpr int kDefaultInner = 1024;
// Static shared memory of dfs_kernel: two 32-entry reduction arrays + a flag.
constexpr int kDfsStaticSmem = 2 * 32 * 8 + 16;
// Search range of the default CTA size.  One 1024-thread CTA per SM holds as
// many warps as two 512-thread CTAs at 14 stack levels (32) but ran an N=21
// count 2.9 % slower (13.97 s against 13.57 s), so the search stops at 512.
constexpr int kMinAutoThreads = 64;
constexpr int kMaxAutoThreads = 512;

// Slots a count launch gets beyond stack_need(): variant 6 pushes on one more row
// than the stated depth (nq_stack_levels) covers, variant 7 (per-owner outputs) on
// two.  A launch with a stated CTA size that has no room for them runs
// kTightStepVar, which needs none.
inline int extra_slots(bool per_owner) { return per_owner ? 2 : 1; }
inline bool slots_fit(int threads, int slots, int smem_optin) {
    return (long long)(threads / 32) * slots * kSlotBytes + kDfsStaticSmem <= smem_optin;
}

// Stack slots per lane that a launch over prefixes with `placed` queens is given
// and that nq_stack_levels states: N-1-placed for node counts and the dihedral
// decomposition (whose steps push on one row fewer), two fewer for counts.  At
// least 1.
inline int stack_need(int N, int placed, bool filtered) {
    const int need = N - 1 - placed - (filtered ? kStackRowsSpared<4> : 0);
    return need < 1 ? 1 : need;
}

// The CTA size (a multiple of 32 in [64, 512]) that keeps the most warps
// resident per SM for `levels` stack slots per lane, the larger CTA on a tie;
// at most cap_per_sm CTAs per SM are counted.  Returns 0 when no size fits.
// Uses only occupancy queries (no allocation, no launch).
template <typename Kernel>
int resident_warp_threads(Kernel fn, int levels, int smem_optin, int cap_per_sm) {
    int best = 0, best_warps = 0;
    for (int t = kMaxAutoThreads; t >= kMinAutoThreads; t -= 32) {
        const long long smem = (long long)(t / 32) * levels * kSlotBytes;
        if (smem + kDfsStaticSmem > smem_optin) continue;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, t, (size_t)smem) != cudaSuccess) {
            (void)cudaGetLastError();
            continue;
        }
        per_sm = per_sm < cap_per_sm ? per_sm : cap_per_sm;
        if (per_sm * (t / 32) > best_warps) {
            best_warps = per_sm * (t / 32);
            best = t;
        }
    }
    return best;
}

// DFS steps between visits to the queue where tasks are dealt out in shares and
// the caller names none: such runs last a few hundred microseconds to
// milliseconds, so a warp must notice soon that others are out of work (1024
// steps are 60-190 us).
constexpr int kShareInner = 256;

// How the queue hands out tasks: the first `coarse` tasks as 2^lg_coarse shares
// of their root level's columns each (share_mask), the others as 2^lg_fine.
// A lane runs a share by itself (until the queue is empty), so a share must be
// short against the whole run: below 4 positions per lane the tasks are dealt
// out finer, and the last ones always are.  Sixteen shares only where eight do
// not give every lane one; half of them are empty (a level rarely has more than
// eight alive columns), and an empty share still costs a visit to the queue.
// Measured: 60,001 prefixes of N=16, k=5 (0.23 per lane) 1.35 ms whole, 0.48 in
// shares; 1501 prefixes of N=13, k=4 0.131 -> 0.097 ms per call.  The line at 8, 4
// and 2 positions per lane: a batch of 512 boards of N=12..17 7.7, 7.7, 8.0 ms;
// 300,007 prefixes of N=17 with node counts (1.6 per lane) 1.63, 1.45, 1.39 ms of
// kernel time; 8 % of N=21's (2.1 per lane) 750, 751, 750 ms; 1.1e6 of N=18 (4.8
// per lane) 16.9 ms at all three.
inline void set_shares(DfsParams &p, long long lanes) {
    const long long n = p.nqueue > 0 ? p.nqueue : p.ntasks;
    p.coarse = n;
    p.lg_coarse = p.lg_fine = 0;
    if (!p.steal) return;
    p.lg_fine = (n << 3) < lanes ? 4 : 3;
    while (p.lg_coarse < p.lg_fine && (n << p.lg_coarse) < 4 * lanes) ++p.lg_coarse;
    const long long m = (2 * lanes) >> p.lg_fine;
    p.coarse = n > m ? n - m : 0;
}

}  // namespace nqb
