// mlp.cu -- the learned subtree-cost model and the longest-first scheduler.
//
// No counterpart in the reference (its tasks run in expander order through
// one atomic ticket, src/n_queens_cuda.cu:10,80).  A small MLP predicts
// log2(1 + DFS nodes) of a prefix task from its three masks; the predictions
// order the task queue longest-first (binned to 1/8 of a log2 unit, stable
// inside a bin).  The order only changes which lane runs which task, never a
// count.
//
// Model: x (96 bits: cols, ld, rd, each as 32 bits with the columns >= N
// cleared) -> 128 ReLU -> 128 ReLU -> 1.  Weights are BF16 for compute with
// FP32 master copies for Adam; biases are FP32; every sum accumulates in
// FP32.  Kernels (all hand-written):
//   mlp_forward_kernel  forward for many tasks on the tensor cores
//   mlp_predict_kernel  the same in FP32 on the CUDA cores, for weights of any size
//   mlp_train_kernel    forward + backward of a minibatch slice; per-CTA
//                       partial gradients (no atomics: deterministic)
//   mlp_adam_kernel     sums the partials in CTA order, Adam step, refreshes
//                       the BF16 copies
// The training kernel's first layer exploits binary inputs: h1 = b1 + sum of the
// W1 columns of the set bits (about 3k of them for a k-row prefix).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <cmath>
#include <cub/device/device_radix_sort.cuh>
#include <mutex>
#include <string>
#include <vector>

#include "dfs_kernel.cuh"
#include "expand.h"
#include "n_queens_b200.h"

namespace nqb {

void set_last_error(const char *msg);
// Status of the exception in flight, for the entries' handlers (defined in capi.cu).
int status_of_exception() noexcept;

namespace {

constexpr int kIn = 96, kH1 = 128, kH2 = 128;
// Flat FP32 parameter layout (also the layout of gradients and of
// nq_mlp_get_params): W1[H1][IN], b1[H1], W2[H2][H1], b2[H2], W3[H2], b3.
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kH1 * kIn;
constexpr int kOffW2 = kOffB1 + kH1;
constexpr int kOffB2 = kOffW2 + kH2 * kH1;
constexpr int kOffW3 = kOffB2 + kH2;
constexpr int kOffB3 = kOffW3 + kH2;
constexpr int kParams = kOffB3 + 1;
constexpr int kGroup = 32;  // tasks per tile of the training kernel

// Offset (bytes) of element (row, k) of a K-major tensor-core operand without
// swizzle: 8-row x 16-byte core matrices, sbo bytes between 8-row groups.
__host__ __device__ constexpr uint32_t off_kmajor(uint32_t row, uint32_t k, uint32_t sbo) {
    return (row >> 3) * sbo + (k >> 3) * 128u + (row & 7u) * 16u + (k & 7u) * 2u;
}
constexpr uint32_t kSbo1 = (kIn / 8) * 128;  // 1536 B: operands with K = 96
constexpr uint32_t kSbo2 = (kH1 / 8) * 128;  // 2048 B: operands with K = 128

// Compute copy of the weights in device memory.
struct Weights {
    // W1 and W2 as the forward kernel's B operands lie in shared memory, so that
    // a CTA loads them by straight 16-byte copies.
    alignas(16) __nv_bfloat16 w1c[kIn * kH1];
    alignas(16) __nv_bfloat16 w2c[kH2 * kH1];
    __nv_bfloat16 w1t[kIn * kH1];  // [input bit][hidden unit]
    __nv_bfloat16 w2[kH2 * kH1];   // [unit of layer 2][unit of layer 1]
    __nv_bfloat16 w3[kH2];
    float b1[kH1];
    float b2[kH2];
    float b3;
};

struct TaskView {
    const uint32_t *cols, *ld, *rd;
    const uint8_t *task_n;  // per-task board size or nullptr
    const uint32_t *index;  // optional indirection (training permutation)
    int N;
};

__device__ __forceinline__ void load_masks(const TaskView &tv, long long t, uint32_t &m0, uint32_t &m1,
                                           uint32_t &m2) {
    const long long i = tv.index ? (long long)tv.index[t] : t;
    const int n = tv.task_n ? (int)tv.task_n[i] : tv.N;
    const uint32_t last = (n >= 32) ? 0xffffffffu : ((1u << n) - 1u);
    m0 = tv.cols[i] & last;
    m1 = tv.ld[i] & last;
    m2 = tv.rd[i] & last;
}

// Layer 1 for one task and hidden unit j: b1[j] + sum of W1 columns of the
// set input bits.  Every thread of the CTA walks the same bits (uniform).
__device__ __forceinline__ float layer1(const __nv_bfloat16 *w1t, float b, uint32_t m0, uint32_t m1, uint32_t m2,
                                        int j) {
    float acc = b;
    while (m0) {
        const int f = __ffs(m0) - 1;
        m0 &= m0 - 1;
        acc += __bfloat162float(w1t[f * kH1 + j]);
    }
    while (m1) {
        const int f = __ffs(m1) - 1 + 32;
        m1 &= m1 - 1;
        acc += __bfloat162float(w1t[f * kH1 + j]);
    }
    while (m2) {
        const int f = __ffs(m2) - 1 + 64;
        m2 &= m2 - 1;
        acc += __bfloat162float(w1t[f * kH1 + j]);
    }
    return acc;
}

// Layer 2 pre-activation of unit j for one task: w2row holds W2[j][:] as
// 64 packed BF16 pairs, h1 the task's 128 layer-1 outputs (broadcast reads).
__device__ __forceinline__ float layer2(const uint32_t (&w2row)[kH1 / 2], float b, const float *h1) {
    float acc = b;
#pragma unroll
    for (int i = 0; i < kH1; i += 4) {
        const float4 h = *reinterpret_cast<const float4 *>(h1 + i);
        const __nv_bfloat162 wa = *reinterpret_cast<const __nv_bfloat162 *>(&w2row[i / 2]);
        const __nv_bfloat162 wb = *reinterpret_cast<const __nv_bfloat162 *>(&w2row[i / 2 + 1]);
        acc = fmaf(__low2float(wa), h.x, acc);
        acc = fmaf(__high2float(wa), h.y, acc);
        acc = fmaf(__low2float(wb), h.z, acc);
        acc = fmaf(__high2float(wb), h.w, acc);
    }
    return acc;
}

__device__ __forceinline__ void load_w2row(const Weights *w, int j, uint32_t (&w2row)[kH1 / 2]) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(w->w2 + j * kH1);
#pragma unroll
    for (int i = 0; i < kH1 / 2; ++i) w2row[i] = src[i];
}

// The general forward of nq_mlp_predict, in FP32 on the CUDA cores: out[t] =
// predicted log2(1 + nodes).  128 threads, thread j = hidden unit j.  Runs where
// the split form's products of zeros and of BF16 parts would differ from FP32's
// (see kWideWeight); elsewhere the split form is faster (200,000 tasks 889 us
// against 55).
__global__ void __launch_bounds__(128) mlp_predict_kernel(TaskView tv, long long n, const Weights *w, float *out) {
    __shared__ __align__(16) __nv_bfloat16 s_w1t[kIn * kH1];
    __shared__ __align__(16) float s_h[kGroup * kH1];
    __shared__ uint32_t s_m[3][kGroup];
    const int j = threadIdx.x;
    for (int i = j; i < kIn * kH1 / 8; i += blockDim.x)
        reinterpret_cast<uint4 *>(s_w1t)[i] = reinterpret_cast<const uint4 *>(w->w1t)[i];
    uint32_t w2row[kH1 / 2];
    load_w2row(w, j, w2row);
    const float b1 = w->b1[j], b2 = w->b2[j], w3 = __bfloat162float(w->w3[j]), b3 = w->b3;
    const int warp = j >> 5, lane = j & 31;
    __syncthreads();
    for (long long g0 = (long long)blockIdx.x * kGroup; g0 < n; g0 += (long long)gridDim.x * kGroup) {
        const int gn = (int)min((long long)kGroup, n - g0);
        if (j < gn) load_masks(tv, g0 + j, s_m[0][j], s_m[1][j], s_m[2][j]);
        __syncthreads();
        for (int s = 0; s < gn; ++s)
            s_h[s * kH1 + j] = fmaxf(layer1(s_w1t, b1, s_m[0][s], s_m[1][s], s_m[2][s], j), 0.f);
        __syncthreads();
        float v[kGroup];
#pragma unroll
        for (int s = 0; s < kGroup; ++s) v[s] = (s < gn) ? fmaxf(layer2(w2row, b2, s_h + s * kH1), 0.f) * w3 : 0.f;
        __syncthreads();
#pragma unroll
        for (int s = 0; s < kGroup; ++s) s_h[s * kH1 + j] = v[s];
        __syncthreads();
        // layer 3: warp w reduces tasks 8w..8w+7, each lane summing 4 units
        for (int s = warp * 8; s < warp * 8 + 8; ++s) {
            const float4 q = *reinterpret_cast<const float4 *>(s_h + s * kH1 + lane * 4);
            float a = (q.x + q.y) + (q.z + q.w);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (lane == 0 && s < gn) out[g0 + s] = a + b3;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Forward pass on the tensor cores (tcgen05).  A CTA runs GROUPS groups of 128
// threads, each on its own tiles of 128 tasks (thread t of a group = task row t
// = TMEM lane t):
//   X (128 x 96 binary, BF16) --tcgen05.mma--> D1 (TMEM, FP32) --relu+b1-->
//   H1 (128 x 128, smem) --tcgen05.mma--> D2 (TMEM) --relu+b2, dot W3, +b3-->
//   out.
// H1 is BF16 in one of two forms: rounded (PARTS 1, the scheduler's forward,
// nq_mlp_predict_tensor), or split into three BF16 parts that add up to the FP32
// value (PARTS 3, nq_mlp_predict), each multiplied by the exact BF16 weights into
// the same FP32 accumulator.
// Operands use the SM100 K-major canonical layout without swizzle: 8-row x
// 16-byte core matrices, LBO = 128 B between the two core matrices of one
// K=16 step, SBO = K/8 * 128 B between 8-row groups.  One thread of a group
// issues its MMAs; completion is signalled through the group's mbarrier
// (tcgen05.commit) and every wait on it is bounded: on expiry the group sets
// *err, gives its remaining tasks the lowest key and their own index (so that a
// sorted order stays a permutation), waits once more, again bounded, for the
// MMAs in flight and stops.
//
// What bounds it: the latency of a tile's chain (X build, MMA, epilogue, MMA,
// epilogue), then issue in the epilogues (52 % at 1.9e6 tasks, tensor pipe 38 %).
// Four groups share one copy of the weights, which is what fits shared memory
// (56 KiB + 4 x 32 KiB) and TMEM (D2 overwrites D1 once its group has read it:
// 128 columns each): 1.9e6 tasks with their sort keys 226 + 10 -> 154 us against two
// CTAs per SM with one tile each and a key kernel of its own.  PARTS 3 keeps D1
// for the later parts (256 columns) and needs two operand buffers, so two groups
// run: 200,000 tasks 889 us on the CUDA cores in FP32 -> 55 us, error against 64
// bits 2.4e-8 (2.3e-8 before; the rounding of the result).
namespace tc {

constexpr uint32_t kOffB1 = 0;                          // W1: 128 units x 96  (24 KiB)
constexpr uint32_t kOffB2 = kOffB1 + kH1 * kSbo1 / 8;   // 24576: W2: 128 x 128 (32 KiB)
constexpr uint32_t kOffA = kOffB2 + kH2 * kSbo2 / 8;    // 57344: operand buffers (4 x 32 KiB)
constexpr uint32_t kABytes = 128 * kSbo2 / 8;
constexpr uint32_t kOffBias = kOffA + 4 * kABytes;      // b1, b2, w3 (fp32)
constexpr uint32_t kOffLut = kOffBias + 3 * 128 * 4;    // 4 bits -> 4 BF16 values (16 x 8 B)
constexpr uint32_t kOffBar = kOffLut + 128;             // one mbarrier per group (8 B)
constexpr uint32_t kOffTmem = kOffBar + 4 * 8;          // TMEM base address word, fail words
constexpr uint32_t kSmemBytes = kOffTmem + 32;
constexpr uint32_t kTmemCols = 512;
// Instruction descriptor, kind::f16: D F32, A and B BF16, both K-major,
// N = 128 (N>>3 at bit 17), M = 128 (M>>4 at bit 24).
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
constexpr unsigned long long kWaitLimit = 1ull << 22;  // polls: a few seconds at most

static_assert(off_kmajor(127, 95, kSbo1) < kOffB2 - kOffB1, "W1 tile bounds");
static_assert(off_kmajor(127, 127, kSbo2) < kOffA - kOffB2, "W2 tile bounds");
static_assert(off_kmajor(127, 127, kSbo2) < kABytes, "A tile bounds");
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one CTA");

// PARTS 3 runs when every weight and bias of the three layers (b3 is added last)
// is below 2^32 in magnitude: then layer 1 stays below 2^39 and layer 2 below
// 2^79, so no part of the split overflows, and no zero input or zero part meets an
// infinity or a NaN (0 * inf), which FP32 over the set bits alone would not have.
// Trained weights are far below; others go to mlp_predict_kernel.
constexpr float kWideWeight = 4294967296.f;
constexpr uint32_t kWideBf16 = 0x4F80u;  // the same in BF16
__device__ __forceinline__ bool wide(uint32_t two_bf16) {
    return (two_bf16 & 0x7fffu) >= kWideBf16 || (two_bf16 >> 16 & 0x7fffu) >= kWideBf16;
}
__device__ __forceinline__ bool wide(const uint4 &v) { return wide(v.x) || wide(v.y) || wide(v.z) || wide(v.w); }

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);  // version 1; base offset 0; no swizzle
}

__device__ __forceinline__ void mma(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(da), "l"(db), "r"(kIdesc), "r"(accumulate));
}

__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Bounded wait (`limit` polls) for the mbarrier phase with the given parity; false on expiry.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, unsigned long long limit) {
    for (unsigned long long i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);  // a -> low half
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

}  // namespace tc

// One barrier per group of 128 threads (barrier 0 is the CTA's).
__device__ __forceinline__ void group_sync(uint32_t group) {
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1u) : "memory");
}

// Sort key of the longest-first order: 1 + predicted log2 cost in 1/8 units
// (key 0 is kept for tasks that must go last, mlp_last_kernel).
__device__ __forceinline__ uint16_t order_key(float pred) {
    const float v = fminf(fmaxf(pred * 8.f + 0.5f, 0.f), 65534.f);
    return (uint16_t)(1.f + v);
}

// out (optional): predictions.  key and idx (both or neither): sort keys and the
// identity permutation for the scheduler.  err: a host word, left alone unless a wait
// of `limit` polls expires (kErrWait) or the weights are out of PARTS 3's range
// (kErrWide: nothing was computed).
enum : int { kErrWait = 1, kErrWide = 2 };
template <int PARTS>
__global__ void __launch_bounds__(PARTS == 1 ? 512 : 256, 1)
    mlp_forward_kernel(TaskView tv, long long n, const Weights *w, float *out, uint16_t *key, uint32_t *idx,
                       volatile int *err, unsigned long long limit) {
    constexpr uint32_t kGroups = PARTS == 1 ? 4 : 2;
    constexpr uint32_t kBufs = 4 / kGroups;  // operand buffers of a group
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(tc_smem);
    const uint32_t tid = threadIdx.x, t = tid & 127u, g = tid >> 7, warp = t >> 5;
    const float *bias = reinterpret_cast<const float *>(tc_smem + tc::kOffBias);
    const uint32_t bar = base + tc::kOffBar + 8 * g;
    const uint32_t abuf = base + tc::kOffA + g * kBufs * tc::kABytes;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tc_smem + tc::kOffTmem);
    volatile int *fail = reinterpret_cast<volatile int *>(tmem_slot + 1 + g);

    {
        const uint4 *src1 = reinterpret_cast<const uint4 *>(w->w1c), *src2 = reinterpret_cast<const uint4 *>(w->w2c);
        uint4 *dst1 = reinterpret_cast<uint4 *>(tc_smem + tc::kOffB1);
        uint4 *dst2 = reinterpret_cast<uint4 *>(tc_smem + tc::kOffB2);
        bool wide = false;
        auto copy = [&](uint4 *dst, const uint4 *src, uint32_t count) {
            for (uint32_t i = tid; i < count; i += blockDim.x) {
                const uint4 v = src[i];
                dst[i] = v;
                if (PARTS == 3) wide |= tc::wide(v);
            }
        };
        copy(dst1, src1, kIn * kH1 / 8);
        copy(dst2, src2, kH2 * kH1 / 8);
        float *b = reinterpret_cast<float *>(tc_smem + tc::kOffBias);
        if (tid < 128) {
            b[tid] = w->b1[tid];
            b[128 + tid] = w->b2[tid];
            b[256 + tid] = __bfloat162float(w->w3[tid]);
            if (PARTS == 3)
                for (int k = 0; k < 3; ++k) wide |= !(fabsf(b[128 * k + tid]) < tc::kWideWeight);
        }
        if (PARTS == 3 && __syncthreads_or(wide)) {
            if (tid == 0) {
                *err = kErrWide;
                __threadfence_system();
            }
            return;
        }
        if (tid < 16) {
            uint32_t *lut = reinterpret_cast<uint32_t *>(tc_smem + tc::kOffLut) + 2 * tid;
            lut[0] = (tid & 1u ? 0x3F80u : 0u) | (tid & 2u ? 0x3F800000u : 0u);
            lut[1] = (tid & 4u ? 0x3F80u : 0u) | (tid & 8u ? 0x3F800000u : 0u);
        }
        if (t == 0) *fail = 0;
    }
    const float b3 = w->b3;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + tc::kOffTmem),
                     "r"(tc::kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const uint32_t d1 = tmem + g * (tc::kTmemCols / kGroups);  // this group's columns
    const uint32_t d2 = PARTS == 1 ? d1 : d1 + 128;
    const uint32_t lane_off = (warp * 32u) << 16;  // this warp's TMEM lanes
    const uint32_t lut = base + tc::kOffLut;
    uint32_t phase = 0;

    // Waits for the group's MMAs; false when the wait expired for some thread.
    auto mma_done = [&]() -> bool {
        if (!tc::wait_phase(bar, phase, limit)) *fail = 1;
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        group_sync(g);
        return *fail == 0;
    };
    // Makes the group's operand writes visible to the MMAs.
    auto operands_ready = [&]() {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        group_sync(g);
    };

    const long long tiles = (n + 127) / 128;
    const long long step = (long long)gridDim.x * kGroups;
    long long tile = blockIdx.x + (long long)gridDim.x * g;
    uint32_t m[3] = {0, 0, 0};
    if (tile * 128 + t < n) load_masks(tv, tile * 128 + t, m[0], m[1], m[2]);
    for (; tile < tiles; tile += step) {
        const long long task = tile * 128 + t;
        // ---- X row of this thread's task (zeros past the end)
#pragma unroll
        for (int c = 0; c < kIn / 8; ++c) {
            const uint32_t byte = m[c >> 2] >> ((c & 3) * 8);
            uint32_t q[4];
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(q[0]), "=r"(q[1]) : "r"(lut + (byte & 15u) * 8u));
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(q[2]), "=r"(q[3]) : "r"(lut + (byte >> 4 & 15u) * 8u));
            tc::sts128(abuf + off_kmajor(t, 8 * c, kSbo1), q[0], q[1], q[2], q[3]);
        }
        operands_ready();
        // ---- layer 1 on the tensor cores: D1 = X * W1^T, K = 96 in 6 steps
        if (t == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int kk = 0; kk < kIn / 16; ++kk)
                tc::mma(d1, tc::smem_desc(abuf + kk * 256, 128, kSbo1),
                        tc::smem_desc(base + tc::kOffB1 + kk * 256, 128, kSbo1), kk > 0);
            tc::commit(bar);
        }
        m[0] = m[1] = m[2] = 0;  // the next tile's masks load meanwhile
        if (task + step * 128 < n) load_masks(tv, task + step * 128, m[0], m[1], m[2]);
        if (!mma_done()) break;
        // ---- relu(D1 + b1) -> BF16 -> H1 rows (the A operand of layer 2); with
        // three parts: the first two, then the third over the first's buffer
#pragma unroll 1
        for (int pass = 0; pass < (PARTS == 1 ? 1 : 2); ++pass) {
#pragma unroll 2
            for (int c = 0; c < kH1 / 16; ++c) {
                float v[16];
                tc::ld16(d1 + lane_off + 16 * c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = fmaxf(v[j] + bias[16 * c + j], 0.f);
                uint32_t q[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) q[j] = tc::pack_bf16(v[2 * j], v[2 * j + 1]);
                if (PARTS == 3) {
                    // what the first part leaves (exact), rounded to the second
                    uint32_t r[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        v[2 * j] -= __uint_as_float(q[j] << 16);
                        v[2 * j + 1] -= __uint_as_float(q[j] & 0xffff0000u);
                        r[j] = tc::pack_bf16(v[2 * j], v[2 * j + 1]);
                    }
                    if (pass == 0) {
                        const uint32_t second = abuf + tc::kABytes;
                        tc::sts128(second + off_kmajor(t, 16 * c, kSbo2), r[0], r[1], r[2], r[3]);
                        tc::sts128(second + off_kmajor(t, 16 * c + 8, kSbo2), r[4], r[5], r[6], r[7]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            q[j] = tc::pack_bf16(v[2 * j] - __uint_as_float(r[j] << 16),
                                                 v[2 * j + 1] - __uint_as_float(r[j] & 0xffff0000u));
                    }
                }
                tc::sts128(abuf + off_kmajor(t, 16 * c, kSbo2), q[0], q[1], q[2], q[3]);
                tc::sts128(abuf + off_kmajor(t, 16 * c + 8, kSbo2), q[4], q[5], q[6], q[7]);
            }
            operands_ready();
            // ---- layer 2: D2 += H1 part * W2^T, 8 steps for each part
            if (t == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int kk = 0; kk < kH1 / 16; ++kk)
                    tc::mma(d2, tc::smem_desc(abuf + kk * 256, 128, kSbo2),
                            tc::smem_desc(base + tc::kOffB2 + kk * 256, 128, kSbo2), kk > 0 || pass > 0);
                if (PARTS == 3 && pass == 0)
#pragma unroll
                    for (int kk = 0; kk < kH1 / 16; ++kk)
                        tc::mma(d2, tc::smem_desc(abuf + tc::kABytes + kk * 256, 128, kSbo2),
                                tc::smem_desc(base + tc::kOffB2 + kk * 256, 128, kSbo2), 1);
                tc::commit(bar);
            }
            if (!mma_done()) break;
        }
        if (*fail) break;
        // ---- layer 3: sum_j relu(D2 + b2)_j * w3_j + b3
        float acc = 0.f;
#pragma unroll 2
        for (int c = 0; c < kH2 / 16; ++c) {
            float v[16];
            tc::ld16(d2 + lane_off + 16 * c, v);
#pragma unroll
            for (int j = 0; j < 16; ++j)
                acc = fmaf(fmaxf(v[j] + bias[128 + 16 * c + j], 0.f), bias[256 + 16 * c + j], acc);
        }
        if (task < n) {
            if (out) out[task] = acc + b3;
            if (key) {
                key[task] = order_key(acc + b3);
                idx[task] = (uint32_t)task;
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        group_sync(g);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (*fail) {
        tc::wait_phase(bar, phase ^ 1u, tc::kWaitLimit);  // MMAs still in flight read this CTA's shared memory
        if (key)
            for (; tile < tiles; tile += step) {
                const long long task = tile * 128 + t;
                if (task < n) {
                    key[task] = 1;
                    idx[task] = (uint32_t)task;
                }
            }
        if (t == 0) {
            *err = kErrWait;
            __threadfence_system();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tc::kTmemCols));
}

// Training: forward + backward of a minibatch slice in FP32 on the CUDA cores
// (the gradient of a batch is 0.4 GFLOP; what counts is that every SM works and
// that a multiply-add costs little more than its own issue slot).  One CTA of 256
// threads per SM takes tiles of 32 tasks:
//   H1 = relu(b1 + X W1^T)   bit by bit of X, a warp per task, four units a lane
//   H2 = relu(b2 + H1 W2^T)  4 tasks x 4 units a thread, steps of 4 along K
//   out, dout                a warp per task
//   dH2 = relu' . dout w3    (over H2)
//   dH1 = relu' . dH2 W2     4 x 4 a thread
//   dW2 += dH2^T H1          8 x 8 a thread, a tile's sum in registers, the tiles'
//                            sum in shared memory
//   dW1 += dH1^T X           8 x 6 a thread, accumulated in registers
// The products read rows of 16-byte vectors; rows are padded to 132 floats, so
// the eight lanes of a quarter-warp that read eight rows cover the banks once.
// What bounds it: the shared-memory reads of the two 32 x 128 x 128 products (5
// wavefronts for 16 multiply-adds of a warp), then FMA issue.  4096 tasks: 201 us
// with 64 CTAs of 128 threads that kept the weight gradients in shared memory and
// summed one unit per thread, 33 us so.  Relative error of dW2 against 64 bits, two
// seeds: 3.5e-7 and 3.0e-7 before, 3.3e-7 and 2.5e-7 so at 4096 tasks; 3.9e-7 and
// 1.9e-7 before, 3.8e-7 and 0.9e-7 so at 200,000 (4.3e-7 and 1.4e-7 with one running
// sum over the tiles, which took 1.08 ms a call instead of 1.11).  Pre-training a cost model (2.3e6 tasks, 4 epochs) 562 -> 136 ms.
constexpr int kTrainThreads = 256;
constexpr int kPad = kH1 + 4;
constexpr int kPartStride = (kParams + 3) & ~3;  // floats between partial gradients (16-byte rows)

struct TrainSmem {
    float w2[kH2 * kPad];                   // 66 KiB: W2[j][i]
    float h1[kGroup * kPad];                // 16.5 KiB: relu(layer 1)
    float h2[kGroup * kPad];                // 16.5 KiB: relu(layer 2), then dL/d(pre-act 2)
    float dh1[kGroup * kPad];               // 16.5 KiB: dL/d(pre-act 1)
    float x[kGroup * kIn];                  // 12 KiB: the tasks' bits
    __nv_bfloat16 w1t[(kIn + 1) * kH1];     // 24.25 KiB: [input bit][unit], row kIn zero
    float w3[kH2], b1[kH1], b2[kH2];
    float dout[kGroup], y[kGroup], loss[kTrainThreads / 32];
    uint32_t m[3][kGroup];
    // 64 KiB: dW2 of the tiles before the current one, [vector of a thread][thread].
    // One running sum over all tiles of a CTA would be 1350 terms long at 200,000 tasks.
    float4 dw2[16][kTrainThreads];
};

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Partial gradient and squared error of tasks [begin, end) of the view
// (mean-squared-error loss with gradient scale `scale` = 2/batch), one of each
// per CTA.
__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_train_kernel(TaskView tv, const float *target, long long begin, long long end, float scale,
                     const Weights *w, float *grad_part, float *loss_part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrainSmem &S = *reinterpret_cast<TrainSmem *>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (int i = t; i < kIn * kH1 / 8; i += kTrainThreads)
        reinterpret_cast<uint4 *>(S.w1t)[i] = reinterpret_cast<const uint4 *>(w->w1t)[i];
    if (t < kH1 / 8) reinterpret_cast<uint4 *>(S.w1t + kIn * kH1)[t] = make_uint4(0, 0, 0, 0);
    for (int i = t; i < kH2 * kH1 / 2; i += kTrainThreads) {
        const uint32_t v = reinterpret_cast<const uint32_t *>(w->w2)[i];
        float *to = S.w2 + (2 * i / kH1) * kPad + 2 * i % kH1;
        to[0] = __uint_as_float(v << 16);
        to[1] = __uint_as_float(v & 0xffff0000u);
    }
    if (t < kH1) {
        S.b1[t] = w->b1[t];
        S.b2[t] = w->b2[t];
        S.w3[t] = __bfloat162float(w->w3[t]);
    }
    const float b3 = w->b3;
    const int ty = t >> 4, tx = t & 15;     // 16 x 16 threads of the weight gradients
    const int col = t & (kH1 - 1), half = t >> 7;  // column sums: a unit and half of the tasks
    float gw2[8][8] = {}, gw1[8][6] = {};
    float gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, loss = 0.f;
    __syncthreads();

    const long long first = begin + (long long)blockIdx.x * kGroup, second = first + (long long)gridDim.x * kGroup;
    for (long long g0 = first; g0 < end; g0 += (long long)gridDim.x * kGroup) {
        const int gn = (int)min((long long)kGroup, end - g0);
        if (t < kGroup) {
            S.m[0][t] = S.m[1][t] = S.m[2][t] = 0;
            S.y[t] = 0.f;
            if (t < gn) {
                load_masks(tv, g0 + t, S.m[0][t], S.m[1][t], S.m[2][t]);
                S.y[t] = target[tv.index ? (long long)tv.index[g0 + t] : g0 + t];
            }
        }
        __syncthreads();
        for (int i = t; i < kGroup * kIn; i += kTrainThreads) {
            const int s = i / kIn, f = i % kIn;
            S.x[i] = (float)(S.m[f >> 5][s] >> (f & 31) & 1u);
        }
        // ---- layer 1, four bits at a time (row kIn of W1t is zero).  The rows that fill a
        // tile up are zero in every layer: they have no error, but 0 times an infinite
        // activation would be NaN.
        for (int s = warp; s < kGroup; s += kTrainThreads / 32) {
            float4 acc = ld4(S.b1 + 4 * lane);
#pragma unroll
            for (int part = 0; part < 3; ++part)
                for (uint32_t m = S.m[part][s]; m;) {
                    uint2 v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int f = m ? 32 * part + __ffs(m) - 1 : kIn;
                        m &= m - 1;
                        v[k] = *reinterpret_cast<const uint2 *>(S.w1t + f * kH1 + 4 * lane);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        acc.x += __uint_as_float(v[k].x << 16);
                        acc.y += __uint_as_float(v[k].x & 0xffff0000u);
                        acc.z += __uint_as_float(v[k].y << 16);
                        acc.w += __uint_as_float(v[k].y & 0xffff0000u);
                    }
                }
            if (s >= gn) acc = make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<float4 *>(S.h1 + s * kPad + 4 * lane) =
                make_float4(fmaxf(acc.x, 0.f), fmaxf(acc.y, 0.f), fmaxf(acc.z, 0.f), fmaxf(acc.w, 0.f));
        }
        __syncthreads();
        // ---- layer 2: tasks 4*warp.., units lane + 32 q
        {
            float acc[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[r][q] = S.b2[lane + 32 * q];
            const float *hp = S.h1 + 4 * warp * kPad, *wp = S.w2 + lane * kPad;
#pragma unroll 4
            for (int i = 0; i < kH1; i += 4) {
                float4 h[4], v[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) h[r] = ld4(hp + r * kPad + i);
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = ld4(wp + 32 * q * kPad + i);
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[r][q] = fmaf(h[r].x, v[q].x, acc[r][q]);
                        acc[r][q] = fmaf(h[r].y, v[q].y, acc[r][q]);
                        acc[r][q] = fmaf(h[r].z, v[q].z, acc[r][q]);
                        acc[r][q] = fmaf(h[r].w, v[q].w, acc[r][q]);
                    }
            }
            // ---- layer 3 and its error, for the warp's own four tasks
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int s = 4 * warp + r;
                float a = 0.f;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[r][q] = s < gn ? fmaxf(acc[r][q], 0.f) : 0.f;
                    S.h2[s * kPad + lane + 32 * q] = acc[r][q];
                    a = fmaf(acc[r][q], S.w3[lane + 32 * q], a);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (lane == 0) {
                    const float e = (s < gn) ? (a + b3 - S.y[s]) : 0.f;
                    S.dout[s] = scale * e;
                    loss += e * e;
                }
            }
        }
        __syncthreads();
        // ---- layer 3 and relu of layer 2 backward
        for (int s = half * (kGroup / 2); s < (half + 1) * (kGroup / 2); ++s) {
            const float h = S.h2[s * kPad + col], d = S.dout[s];
            gw3 = fmaf(d, h, gw3);
            const float dh = (h > 0.f) ? d * S.w3[col] : 0.f;
            S.h2[s * kPad + col] = dh;
            gb2 += dh;
            if (col == 0) gb3 += d;
        }
        __syncthreads();
        // ---- dH1 = relu' . dH2 W2: tasks 4*warp.., units 4*lane..
        bool unbounded = false;  // an infinite or NaN dH1
        {
            float acc[4][4] = {};
            const float *dp = S.h2 + 4 * warp * kPad, *wp = S.w2 + 4 * lane;
#pragma unroll 4
            for (int j = 0; j < kH2; j += 4) {
                float4 d[4], v[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) d[r] = ld4(dp + r * kPad + j);
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = ld4(wp + (j + q) * kPad);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float dd[4] = {d[r].x, d[r].y, d[r].z, d[r].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        acc[r][0] = fmaf(dd[q], v[q].x, acc[r][0]);
                        acc[r][1] = fmaf(dd[q], v[q].y, acc[r][1]);
                        acc[r][2] = fmaf(dd[q], v[q].z, acc[r][2]);
                        acc[r][3] = fmaf(dd[q], v[q].w, acc[r][3]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int s = 4 * warp + r;
                const float4 h = ld4(S.h1 + s * kPad + 4 * lane);
                const float4 d =
                    make_float4(h.x > 0.f ? acc[r][0] : 0.f, h.y > 0.f ? acc[r][1] : 0.f, h.z > 0.f ? acc[r][2] : 0.f,
                                h.w > 0.f ? acc[r][3] : 0.f);
                *reinterpret_cast<float4 *>(S.dh1 + s * kPad + 4 * lane) = d;
                unbounded |= !(fabsf((d.x + d.y) + (d.z + d.w)) <= 3.4e38f);
            }
        }
        unbounded = __syncthreads_or(unbounded);
        // ---- the last tile's dW2 joins those before it
        if (g0 != first) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                float *r = &gw2[q >> 1][(q & 1) * 4];
                if (g0 != second) {
                    const float4 v = S.dw2[q][t];
                    r[0] += v.x, r[1] += v.y, r[2] += v.z, r[3] += v.w;
                }
                S.dw2[q][t] = make_float4(r[0], r[1], r[2], r[3]);
                r[0] = r[1] = r[2] = r[3] = 0.f;
            }
        }
        // ---- dW2 and dW1: rows 4*ty + {0..3, 64..67}; columns 4*tx + {0..3, 64..67}
        // of dW2 and 2*tx + 32*q + {0, 1} of dW1.  dW1 is the sum of dH1 over the tasks
        // that have the bit set: a product with the bits, unless dH1 is unbounded.
#pragma unroll 2
        for (int s = 0; s < kGroup; ++s) {
            const float4 da = ld4(S.h2 + s * kPad + 4 * ty), db = ld4(S.h2 + s * kPad + 64 + 4 * ty);
            const float4 ha = ld4(S.h1 + s * kPad + 4 * tx), hb = ld4(S.h1 + s * kPad + 64 + 4 * tx);
            const float d[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
            const float h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int b = 0; b < 8; ++b) gw2[a][b] = fmaf(d[a], h[b], gw2[a][b]);
        }
        auto dw1 = [&](auto add) {
#pragma unroll 2
            for (int s = 0; s < kGroup; ++s) {
                const float4 da = ld4(S.dh1 + s * kPad + 4 * ty), db = ld4(S.dh1 + s * kPad + 64 + 4 * ty);
                const float d[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
                float x[6];
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    const float2 v = *reinterpret_cast<const float2 *>(S.x + s * kIn + 2 * tx + 32 * q);
                    x[2 * q] = v.x;
                    x[2 * q + 1] = v.y;
                }
#pragma unroll
                for (int a = 0; a < 8; ++a)
#pragma unroll
                    for (int b = 0; b < 6; ++b) gw1[a][b] = add(d[a], x[b], gw1[a][b]);
            }
        };
        if (unbounded)
            dw1([](float d, float x, float sum) { return x != 0.f ? sum + d : sum; });
        else
            dw1([](float d, float x, float sum) { return fmaf(d, x, sum); });
        for (int s = half * (kGroup / 2); s < (half + 1) * (kGroup / 2); ++s) gb1 += S.dh1[s * kPad + col];
        __syncthreads();
    }

    if (second < end) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            float *r = &gw2[q >> 1][(q & 1) * 4];
            const float4 v = S.dw2[q][t];
            r[0] += v.x, r[1] += v.y, r[2] += v.z, r[3] += v.w;
        }
    }
    // ---- partial gradient of this CTA in the flat parameter layout
    float *g = grad_part + (size_t)blockIdx.x * kPartStride;
#pragma unroll
    for (int a = 0; a < 8; ++a) {
        const int row = 4 * ty + (a & 3) + 16 * (a & 4);
        float *g1 = g + kOffW1 + row * kIn + 2 * tx, *g2 = g + kOffW2 + row * kH1 + 4 * tx;
#pragma unroll
        for (int q = 0; q < 3; ++q)
            *reinterpret_cast<float2 *>(g1 + 32 * q) = make_float2(gw1[a][2 * q], gw1[a][2 * q + 1]);
        *reinterpret_cast<float4 *>(g2) = make_float4(gw2[a][0], gw2[a][1], gw2[a][2], gw2[a][3]);
        *reinterpret_cast<float4 *>(g2 + 64) = make_float4(gw2[a][4], gw2[a][5], gw2[a][6], gw2[a][7]);
    }
    // column sums: the second half of the tasks through shared memory
    float *other = S.h1;
    if (half) {
        other[col] = gb1;
        other[kH1 + col] = gb2;
        other[2 * kH1 + col] = gw3;
        if (col == 0) other[3 * kH1] = gb3;
    }
    if (lane == 0) S.loss[warp] = loss;
    __syncthreads();
    if (!half) {
        g[kOffB1 + col] = gb1 + other[col];
        g[kOffB2 + col] = gb2 + other[kH1 + col];
        g[kOffW3 + col] = gw3 + other[2 * kH1 + col];
        if (col == 0) g[kOffB3] = gb3 + other[3 * kH1];
    }
    if (t == 0) {
        float l = 0.f;
        for (int k = 0; k < kTrainThreads / 32; ++k) l += S.loss[k];
        loss_part[blockIdx.x] = l;
    }
}
static_assert(sizeof(TrainSmem) <= 227 * 1024, "shared memory of one CTA");
static_assert(kGroup == 4 * (kTrainThreads / 32) && kOffW2 % 4 == 0 && kOffW1 % 2 == 0, "tile and vector layout");

// Master weights -> compute copy (round to nearest even BF16).
__device__ __forceinline__ void refresh_one(int p, float v, Weights *w) {
    if (p < kOffB1) {
        const int i = (p - kOffW1) / kIn, f = (p - kOffW1) % kIn;
        w->w1t[f * kH1 + i] = __float2bfloat16_rn(v);
        w->w1c[off_kmajor(i, f, kSbo1) / 2] = __float2bfloat16_rn(v);
    } else if (p < kOffW2) {
        w->b1[p - kOffB1] = v;
    } else if (p < kOffB2) {
        const int j = (p - kOffW2) / kH1, i = (p - kOffW2) % kH1;
        w->w2[p - kOffW2] = __float2bfloat16_rn(v);
        w->w2c[off_kmajor(j, i, kSbo2) / 2] = __float2bfloat16_rn(v);
    } else if (p < kOffW3) {
        w->b2[p - kOffB2] = v;
    } else if (p < kOffB3) {
        w->w3[p - kOffW3] = __float2bfloat16_rn(v);
    } else {
        w->b3 = v;
    }
}

__global__ void mlp_refresh_kernel(const float *master, Weights *w) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < kParams; p += gridDim.x * blockDim.x)
        refresh_one(p, master[p], w);
}

// Sums the per-CTA partial gradients (deterministic: four interleaved runs over
// the CTAs, then those in order), applies one Adam step to the master weights and
// refreshes the compute copy.  With apply == 0 it only sums (gradient check):
// grad_out receives the gradient.  64 parameters x 4 runs per CTA: the reads of
// 15 MB of partials (128 CTAs) have four times the loads in flight of one thread
// per parameter.
constexpr int kSumRuns = 4, kSumParams = 64;
__global__ void __launch_bounds__(kSumRuns * kSumParams)
    mlp_adam_kernel(float *master, float *m1, float *m2, const float *grad_part, int nparts, float lr, float beta1,
                    float beta2, float eps, float bc1, float bc2, Weights *w, float *grad_out, int apply) {
    __shared__ float s_sum[kSumRuns][kSumParams];
    const int x = threadIdx.x % kSumParams, run = threadIdx.x / kSumParams;
    const int p = blockIdx.x * kSumParams + x;
    float g = 0.f;
    if (p < kParams) {
#pragma unroll 8
        for (int b = run; b < nparts; b += kSumRuns) g += grad_part[(size_t)b * kPartStride + p];
    }
    s_sum[run][x] = g;
    __syncthreads();
    if (run || p >= kParams) return;
    g = (s_sum[0][x] + s_sum[1][x]) + (s_sum[2][x] + s_sum[3][x]);
    if (grad_out) grad_out[p] = g;
    if (!apply) return;
    const float a = beta1 * m1[p] + (1.f - beta1) * g;
    const float v = beta2 * m2[p] + (1.f - beta2) * g * g;
    m1[p] = a;
    m2[p] = v;
    const float upd = (a / bc1) / (sqrtf(v / bc2) + eps);
    const float nw = master[p] - lr * upd;
    master[p] = nw;
    refresh_one(p, nw, w);
}

// Moves the listed tasks behind every other task of the order (key 0).
// Indices at or beyond n are ignored.
__global__ void mlp_last_kernel(const uint32_t *last, long long n_last, long long n, uint16_t *key) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_last;
         i += (long long)gridDim.x * blockDim.x) {
        const uint32_t t = last[i];
        if ((long long)t < n) key[t] = 0;
    }
}

}  // namespace
}  // namespace nqb

using namespace nqb;

struct nq_mlp {
    std::mutex mu;
    int device = 0;
    int sms = 0;
    cudaStream_t stream = nullptr;
    void *block = nullptr;  // holds the next five
    float *master = nullptr, *adam1 = nullptr, *adam2 = nullptr;
    Weights *w = nullptr;
    long long steps = 0;
    // scratch
    float *grad_part = nullptr;
    int grad_parts_cap = 0;
    float *gsum = nullptr;  // summed gradient (nq_mlp_grad)
    // kErr* words of the forward kernels: [0] nq_mlp_predict*, [1] the scheduler.  In
    // host memory (take_err_words), so that reading them costs a call neither a
    // memset nor a copy.
    volatile int *err = nullptr;
    unsigned long long wait_limit = tc::kWaitLimit;
    void *loss_part = nullptr;  // floats
    size_t loss_cap = 0;
    void *data = nullptr;
    size_t data_cap = 0;
    void *sort_tmp = nullptr;
    size_t sort_tmp_cap = 0;
};

namespace {

int mlp_fail(cudaError_t e, const char *what) {
    set_last_error((std::string(what) + ": " + cudaGetErrorString(e)).c_str());
    (void)cudaGetLastError();
    return e == cudaErrorMemoryAllocation ? NQ_ERR_OOM : NQ_ERR_CUDA;
}

#define MLP_CUDA(call)                                          \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return mlp_fail(e_, #call);      \
    } while (0)

int grow(void *&p, size_t &cap, size_t need) {
    if (need <= cap) return NQ_OK;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    const size_t want = need + need / 4 + 256;
    MLP_CUDA(cudaMalloc(&p, want));
    cap = want;
    return NQ_OK;
}

// Error words of models come from pinned pages of 64 models each, kept until exit:
// a pinned allocation of its own took a model's creation from 1.1 to 4.2 ms.
constexpr size_t kErrPage = 4096, kErrSlot = 64;
std::mutex g_err_mu;
std::vector<volatile int *> &g_err_free = *new std::vector<volatile int *>;  // outlives every model
size_t g_err_slots = 0;

cudaError_t take_err_words(volatile int *&words) {
    std::lock_guard<std::mutex> lock(g_err_mu);
    if (g_err_free.empty()) {
        g_err_free.reserve(g_err_slots + kErrPage / kErrSlot);  // room for every slot, so that giving back cannot fail
        void *page = nullptr;
        const cudaError_t e = cudaHostAlloc(&page, kErrPage, cudaHostAllocPortable);
        if (e != cudaSuccess) return e;
        g_err_slots += kErrPage / kErrSlot;
        for (size_t at = 0; at < kErrPage; at += kErrSlot) g_err_free.push_back((volatile int *)((char *)page + at));
    }
    words = g_err_free.back();
    g_err_free.pop_back();
    words[0] = words[1] = 0;
    return cudaSuccess;
}

void give_err_words(volatile int *words) {
    if (!words) return;
    std::lock_guard<std::mutex> lock(g_err_mu);
    g_err_free.push_back(words);
}

int train_blocks(nq_mlp *m) { return m->sms; }

uint64_t splitmix(uint64_t &s) {
    s += 0x9E3779B97F4A7C15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Uploads a task list (+ per-task N and targets) into the model's scratch:
// [cols | ld | rd | index] u32, [target] f32, [task_n] u8.
struct Staged {
    uint32_t *cols, *ld, *rd, *index;
    float *target;
    uint8_t *task_n;
};

int stage(nq_mlp *m, const uint8_t *task_n, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd,
          const float *target, int64_t n, Staged &st) {
    const size_t need = (size_t)n * (4 * 4 + 4 + 1) + 1024;
    int rc = grow(m->data, m->data_cap, need);
    if (rc) return rc;
    char *b = (char *)m->data;
    st.cols = (uint32_t *)b;
    st.ld = st.cols + n;
    st.rd = st.ld + n;
    st.index = st.rd + n;
    st.target = (float *)(st.index + n);
    st.task_n = (uint8_t *)(st.target + n);
    MLP_CUDA(cudaMemcpyAsync(st.cols, cols, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    MLP_CUDA(cudaMemcpyAsync(st.ld, ld, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    MLP_CUDA(cudaMemcpyAsync(st.rd, rd, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    if (target) MLP_CUDA(cudaMemcpyAsync(st.target, target, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    if (task_n) MLP_CUDA(cudaMemcpyAsync(st.task_n, task_n, (size_t)n, cudaMemcpyHostToDevice, m->stream));
    return NQ_OK;
}

// Room for `parts` partial gradients and `losses` partial losses.
int ensure_grad_parts(nq_mlp *m, int parts, size_t losses) {
    if (parts > m->grad_parts_cap) {
        if (m->grad_part) cudaFree(m->grad_part);
        m->grad_part = nullptr;
        m->grad_parts_cap = 0;
        MLP_CUDA(cudaMalloc(&m->grad_part, (size_t)parts * kPartStride * sizeof(float)));
        m->grad_parts_cap = parts;
    }
    return grow(m->loss_part, m->loss_cap, losses * sizeof(float));
}

// CTAs (and partial gradients) of a minibatch of `count` tasks: one per tile of
// kGroup tasks up to one per SM (the kernel takes most of its shared memory).
int train_parts(nq_mlp *m, long long count) {
    return (int)std::min<long long>(train_blocks(m), std::max<long long>((count + kGroup - 1) / kGroup, 1));
}

// One forward+backward over [begin, end) into the first `parts` partial
// gradients and d_loss[0..parts).
int launch_train(nq_mlp *m, const TaskView &tv, const float *target, long long begin, long long end, float scale,
                 int parts, float *d_loss) {
    mlp_train_kernel<<<parts, kTrainThreads, sizeof(TrainSmem), m->stream>>>(tv, target, begin, end, scale, m->w,
                                                                             m->grad_part, d_loss);
    MLP_CUDA(cudaGetLastError());
    return NQ_OK;
}

void launch_adam(nq_mlp *m, int parts, float lr, float beta1, float beta2, float eps, float bc1, float bc2,
                 float *grad_out, int apply) {
    mlp_adam_kernel<<<(kParams + kSumParams - 1) / kSumParams, kSumRuns * kSumParams, 0, m->stream>>>(
        m->master, m->adam1, m->adam2, m->grad_part, parts, lr, beta1, beta2, eps, bc1, bc2, m->w, grad_out, apply);
}

// Forward pass over n device-resident tasks of board size N (parts: see
// mlp_forward_kernel).  One CTA per SM; a short list spreads its tiles over the
// SMs before it fills their groups.
int launch_forward(nq_mlp *m, int parts, const TaskView &tv, long long n, float *d_out, uint16_t *key, uint32_t *idx,
                   cudaStream_t s) {
    const int grid = (int)std::min<long long>((n + 127) / 128, m->sms);
    if (parts == 1)
        mlp_forward_kernel<1>
            <<<grid, 512, tc::kSmemBytes, s>>>(tv, n, m->w, d_out, key, idx, m->err + (key ? 1 : 0), m->wait_limit);
    else
        mlp_forward_kernel<3><<<grid, 256, tc::kSmemBytes, s>>>(tv, n, m->w, d_out, key, idx, m->err, m->wait_limit);
    MLP_CUDA(cudaGetLastError());
    return NQ_OK;
}

// What the forward kernels reported since the last look (they have finished).
int take_error(volatile int *err) {
    const int e = *err;
    *err = 0;
    if (e == kErrWait) set_last_error("tensor-core MMA completion wait expired");
    return e;
}

// Predictions of n host tasks into a host array.
int predict_host(nq_mlp *m, int parts, int N, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd, int64_t n,
                 float *out) {
    Staged st;
    int rc = stage(m, nullptr, cols, ld, rd, nullptr, n, st);
    if (rc) return rc;
    TaskView tv{st.cols, st.ld, st.rd, nullptr, nullptr, N};
    rc = launch_forward(m, parts, tv, n, st.target, nullptr, nullptr, m->stream);
    if (rc) return rc;
    MLP_CUDA(cudaMemcpyAsync(out, st.target, (size_t)n * 4, cudaMemcpyDeviceToHost, m->stream));
    MLP_CUDA(cudaStreamSynchronize(m->stream));
    const int e = take_error(m->err);
    if (e == kErrWide) {
        const int grid = (int)std::min<long long>((n + kGroup - 1) / kGroup, (long long)m->sms * 8);
        mlp_predict_kernel<<<grid, kH1, 0, m->stream>>>(tv, n, m->w, st.target);
        MLP_CUDA(cudaGetLastError());
        MLP_CUDA(cudaMemcpyAsync(out, st.target, (size_t)n * 4, cudaMemcpyDeviceToHost, m->stream));
        MLP_CUDA(cudaStreamSynchronize(m->stream));
    }
    return e == kErrWait ? NQ_ERR_TIMEOUT : NQ_OK;
}

int check_model(nq_mlp *m) {
    if (!m) return NQ_ERR_ARG;
    MLP_CUDA(cudaSetDevice(m->device));
    return NQ_OK;
}

}  // namespace

// For nq_count_learned (capi.cu): forgets the scheduler's expired waits, and
// tells whether one has expired since (its stream synchronised).
namespace nqb {
void clear_schedule_error(nq_mlp *m) { m->err[1] = 0; }
bool schedule_error(nq_mlp *m) { return take_error(m->err + 1) == kErrWait; }
}  // namespace nqb

extern "C" {

int nq_mlp_num_params(void) { return kParams; }

int nq_mlp_create(int device, uint64_t seed, nq_mlp **out) try {
    if (!out) return NQ_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        (void)cudaGetLastError();
        set_last_error("no CUDA device");
        return NQ_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= ndev) return NQ_ERR_ARG;
    MLP_CUDA(cudaSetDevice(device));
    nq_mlp *m = new nq_mlp();
    m->device = device;
    cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device);
    cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    // one allocation for everything whose size is known here
    auto room = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    const size_t vec = room(kParams * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->block, 4 * vec + room(sizeof(Weights)));
    if (e == cudaSuccess) e = take_err_words(m->err);
    char *at = (char *)m->block;
    for (float **v : {&m->master, &m->adam1, &m->adam2, &m->gsum}) {
        *v = (float *)at;
        at += vec;
    }
    m->w = (Weights *)at;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_forward_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_forward_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc::kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(TrainSmem));
    if (e != cudaSuccess) {
        nq_mlp_destroy(m);
        return mlp_fail(e, "nq_mlp_create");
    }
    // Uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) for every weight and bias,
    // from SplitMix64(seed).
    std::vector<float> p(kParams);
    uint64_t s = seed;
    auto uni = [&](float bound) {
        const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
        return (float)((2.0 * u - 1.0) * bound);
    };
    for (int i = kOffW1; i < kOffB1; ++i) p[i] = uni(1.f / std::sqrt((float)kIn));
    for (int i = kOffB1; i < kOffW2; ++i) p[i] = uni(1.f / std::sqrt((float)kIn));
    for (int i = kOffW2; i < kOffB2; ++i) p[i] = uni(1.f / std::sqrt((float)kH1));
    for (int i = kOffB2; i < kOffW3; ++i) p[i] = uni(1.f / std::sqrt((float)kH1));
    for (int i = kOffW3; i < kOffB3; ++i) p[i] = uni(1.f / std::sqrt((float)kH2));
    p[kOffB3] = uni(1.f / std::sqrt((float)kH2));
    *out = m;
    return nq_mlp_set_params(m, p.data());
} catch (...) {
    return status_of_exception();
}

int nq_mlp_destroy(nq_mlp *m) try {
    if (!m) return NQ_OK;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->block);
    cudaFree(m->grad_part);
    cudaFree(m->loss_part);
    cudaFree(m->data);
    cudaFree(m->sort_tmp);
    give_err_words(m->err);  // after cudaFree, which waits for the device
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_mlp_get_params(nq_mlp *m, float *out) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (!out) return NQ_ERR_ARG;
    std::lock_guard<std::mutex> lock(m->mu);
    MLP_CUDA(cudaMemcpyAsync(out, m->master, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MLP_CUDA(cudaStreamSynchronize(m->stream));
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_mlp_set_params(nq_mlp *m, const float *in) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (!in) return NQ_ERR_ARG;
    std::lock_guard<std::mutex> lock(m->mu);
    MLP_CUDA(cudaMemcpyAsync(m->master, in, kParams * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MLP_CUDA(cudaMemsetAsync(m->adam1, 0, kParams * sizeof(float), m->stream));
    MLP_CUDA(cudaMemsetAsync(m->adam2, 0, kParams * sizeof(float), m->stream));
    mlp_refresh_kernel<<<(kParams + 255) / 256, 256, 0, m->stream>>>(m->master, m->w);
    MLP_CUDA(cudaGetLastError());
    MLP_CUDA(cudaStreamSynchronize(m->stream));
    m->steps = 0;
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_mlp_set_wait_limit(nq_mlp *m, uint64_t polls) try {
    if (!m) return NQ_ERR_ARG;
    std::lock_guard<std::mutex> lock(m->mu);
    m->wait_limit = std::min<uint64_t>(polls, tc::kWaitLimit);
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_mlp_predict(nq_mlp *m, int N, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd, int64_t n,
                   float *out) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (N < 1 || N > NQ_MAX_N || n < 0 || (n > 0 && (!cols || !ld || !rd || !out))) return NQ_ERR_ARG;
    if (n == 0) return NQ_OK;
    std::lock_guard<std::mutex> lock(m->mu);
    return predict_host(m, 3, N, cols, ld, rd, n, out);
} catch (...) {
    return status_of_exception();
}

int nq_mlp_predict_tensor(nq_mlp *m, int N, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd, int64_t n,
                          float *out) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (N < 1 || N > NQ_MAX_N || n < 0 || (n > 0 && (!cols || !ld || !rd || !out))) return NQ_ERR_ARG;
    if (n == 0) return NQ_OK;
    std::lock_guard<std::mutex> lock(m->mu);
    return predict_host(m, 1, N, cols, ld, rd, n, out);
} catch (...) {
    return status_of_exception();
}

int nq_mlp_grad(nq_mlp *m, const uint8_t *task_n, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd,
                const float *target, int64_t n, float *grad_out, float *loss_out) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (n <= 0 || !task_n || !cols || !ld || !rd || !target || !grad_out) return NQ_ERR_ARG;
    std::lock_guard<std::mutex> lock(m->mu);
    Staged st;
    rc = stage(m, task_n, cols, ld, rd, target, n, st);
    if (rc) return rc;
    TaskView tv{st.cols, st.ld, st.rd, st.task_n, nullptr, 0};
    const int parts = train_parts(m, n);
    rc = ensure_grad_parts(m, parts, parts);
    if (rc) return rc;
    rc = launch_train(m, tv, st.target, 0, n, 2.f / (float)n, parts, (float *)m->loss_part);
    if (rc) return rc;
    launch_adam(m, parts, 0.f, 0.f, 0.f, 0.f, 1.f, 1.f, m->gsum, 0);
    cudaError_t e = cudaGetLastError();
    std::vector<float> lp(parts);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(grad_out, m->gsum, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(lp.data(), m->loss_part, parts * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
    if (e != cudaSuccess) return mlp_fail(e, "nq_mlp_grad");
    if (loss_out) {
        double l = 0;
        for (float v : lp) l += v;
        *loss_out = (float)(l / (double)n);
    }
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_mlp_train(nq_mlp *m, const uint8_t *task_n, const uint32_t *cols, const uint32_t *ld, const uint32_t *rd,
                 const float *target, int64_t n, int epochs, int batch, float lr, uint64_t seed,
                 float *epoch_loss) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (n <= 0 || !task_n || !cols || !ld || !rd || !target || epochs < 0 || batch < kGroup || lr <= 0.f)
        return NQ_ERR_ARG;
    if (n > 0xffffffffll) return NQ_ERR_ARG;
    std::lock_guard<std::mutex> lock(m->mu);
    Staged st;
    rc = stage(m, task_n, cols, ld, rd, target, n, st);
    if (rc) return rc;
    std::vector<uint32_t> perm((size_t)n);
    uint64_t s = seed;
    const int parts_max = train_parts(m, batch);
    const long long nsteps_epoch = (n + batch - 1) / batch;
    // The losses of an epoch's steps stay on the device until its end: a copy per
    // step would make the host wait for each.
    rc = ensure_grad_parts(m, parts_max, (size_t)parts_max * nsteps_epoch);
    if (rc) return rc;
    std::vector<float> lp((size_t)parts_max * nsteps_epoch);
    for (int ep = 0; ep < epochs; ++ep) {
        // Fisher-Yates shuffle from SplitMix64(seed), one per epoch.
        for (int64_t i = 0; i < n; ++i) perm[i] = (uint32_t)i;
        for (int64_t i = n - 1; i > 0; --i) {
            const int64_t k = (int64_t)(splitmix(s) % (uint64_t)(i + 1));
            std::swap(perm[i], perm[k]);
        }
        MLP_CUDA(cudaMemcpyAsync(st.index, perm.data(), (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
        TaskView tv{st.cols, st.ld, st.rd, st.task_n, st.index, 0};
        double eloss = 0;
        for (long long b0 = 0, stepi = 0; b0 < n; b0 += batch, ++stepi) {
            const long long b1 = std::min<long long>(n, b0 + batch);
            const int parts = train_parts(m, b1 - b0);
            float *d_loss = (float *)m->loss_part + (size_t)stepi * parts_max;
            rc = launch_train(m, tv, st.target, b0, b1, 2.f / (float)(b1 - b0), parts, d_loss);
            if (rc) return rc;
            if (parts < parts_max) MLP_CUDA(cudaMemsetAsync(d_loss + parts, 0, (parts_max - parts) * 4, m->stream));
            m->steps += 1;
            const float bc1 = 1.f - std::pow(0.9f, (float)m->steps);
            const float bc2 = 1.f - std::pow(0.999f, (float)m->steps);
            launch_adam(m, parts, lr, 0.9f, 0.999f, 1e-8f, bc1, bc2, nullptr, 1);
            MLP_CUDA(cudaGetLastError());
        }
        if (epoch_loss) {
            MLP_CUDA(cudaMemcpyAsync(lp.data(), m->loss_part, lp.size() * sizeof(float), cudaMemcpyDeviceToHost,
                                     m->stream));
            MLP_CUDA(cudaStreamSynchronize(m->stream));
            for (float v : lp) eloss += v;
            epoch_loss[ep] = (float)(eloss / (double)n);
        }
    }
    MLP_CUDA(cudaStreamSynchronize(m->stream));
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

// Longest-first order of device-resident tasks: predictions -> keys in
// 1/8-log2 bins -> stable descending radix sort of task indices.
int nq_schedule_device_last(nq_mlp *m, int N, const uint32_t *d_cols, const uint32_t *d_ld, const uint32_t *d_rd,
                            int64_t n, const uint32_t *d_last, int64_t n_last, uint32_t *d_order, float *d_pred,
                            void *stream) try {
    int rc = check_model(m);
    if (rc) return rc;
    if (N < 1 || N > NQ_MAX_N || n < 0 || n > 0xffffffffll || (n > 0 && (!d_cols || !d_ld || !d_rd || !d_order)))
        return NQ_ERR_ARG;
    if (n_last < 0 || (n_last > 0 && !d_last)) return NQ_ERR_ARG;
    if (n == 0) return NQ_OK;
    std::lock_guard<std::mutex> lock(m->mu);
    cudaStream_t s = (cudaStream_t)stream;  // NULL: the legacy default stream, as in every device entry
    // scratch: key u16 | key_out u16 | idx u32
    const size_t need = (size_t)n * (2 + 2 + 4) + 1024;
    rc = grow(m->data, m->data_cap, need);
    if (rc) return rc;
    uint16_t *key = (uint16_t *)m->data;
    uint16_t *key2 = key + n;
    uint32_t *idx = (uint32_t *)(((uintptr_t)(key2 + n) + 15) & ~(uintptr_t)15);
    TaskView tv{d_cols, d_ld, d_rd, nullptr, nullptr, N};
    rc = launch_forward(m, 1, tv, n, d_pred, key, idx, s);
    if (rc) return rc;
    if (n_last > 0) {
        mlp_last_kernel<<<m->sms * 4, 256, 0, s>>>(d_last, n_last, n, key);
        MLP_CUDA(cudaGetLastError());
    }
    size_t tmp = 0;
    MLP_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, key, key2, idx, d_order, (int)n, 0, 16, s));
    rc = grow(m->sort_tmp, m->sort_tmp_cap, tmp);
    if (rc) return rc;
    MLP_CUDA(cub::DeviceRadixSort::SortPairsDescending(m->sort_tmp, tmp, key, key2, idx, d_order, (int)n, 0, 16, s));
    return NQ_OK;
} catch (...) {
    return status_of_exception();
}

int nq_schedule_device(nq_mlp *m, int N, const uint32_t *d_cols, const uint32_t *d_ld, const uint32_t *d_rd,
                       int64_t n, uint32_t *d_order, float *d_pred, void *stream) try {
    return nq_schedule_device_last(m, N, d_cols, d_ld, d_rd, n, nullptr, 0, d_order, d_pred, stream);
} catch (...) {
    return status_of_exception();
}

}  // extern "C"
