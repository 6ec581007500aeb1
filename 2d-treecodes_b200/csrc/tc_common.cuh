// tc_common.cuh -- shared constants, error plumbing and device helpers of the B200 treecode.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#include "treecodes_b200.h"

namespace tc {

// Compile-time parameters of the reference build (Makefile:13-15 of the reference,
// drivers/Makefile:20): expansion order 12 for the potential, 24 for the force, MRAG block
// of 32 x 32 targets, deepest level 15, leaf capacities 512 / 192
// (drivers/treecode-potential.cpp:99, drivers/treecode-force.cpp:216), bricks of 8 x 8
// (drivers/treecode-force.cpp:91).
constexpr int LMAX = 15;
constexpr int BLOCKSIZE = 32;
constexpr int TILE = 8;
constexpr int ORDER_POTENTIAL = 12;
constexpr int ORDER_FORCE = 24;
constexpr int LEAF_POTENTIAL = 32 * 16;
constexpr int LEAF_FORCE = 192;
constexpr int MAX_ORDER = 32;

// Status codes: tc_status of the C ABI (treecodes_b200.h).

// Device-side error word bits (set by kernels, read by the host after the call).
enum DeviceError : unsigned {
    DEVERR_SPIN_LIMIT = 1u << 0,   // a bounded wait gave up
    DEVERR_STACK = 1u << 1,        // traversal stack overflow
    DEVERR_TREE = 1u << 2,         // inconsistent tree bookkeeping
    DEVERR_BOUNDS = 1u << 3,       // an index failed its bounds check (access skipped)
};

// Coordinate frame of a source set: sort-sources.cpp:78-82 of the reference.
struct Frame {
    double xmin, ymin, ext;   // padded bounding square
    double scale;             // (1 / ext) * 2^LMAX, the factor the compiled reference uses
};

// Targets and sources that differ by less than this in x and in y have squared distances below
// 2 (2^509)^2 = 2^1019, which the FP64 potential's logarithm and reciprocal are made for (log_near).
constexpr double NEAR_REACH = 0x1p509;

// A brick's near field is cut into segments of P2P_SEG sources, so that the few bricks on a dense
// region do not serialise the kernel.  The segments also fix the grid of source tiles (a
// segment's tiles start at its own start, at a leaf's start, or 32 sources after another), and
// with it how the mixed form's FP32 sums are grouped.
constexpr int P2P_SEG = 2048;
// With few bricks a segment is cut further, at tile starts, into tasks of `seg` sources (a
// divisor of P2P_SEG).
constexpr int P2P_MIN_SEG = 64;
constexpr int P2P_FULL_BRICKS = 32768;

// Near-field sources per task.  The kernel holds about 4700 resident warps; with whole segments
// fewer than ~32K bricks leave warps idle or waiting for the longest task.  The kernel alone,
// whole segments and this rule: 16 bricks (seg 64), mixed, 72 -> 35 us; 5476 bricks (seg 256),
// mixed, 126 -> 81 us; 16,384 bricks (seg 1024), FP64, 596 -> 555 us.
constexpr int near_segment(int nbricks) {
    int seg = P2P_SEG;
    while (seg > P2P_MIN_SEG && (long long)nbricks * P2P_SEG < (long long)P2P_FULL_BRICKS * seg)
        seg >>= 1;
    return seg;
}

constexpr unsigned FULL_MASK = 0xffffffffu;

// Reads without progress after which a device wait on another CTA's published state gives up
// and raises DEVERR_SPIN_LIMIT (a context's test setting can lower it, tc_set_wait_test).
constexpr int DEFAULT_SPIN_LIMIT = 1 << 22;

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// Programmatic dependent launch (launch_pdl): a kernel may be scheduled while the kernel before
// it on its stream is still draining.  A kernel so launched calls this before it reads what that
// kernel writes, and before it writes anything: it waits until that kernel has completed and its
// writes are visible, then lets the kernel after it be scheduled in turn.  Both are no-ops without
// the launch attribute.
// The order of the two is what early reads rest on.  Every kernel of a chain waits before it releases
// the next, so when a kernel starts, the one before it has seen its own predecessor complete:
// whatever is older than the preceding kernel may be read ahead of pdl_begin (merge_geom,
// k_moments_level, k_potential_gather_parts, the log tables), and nothing else.  A kernel that
// released the next before its wait would break every chain that it stands in.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Approximate FP64 reciprocal from the SFU (PTX rcp.approx.ftz.f64, good to about 2^-20), refined
// by one third-order step: with e = 1 - d y, 1/d = y / (1 - e) = y (1 + e + e^2) + O(e^3), so the
// error left is about 2^-60.  Three FP64 operations, against four of two Newton steps.
__device__ __forceinline__ double rcp_nr(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    const double t = fma(e, e, e);
    return fma(y, t, y);
}

// 1 / d for any d: rcp_nr from 2^-1000 to 2^1000 (its approximation flushes 1 / d to 0 from 2^1022
// on, and its correction makes a NaN of infinity), decided on the high word.
__device__ __forceinline__ double rcp_any(double d) {
    return (unsigned)__double2hiint(d) - 0x01700000u < 0x7e700000u - 0x01700000u ? rcp_nr(d) : 1.0 / d;
}

__device__ __forceinline__ double shfl_xor_d(double v, int m) {
    return __shfl_xor_sync(FULL_MASK, v, m);
}

// Morton interleave of a 15-bit coordinate: sort-sources.cpp:96-104 of the reference.
__host__ __device__ __forceinline__ int spread_bits(int x) {
    x = (x | (x << 8)) & 0x00FF00FF;
    x = (x | (x << 4)) & 0x0F0F0F0F;
    x = (x | (x << 2)) & 0x33333333;
    x = (x | (x << 1)) & 0x55555555;
    return x;
}

__host__ __device__ __forceinline__ int compact_bits(int x) {
    x &= 0x55555555;
    x = (x | (x >> 1)) & 0x33333333;
    x = (x | (x >> 2)) & 0x0F0F0F0F;
    x = (x | (x >> 4)) & 0x00FF00FF;
    x = (x | (x >> 8)) & 0x0000FFFF;
    return x;
}

// Node record read by the traversals: centre of mass, radius, first child (-1: leaf) and the
// number of sources the node hands to P2P (0 for empty leaves).
struct __align__(32) TNode {
    double xcom, ycom, r;
    int child;
    int count;
};

// Longest tasks first: persistent warps that take tasks from a counter end together only if no long
// task is taken late.  Tasks are appended to TASK_BINS bins of falling work, bin b at b * stride;
// `fill` counts each bin's tasks.  A consumer reads the counts once (every lane of the warp) and maps
// the i-th task to its place.
constexpr int TASK_BINS = 8;
struct TaskBins {
    int incl;   // lane b < TASK_BINS: tasks in bins 0 .. b
    __device__ __forceinline__ explicit TaskBins(const int *fill) {
        const int lane = threadIdx.x & 31;
        incl = fill && lane < TASK_BINS ? fill[lane] : 0;
        for (int o = 1; o < TASK_BINS; o <<= 1) {
            const int t = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= o) incl += t;
        }
    }
    // place of the i-th task, i below the total
    __device__ __forceinline__ int place(int i, int stride) const {
        const int lane = threadIdx.x & 31;
        const int bin = __popc(__ballot_sync(FULL_MASK, lane < TASK_BINS - 1 && incl <= i));
        const int before = __shfl_sync(FULL_MASK, incl, bin ? bin - 1 : 0);
        return bin * stride + i - (bin ? before : 0);
    }
};

// Block-wide exclusive scan of one int per thread (blockDim.x a multiple of 32, <= 1024); the
// block total goes to *total when total is not null.  Every thread of the block must call it.
__device__ __forceinline__ int block_exclusive_scan(int v, int *total) {
    __shared__ int warp_sums[32];
    const int lane = lane_id(), w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL_MASK, inc, o);
        if (lane >= o) inc += t;
    }
    __syncthreads();
    if (lane == 31) warp_sums[w] = inc;
    __syncthreads();
    if (w == 0) {
        int s = lane < nw ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL_MASK, s, o);
            if (lane >= o) s += t;
        }
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    const int base = w ? warp_sums[w - 1] : 0;
    if (total) *total = warp_sums[nw - 1];
    return base + inc - v;
}

}  // namespace tc

#define TC_CUDA_TRY(expr)                                                            \
    do {                                                                             \
        cudaError_t err__ = (expr);                                                  \
        if (err__ != cudaSuccess) {                                                  \
            ::tc::set_error(::TC_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__,       \
                            #expr, cudaGetErrorString(err__));                       \
            return ::TC_ERR_CUDA;                                                    \
        }                                                                            \
    } while (0)

// Every kernel launch site is followed by TC_KERNEL_CHECK(), which also counts the launch.
#define TC_KERNEL_CHECK()          \
    do {                           \
        ++::tc::g_launches;        \
        TC_CUDA_TRY(cudaGetLastError()); \
    } while (0)

namespace tc {
// Kernel launches issued by this thread since the counter was last reset (per solve).
extern thread_local long long g_launches;
// Records status and message for treecode_last_status / treecode_last_error (thread-local).
void set_error(int status, const char *fmt, ...);
}
