// sort.cu -- bounding square, Morton keys, LSD radix sort with a stable permutation, and the
// sorted source arrays.  Restates drivers/sort-sources.cpp:23-132 of the reference.
//
// Data flow per solve (N sources, all FP64 SoA in HBM), with the values resident (the device
// entry points):
//   k_bbox            x, y        -> Frame (xmin, ymin, ext, scale)          16 B/src read
//   k_key_hist        x, y        -> histograms of the 4 key digits and of   16 B read
//                                    the 256 spatial buckets (top 8 key bits)
//   k_onesweep_items  x, y, v     -> 32-byte records (x, y, v, index) in     24 B read, 40 B written
//     (first pass)                   their buckets, items (key << 32 | slot)
//                                    sorted by the first digit
//   k_onesweep_items  items       -> items sorted by the next 8-bit digit    8 B read, 8 B written
//                                    (3 passes)
//   k_gather_sources  items, recs -> sorted keys, permutation, x, y, v       8 B + one record
//                                                                            read, 32 B written
// With values that arrive after x and y (the host entry points): k_keys_pack writes the items
// (key << 32 | index) and the histograms, four passes sort them, k_items_split writes keys and
// permutation, k_gather_xy the sorted x and y, and k_gather_v the sorted v once it is in.
//
// Up to 16,384 sources (SMALL_SORT) all of it is one block and one launch, k_sort_small.
//
// The radix sort is a one-pass-per-digit ("onesweep") LSD sort: every CTA counts the digits of
// a tile of items, finds its global digit offsets by a decoupled look-back over the tiles
// before it, ranks the tile in shared memory with warp digit ballots and writes it out in
// runs of equal digits.  Tiles take their ids from an atomic counter, so each waits only on
// tiles that already run; the waits are bounded and raise DEVERR_SPIN_LIMIT instead of
// hanging.  Ties keep input order, so the order is the reference's (key, index) order.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "tc_internal.h"

namespace tc {

// ---------------------------------------------------------------------------- bbox
constexpr int BBOX_THREADS = 256;

__device__ __forceinline__ void warp_minmax(double &a, double &b, double &c, double &d) {
    for (int m = 16; m; m >>= 1) {
        a = fmin(a, shfl_xor_d(a, m));
        b = fmax(b, shfl_xor_d(b, m));
        c = fmin(c, shfl_xor_d(c, m));
        d = fmax(d, shfl_xor_d(d, m));
    }
}

// The padded square of extrema (xmin, xmax, ymin, ymax): sort-sources.cpp:98-110, with the
// arithmetic the compiled reference executes: ext = max(ex, ey) * (1 + 2 eps);
// xmin -= eps * ext; keys use (1/ext) * 2^15.
__device__ __forceinline__ Frame frame_of(const double4 &r) {
    const double eps = 10000.0 * DBL_EPSILON;
    const double ext0 = __dsub_rn(r.y, r.x);
    const double ext1 = __dsub_rn(r.w, r.z);
    const double ext = __dmul_rn(ext0 < ext1 ? ext1 : ext0, 1.0 + 2.0 * eps);
    Frame f;
    f.xmin = __dsub_rn(r.x, __dmul_rn(eps, ext));
    f.ymin = __dsub_rn(r.z, __dmul_rn(eps, ext));
    f.ext = ext;
    f.scale = __dmul_rn(__ddiv_rn(1.0, ext), (double)(1 << LMAX));
    return f;
}

// Per-CTA min/max, then the last CTA to finish reduces the partials and derives the frame.
// Initial extrema follow upward-common.ispc:132 (min 1e13, max 0) and sort-sources.cpp:48.
__global__ __launch_bounds__(BBOX_THREADS) void k_bbox(const double *__restrict__ x,
                                                       const double *__restrict__ y, int n,
                                                       double4 *partials, unsigned *done,
                                                       Frame *frame) {
    pdl_begin();
    double xmi = 1e13, xma = 0, ymi = 1e13, yma = 0;
    auto take = [&](double xv, double yv) {
        xmi = fmin(xmi, xv);
        xma = fmax(xma, xv);
        ymi = fmin(ymi, yv);
        yma = fmax(yma, yv);
    };
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
        // 16-byte loads, two pairs per thread in flight
        const double2 *x2 = reinterpret_cast<const double2 *>(x);
        const double2 *y2 = reinterpret_cast<const double2 *>(y);
        const int n2 = n / 2;
        int i = gid;
        for (; i + stride < n2; i += 2 * stride) {
            const double2 a = x2[i], b = y2[i], c = x2[i + stride], e = y2[i + stride];
            take(a.x, b.x);
            take(a.y, b.y);
            take(c.x, e.x);
            take(c.y, e.y);
        }
        if (i < n2) {
            const double2 a = x2[i], b = y2[i];
            take(a.x, b.x);
            take(a.y, b.y);
        }
        if ((n & 1) && gid == 0) take(x[n - 1], y[n - 1]);
    } else {
        for (int i = gid; i < n; i += stride) take(x[i], y[i]);
    }
    warp_minmax(xmi, xma, ymi, yma);
    __shared__ double4 s[BBOX_THREADS / 32];
    __shared__ bool last;
    const int w = threadIdx.x >> 5;
    if (lane_id() == 0) s[w] = make_double4(xmi, xma, ymi, yma);
    __syncthreads();
    if (threadIdx.x == 0) {
        double4 r = s[0];
        for (int i = 1; i < BBOX_THREADS / 32; ++i) {
            r.x = fmin(r.x, s[i].x); r.y = fmax(r.y, s[i].y);
            r.z = fmin(r.z, s[i].z); r.w = fmax(r.w, s[i].w);
        }
        partials[blockIdx.x] = r;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    xmi = 1e13; xma = 0; ymi = 1e13; yma = 0;
    for (int i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
        const double2 ra = __ldcg(reinterpret_cast<const double2 *>(&partials[i]));
        const double2 rb = __ldcg(reinterpret_cast<const double2 *>(&partials[i]) + 1);
        xmi = fmin(xmi, ra.x); xma = fmax(xma, ra.y);
        ymi = fmin(ymi, rb.x); yma = fmax(yma, rb.y);
    }
    warp_minmax(xmi, xma, ymi, yma);
    __syncthreads();
    if (lane_id() == 0) s[w] = make_double4(xmi, xma, ymi, yma);
    __syncthreads();
    if (threadIdx.x == 0) {
        double4 r = s[0];
        for (int i = 1; i < BBOX_THREADS / 32; ++i) {
            r.x = fmin(r.x, s[i].x); r.y = fmax(r.y, s[i].y);
            r.z = fmin(r.z, s[i].z); r.w = fmax(r.w, s[i].w);
        }
        *frame = frame_of(r);
        *done = 0;
    }
}

// ---------------------------------------------------------------------------- keys
// sort-sources.cpp:114-137: x = floor((x - xmin) * scale), bits interleaved, x on even bits.
__device__ __forceinline__ int quantize(double v, double vmin, double scale) {
    return (int)floor(__dmul_rn(__dsub_rn(v, vmin), scale));
}

// Target keys in the source frame, clamped to the quantisation range (targets may lie outside
// the sources' square).  Used only to group nearby targets; it does not affect results.
__device__ __forceinline__ int target_key(double x, double y, const Frame &f) {
    const double hi = (double)((1 << LMAX) - 1);
    double qx = floor((x - f.xmin) * f.scale);
    double qy = floor((y - f.ymin) * f.scale);
    qx = fmin(fmax(qx, 0.0), hi);
    qy = fmin(fmax(qy, 0.0), hi);
    if (qx != qx) qx = 0;
    if (qy != qy) qy = 0;
    return spread_bits((int)qx) | (spread_bits((int)qy) << 1);
}

// A target may be NEAR_REACH or more away from a source in x or in y (every source is in the frame).
__device__ __forceinline__ bool target_wide(double x, double y, const Frame &f) {
    return x <= f.xmin + f.ext - NEAR_REACH || x >= f.xmin + NEAR_REACH ||
           y <= f.ymin + f.ext - NEAR_REACH || y >= f.ymin + NEAR_REACH;
}

__global__ void k_target_keys(const double *__restrict__ x, const double *__restrict__ y, int n,
                              const Frame *__restrict__ frame, int *__restrict__ keys, int *wide) {
    pdl_begin();
    const Frame f = *frame;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double xi = x[i], yi = y[i];
        keys[i] = target_key(xi, yi, f);
        if (target_wide(xi, yi, f)) atomicOr(wide, 1);
    }
}

// ---------------------------------------------------------------------------- radix sort
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_RADIX = 256;
constexpr unsigned RS_FLAG_AGG = 1u << 30;
constexpr unsigned RS_FLAG_INC = 2u << 30;
constexpr unsigned RS_VALMASK = (1u << 30) - 1;
constexpr int RS_SPIN_LIMIT = DEFAULT_SPIN_LIMIT;
constexpr int RS_MAX_PASSES = 4;

// Histograms of every 8-bit digit of the keys, in one read.
__global__ __launch_bounds__(256) void k_hist(const int *__restrict__ keys, int n, int npasses,
                                              int *__restrict__ hist) {
    pdl_begin();
    __shared__ int s[RS_MAX_PASSES][RS_RADIX];
    for (int i = threadIdx.x; i < RS_MAX_PASSES * RS_RADIX; i += blockDim.x) (&s[0][0])[i] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned k = (unsigned)keys[i];
        for (int p = 0; p < npasses; ++p) atomicAdd(&s[p][(k >> (8 * p)) & 0xFF], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npasses * RS_RADIX; i += blockDim.x) {
        const int c = (&s[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

__global__ __launch_bounds__(RS_RADIX) void k_hist_scan(const int *__restrict__ hist,
                                                        int *__restrict__ offsets) {
    pdl_begin();
    const int p = blockIdx.x;
    const int v = hist[p * RS_RADIX + threadIdx.x];
    offsets[p * RS_RADIX + threadIdx.x] = block_exclusive_scan(v, nullptr);
}

__device__ __forceinline__ unsigned ld_volatile(const unsigned *p) {
    return *(const volatile unsigned *)p;
}

// The lanes of `vmask` whose 8-bit digit equals this lane's: one ballot per digit bit
// (eight cheap votes instead of one match.any, which has a much lower issue rate).
__device__ __forceinline__ unsigned digit_peers(unsigned vmask, int d) {
    unsigned peers = vmask;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1;
        const unsigned bal = __ballot_sync(FULL_MASK, bit);
        peers &= bit ? bal : ~bal;
    }
    return peers;
}

// Exclusive prefix of digit d over the tiles before `tile` (decoupled look-back): walk back
// over the predecessors' statuses, adding aggregates, until the first inclusive prefix.  The
// statuses of LB_WINDOW predecessors are read at once (independent loads, each coalesced over
// the CTA's digit threads), which cuts the walk of ~17 dependent L2 round trips measured on
// 16M keys to ~6.  A predecessor that has published nothing yet is read again from there; the
// number of reads without progress is bounded by `spin_limit` (DEVERR_SPIN_LIMIT).
constexpr int LB_WINDOW = 4;

__device__ __forceinline__ int lookback(const unsigned *status, int tile, int d, unsigned *err,
                                        int spin_limit = RS_SPIN_LIMIT) {
    int excl = 0;
    int spins = 0;
    int j = tile - 1;
    while (j >= 0) {
        unsigned s[LB_WINDOW];
#pragma unroll
        for (int q = 0; q < LB_WINDOW; ++q)
            s[q] = j - q >= 0 ? ld_volatile(status + (size_t)(j - q) * RS_RADIX + d) : RS_FLAG_INC;
        int used = 0;
        bool stop = false;
#pragma unroll
        for (int q = 0; q < LB_WINDOW; ++q) {
            if (stop) continue;
            const unsigned flag = s[q] & ~RS_VALMASK;
            if (flag == 0) {
                stop = true;   // not published yet: read again from here
                continue;
            }
            excl += (int)(s[q] & RS_VALMASK);
            ++used;
            if (flag == RS_FLAG_INC) return excl;
        }
        j -= used;
        if (used == 0 && ++spins > spin_limit) {
            atomicOr(err, DEVERR_SPIN_LIMIT);
            break;
        }
    }
    return excl;
}

__global__ __launch_bounds__(RS_THREADS) void k_onesweep(
    const int *__restrict__ keys_in, const int *__restrict__ vals_in, int *__restrict__ keys_out,
    int *__restrict__ vals_out, int n, int shift, const int *__restrict__ digit_offsets,
    unsigned *status, int *tile_counter, unsigned *err) {
    pdl_begin();
    __shared__ int s_keys[RS_TILE];
    __shared__ int s_vals[RS_TILE];
    __shared__ int s_whist[RS_WARPS][RS_RADIX];
    __shared__ int s_tile_start[RS_RADIX];
    __shared__ int s_global[RS_RADIX];
    __shared__ int s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1);
    for (int i = tid; i < RS_WARPS * RS_RADIX; i += RS_THREADS) (&s_whist[0][0])[i] = 0;
    __syncthreads();
    const int tile = s_tile;
    const int tile_base = tile * RS_TILE;
    const int warp_base = tile_base + warp * (RS_ITEMS * 32);

    int key[RS_ITEMS], val[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        const int idx = warp_base + k * 32 + lane;
        const bool valid = idx < n;
        key[k] = valid ? keys_in[idx] : 0;
        val[k] = valid ? (vals_in ? vals_in[idx] : idx) : 0;
    }

    // Stable rank within the warp: items are visited in their original order (k, lane).
    const unsigned lt = lanemask_lt();
    int *hist = s_whist[warp];
#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        const int idx = warp_base + k * 32 + lane;
        const bool valid = idx < n;
        const unsigned vmask = __ballot_sync(FULL_MASK, valid);
        const int d = (key[k] >> shift) & 0xFF;
        unsigned peers = digit_peers(vmask, d);
        if (!valid) peers = 0;
        const int old = valid ? hist[d] : 0;
        __syncwarp();
        if (valid && (peers & lt) == 0) hist[d] = old + __popc(peers);
        __syncwarp();
        rank[k] = old + __popc(peers & lt);
    }
    __syncthreads();

    // Thread `tid` owns digit `tid`: exclusive prefix over warps and the tile's count.
    const int d = tid;
    int total = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
        const int c = s_whist[w][d];
        s_whist[w][d] = total;
        total += c;
    }

    // Decoupled look-back for this digit.
    unsigned *mine = status + (size_t)tile * RS_RADIX + d;
    int excl = 0;
    if (tile == 0) {
        atomicExch(mine, RS_FLAG_INC | (unsigned)total);
    } else {
        atomicExch(mine, RS_FLAG_AGG | (unsigned)total);
        excl = lookback(status, tile, d, err);
        atomicExch(mine, RS_FLAG_INC | (unsigned)(excl + total));
    }

    const int start = block_exclusive_scan(total, nullptr);
    s_tile_start[d] = start;
    s_global[d] = digit_offsets[d] + excl - start;
    __syncthreads();

#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        const int idx = warp_base + k * 32 + lane;
        if (idx < n) {
            const int dk = (key[k] >> shift) & 0xFF;
            const int pos = s_tile_start[dk] + s_whist[warp][dk] + rank[k];
            if ((unsigned)pos >= (unsigned)RS_TILE) {
                atomicOr(err, DEVERR_BOUNDS);
                continue;
            }
            s_keys[pos] = key[k];
            s_vals[pos] = val[k];
        }
    }
    __syncthreads();

    const int tile_n = min(RS_TILE, n - tile_base);
    for (int j = tid; j < tile_n; j += RS_THREADS) {
        const int kk = s_keys[j];
        const int g = s_global[(kk >> shift) & 0xFF] + j;
        if ((unsigned)g >= (unsigned)n) {
            atomicOr(err, DEVERR_BOUNDS);
            continue;
        }
        keys_out[g] = kk;
        vals_out[g] = s_vals[j];
    }
}

// ---------------------------------------------------------------------------- source sort
// The sources are sorted as 8-byte items key << 32 | payload by four onesweep passes (8-bit
// digits of the key half, 16 B of traffic per item and pass).  Ties keep input order, so the
// result is the (key, index) lexicographic order.
// k_keys_pack: the items (key << 32 | index) in input order and the histograms of the four
// digits (the late-values path and the allocation-free sort).
__global__ __launch_bounds__(256) void k_keys_pack(const double *__restrict__ x,
                                                   const double *__restrict__ y, int n,
                                                   const Frame *__restrict__ frame,
                                                   unsigned long long *__restrict__ items,
                                                   int npasses, int *__restrict__ hist) {
    pdl_begin();
    __shared__ int s[RS_MAX_PASSES][RS_RADIX];
    for (int i = threadIdx.x; i < RS_MAX_PASSES * RS_RADIX; i += blockDim.x) (&s[0][0])[i] = 0;
    __syncthreads();
    const Frame f = *frame;
    auto item_of = [&](double xv, double yv, int i) {
        const int k = spread_bits(quantize(xv, f.xmin, f.scale)) |
                      (spread_bits(quantize(yv, f.ymin, f.scale)) << 1);
        for (int p = 0; p < npasses; ++p) atomicAdd(&s[p][((unsigned)k >> (8 * p)) & 0xFF], 1);
        return ((unsigned long long)(unsigned)k << 32) | (unsigned)i;
    };
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
          reinterpret_cast<uintptr_t>(items)) & 15) == 0) {
        // 16-byte loads and stores: two sources per thread and step
        const double2 *x2 = reinterpret_cast<const double2 *>(x);
        const double2 *y2 = reinterpret_cast<const double2 *>(y);
        ulonglong2 *it2 = reinterpret_cast<ulonglong2 *>(items);
        for (int i = gid; i < n / 2; i += stride) {
            const double2 a = x2[i], b = y2[i];
            it2[i] = make_ulonglong2(item_of(a.x, b.x, 2 * i), item_of(a.y, b.y, 2 * i + 1));
        }
        if ((n & 1) && gid == 0) {
            const int i = n - 1;
            items[i] = item_of(x[i], y[i], i);
        }
    } else {
        for (int i = gid; i < n; i += stride) items[i] = item_of(x[i], y[i], i);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npasses * RS_RADIX; i += blockDim.x) {
        const int c = (&s[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// Resident values (the device entry points): the records are written by the first radix pass
// itself, grouped by the top 8 bits of the key (256 buckets, each a square of 1/16 of the
// frame's side), so that the final gather reads a window of the sorted order from a compact
// range of records, L2-resident, instead of from anywhere in HBM:
//   * k_key_hist reads x and y once and writes the histograms of the four radix digits and of
//     the top 8 key bits (the buckets);
//   * k_onesweep_items<.., true> (the first pass) reads x, y, v, forms the keys, claims each
//     source a record slot in its bucket (tile counts in shared memory, one global atomic per
//     tile and bucket) and writes the record (x, y, v, index); its items carry the record's
//     position, key << 32 | slot;
//   * three more passes over the items; the gather reads each record from its bucket.
// Slots within a bucket depend on tile timing, but they are only payload: the passes order by
// the key half alone and keep input order for equal keys, so the sorted keys, permutation and
// sources do not depend on them.
constexpr int NB_BUCKETS = 256;
constexpr int BUCKET_SHIFT = 2 * LMAX - 8;   // the top 8 of the 30 key bits

__device__ __forceinline__ int morton_key(double xv, double yv, const Frame &f) {
    return spread_bits(quantize(xv, f.xmin, f.scale)) |
           (spread_bits(quantize(yv, f.ymin, f.scale)) << 1);
}

__global__ __launch_bounds__(256) void k_key_hist(const double *__restrict__ x,
                                                  const double *__restrict__ y, int n,
                                                  const Frame *__restrict__ frame, int npasses,
                                                  int *__restrict__ hist) {
    pdl_begin();
    __shared__ int s[RS_MAX_PASSES + 1][RS_RADIX];
    for (int i = threadIdx.x; i < (RS_MAX_PASSES + 1) * RS_RADIX; i += blockDim.x)
        (&s[0][0])[i] = 0;
    __syncthreads();
    const Frame f = *frame;
    auto count = [&](double xv, double yv) {
        const unsigned k = (unsigned)morton_key(xv, yv, f);
        for (int p = 0; p < npasses; ++p) atomicAdd(&s[p][(k >> (8 * p)) & 0xFF], 1);
        atomicAdd(&s[RS_MAX_PASSES][k >> BUCKET_SHIFT], 1);
    };
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0) {
        const double2 *x2 = reinterpret_cast<const double2 *>(x);
        const double2 *y2 = reinterpret_cast<const double2 *>(y);
        for (int i = gid; i < n / 2; i += stride) {
            const double2 a = x2[i], b = y2[i];
            count(a.x, b.x);
            count(a.y, b.y);
        }
        if ((n & 1) && gid == 0) count(x[n - 1], y[n - 1]);
    } else {
        for (int i = gid; i < n; i += stride) count(x[i], y[i]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (RS_MAX_PASSES + 1) * RS_RADIX; i += blockDim.x) {
        const int c = (&s[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// One 32-byte store of four doubles (st.global.v4.f64; `p` 32-byte aligned).
__device__ __forceinline__ void st_global_v4(double2 *p, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c),
                 "d"(d)
                 : "memory");
}

// One 32-byte load of four doubles (`p` 32-byte aligned).
__device__ __forceinline__ void ld_global_v4(const double2 *p, double2 &a, double2 &b) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
                 : "l"(p));
}

// The first pass's inputs: the resident sources, the frame, and where records go.
struct FirstPass {
    const double *x, *y, *v;
    const Frame *frame;
    double2 *rec;               // 2 per source: (x, y), (v, index as bits)
    const int *bucket_off;      // exclusive scan of the bucket histogram
    int *bucket_fill;           // slots claimed per bucket so far (zeroed per sort)
};

// One onesweep pass over 8-byte items, digit (item >> shift) & 0xFF: tiles of 256 threads x ITEMS;
// the tile's digit counts, then the global digit offsets by decoupled look-back, then the stable
// rank within each warp from digit ballots; items are placed in sorted order in shared memory and
// written out in runs of equal digits.  ITEMS is 12 (four CTAs per SM), or 8 where that is few tiles
// per SM and a pass lasts as long as one tile's phases (sort_tile): potential of 64K sources 359 ->
// 352 us, force 64K 234 -> 226, 256K 392 -> 374, 1M 1014 -> 1007, potential 700,001 1437 -> 1417;
// at 16M it is the slower one (sort 1057 -> 1128).  Mixed solves of a sheet on 256 blocks: 512K 357 ->
// 349, 1.5M 531 -> 528, 2M and 4M the same, 8M 1980 -> 2001 us.
// `stall_tile` (a test setting, -1 otherwise) names a tile that publishes into `sink` instead
// of its status words, so that the tiles after it wait until `spin_limit` and report
// DEVERR_SPIN_LIMIT.
constexpr int PS_THREADS = 256;
constexpr int PS_WARPS = PS_THREADS / 32;
constexpr int PS_TILE = PS_THREADS * 12;         // a tile of the general form
constexpr int PS_SMALL_TILE = PS_THREADS * 8;
constexpr int PS_SMALL_MAX = 3 << 19;             // sources up to which tiles are the small ones
inline int sort_tile(int n) { return n <= PS_SMALL_MAX ? PS_SMALL_TILE : PS_TILE; }
inline int sort_tiles(int n) { return (n + sort_tile(n) - 1) / sort_tile(n); }

// FIRST: the first pass of resident values (the tile's items formed from x, y, v, records
// written to their buckets, see FirstPass); otherwise the items are read from `in`.  STALL:
// the instance that honours stall_tile (the test setting; the others ignore it).
template <int ITEMS, bool FIRST, bool STALL = false>
__global__ __launch_bounds__(PS_THREADS, FIRST ? 3 : 4) void k_onesweep_items(
    const unsigned long long *__restrict__ in, unsigned long long *__restrict__ out, int n,
    int shift, const int *__restrict__ digit_offsets, unsigned *status, int *tile_counter,
    unsigned *err, int spin_limit, int stall_tile, unsigned *sink, FirstPass fp) {
    constexpr int TILE = PS_THREADS * ITEMS;
    pdl_begin();
    __shared__ unsigned long long s_items[TILE];
    __shared__ int s_whist[PS_WARPS][RS_RADIX];
    __shared__ int s_count[RS_RADIX];
    __shared__ int s_tile_start[RS_RADIX];
    __shared__ int s_global[RS_RADIX];
    __shared__ int s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the pass's digit is a whole byte of the key half: one byte permutation
    const unsigned digit_sel = 0x4440u | (unsigned)(shift - 32) >> 3;
    auto digit_of = [&](unsigned long long it) {
        return (int)__byte_perm((unsigned)(it >> 32), 0u, digit_sel);
    };
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1);
    for (int i = tid; i < PS_WARPS * RS_RADIX; i += PS_THREADS) (&s_whist[0][0])[i] = 0;
    s_count[tid] = 0;
    if (FIRST) s_global[tid] = 0;   // the tile's count per bucket, first
    __syncthreads();
    const int tile = s_tile;
    const int tile_base = tile * TILE;
    const int tile_n = min(TILE, n - tile_base);
    const int warp_base = tile_base + warp * (ITEMS * 32);

    unsigned long long item[ITEMS];
    int rank[ITEMS];
    constexpr int FB = 4;   // the first pass's loads in flight
    static_assert(ITEMS % FB == 0, "whole batches");
    if constexpr (FIRST) {
        // keys, digit counts and each source's slot among the tile's sources of its bucket; the
        // loads are issued in batches of FB before the shared atomics that consume them
        const Frame f = *fp.frame;
#pragma unroll
        for (int k0 = 0; k0 < ITEMS; k0 += FB) {
            double xv[FB], yv[FB];
#pragma unroll
            for (int k = 0; k < FB; ++k) {
                const int idx = warp_base + (k0 + k) * 32 + lane;
                xv[k] = idx < n ? __ldg(fp.x + idx) : 0.0;
                yv[k] = idx < n ? __ldg(fp.y + idx) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < FB; ++k) {
                const int idx = warp_base + (k0 + k) * 32 + lane;
                int key = 0, slot = 0;
                if (idx < n) {
                    key = morton_key(xv[k], yv[k], f);
                    slot = atomicAdd(&s_global[(unsigned)key >> BUCKET_SHIFT], 1);
                    atomicAdd(&s_count[__byte_perm((unsigned)key, 0u, digit_sel)], 1);
                }
                item[k0 + k] = ((unsigned long long)(unsigned)key << 32) | (unsigned)slot;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int idx = warp_base + k * 32 + lane;
            item[k] = idx < n ? in[idx] : 0ull;
        }
#pragma unroll
        for (int k = 0; k < ITEMS; ++k)
            if (warp_base + k * 32 + lane < n)
                atomicAdd(&s_count[digit_of(item[k])], 1);
    }
    // Early counts: the tile's digit totals first (shared atomics), so that its aggregate is
    // published and the look-back done before the ranking (and the first pass's records), not
    // after it: the tiles behind wait for it.  (The first pass with its look-back after the
    // records and the bucket claims: 341 us on the 16M sheet, so ~285.)
    const int d = tid;   // one digit per thread
    __syncthreads();
    const int total = s_count[d];
    int bucket_base = 0;
    if constexpr (FIRST) {
        // the tile's slots in each bucket, one global claim per bucket (used after the look-back)
        const int c = s_global[tid];
        if (c) bucket_base = fp.bucket_off[tid] + atomicAdd(&fp.bucket_fill[tid], c);
    }
    // tile == stall_tile (a test setting): this tile publishes into `sink`, which no look-back
    // reads, so the tiles after it wait until spin_limit
    unsigned *mine = (STALL && tile == stall_tile ? sink : status + (size_t)tile * RS_RADIX) + d;
    int excl = 0;
    if (tile == 0) {
        atomicExch(mine, RS_FLAG_INC | (unsigned)total);
    } else {
        atomicExch(mine, RS_FLAG_AGG | (unsigned)total);
        excl = lookback(status, tile, d, err, spin_limit);
        atomicExch(mine, RS_FLAG_INC | (unsigned)(excl + total));
    }
    if constexpr (FIRST) {
        s_tile_start[tid] = bucket_base;
        __syncthreads();
        // each record with one 32-byte store (one whole DRAM sector), batches of FB loads first
#pragma unroll
        for (int k0 = 0; k0 < ITEMS; k0 += FB) {
            double xv[FB], yv[FB], vv[FB];
#pragma unroll
            for (int k = 0; k < FB; ++k) {
                const int idx = warp_base + (k0 + k) * 32 + lane;
                xv[k] = idx < n ? __ldg(fp.x + idx) : 0.0;
                yv[k] = idx < n ? __ldg(fp.y + idx) : 0.0;
                vv[k] = idx < n ? __ldg(fp.v + idx) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < FB; ++k) {
                const int idx = warp_base + (k0 + k) * 32 + lane;
                if (idx >= n) continue;
                const unsigned key = (unsigned)(item[k0 + k] >> 32);
                const int pos = s_tile_start[key >> BUCKET_SHIFT] + (int)(unsigned)item[k0 + k];
                if ((unsigned)pos >= (unsigned)n) {
                    atomicOr(err, DEVERR_BOUNDS);
                    continue;
                }
                st_global_v4(fp.rec + 2 * (size_t)pos, xv[k], yv[k], vv[k],
                             __longlong_as_double((long long)idx));
                item[k0 + k] = ((unsigned long long)key << 32) | (unsigned)pos;
            }
        }
    }

    const unsigned lt = lanemask_lt();
    int *hist = s_whist[warp];
    auto ranks = [&](auto full) {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const bool valid = decltype(full)::value || warp_base + k * 32 + lane < n;
            const unsigned vmask = decltype(full)::value ? FULL_MASK : __ballot_sync(FULL_MASK, valid);
            const int dk = digit_of(item[k]);
            unsigned peers = digit_peers(vmask, dk);
            if (!valid) peers = 0;
            const int old = valid ? hist[dk] : 0;
            __syncwarp();
            if (valid && (peers & lt) == 0) hist[dk] = old + __popc(peers);
            __syncwarp();
            rank[k] = old + __popc(peers & lt);
        }
    };
    const bool full_tile = tile_n == TILE;
    if (full_tile)
        ranks(std::true_type{});
    else
        ranks(std::false_type{});
    __syncthreads();
    const int start = block_exclusive_scan(total, nullptr);
    int run = start;
#pragma unroll
    for (int w = 0; w < PS_WARPS; ++w) {
        const int c = s_whist[w][d];
        s_whist[w][d] = run;
        run += c;
    }
    s_global[d] = digit_offsets[d] + excl - start;
    __syncthreads();

#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (full_tile || warp_base + k * 32 + lane < n) {
            const int dk = digit_of(item[k]);
            const int p = s_whist[warp][dk] + rank[k];
            if ((unsigned)p >= (unsigned)tile_n) {
                atomicOr(err, DEVERR_BOUNDS);
                continue;
            }
            s_items[p] = item[k];
        }
    }
    __syncthreads();

    auto write = [&](int j) {
        const unsigned long long it = s_items[j];
        const int g = s_global[digit_of(it)] + j;
        if ((unsigned)g >= (unsigned)n)
            atomicOr(err, DEVERR_BOUNDS);
        else
            out[g] = it;
    };
    if (full_tile) {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) write(tid + k * PS_THREADS);
    } else {
        for (int j = tid; j < tile_n; j += PS_THREADS) write(j);
    }
}

// Sorted keys, permutation, x, y and v from the sorted items and the input-order records.
constexpr int GS_THREADS = 256;
constexpr int GS_ITEMS = 8;

// The sorted sources from the sorted items (key << 32 | record slot) and the bucketed records
// (x, y, v, index): the sorted keys, the permutation (the records' indices) and x, y, v.
__global__ __launch_bounds__(GS_THREADS) void k_gather_sources(
    const unsigned long long *__restrict__ items, const double2 *__restrict__ rec, int n,
    int *__restrict__ keys, int *__restrict__ perm, double *__restrict__ xs,
    double *__restrict__ ys, double *__restrict__ vs, unsigned *err) {
    pdl_begin();
    const int stride = gridDim.x * GS_THREADS * GS_ITEMS;
    for (int base = blockIdx.x * GS_THREADS * GS_ITEMS + threadIdx.x; base < n; base += stride) {
        unsigned long long it[GS_ITEMS];
        double2 a[GS_ITEMS], b[GS_ITEMS];
#pragma unroll
        for (int k = 0; k < GS_ITEMS; ++k) {
            const int i = base + k * GS_THREADS;
            it[k] = i < n ? __ldcs(items + i) : 0ull;
        }
#pragma unroll
        for (int k = 0; k < GS_ITEMS; ++k) {
            const int i = base + k * GS_THREADS;
            const unsigned id = (unsigned)it[k];
            if (i < n && id < (unsigned)n) ld_global_v4(rec + 2 * (size_t)id, a[k], b[k]);
        }
#pragma unroll
        for (int k = 0; k < GS_ITEMS; ++k) {
            const int i = base + k * GS_THREADS;
            if (i >= n) continue;
            if ((unsigned)it[k] >= (unsigned)n) {
                atomicOr(err, DEVERR_BOUNDS);
                continue;
            }
            __stcs(keys + i, (int)(it[k] >> 32));
            __stcs(perm + i, (int)__double_as_longlong(b[k].y));
            __stcs(xs + i, a[k].x);
            __stcs(ys + i, a[k].y);
            __stcs(vs + i, b[k].x);
        }
    }
}

// Late values, before they arrive: x and y in sorted order, gathered by the permutation from
// the input arrays (off the critical path, while v is still being copied in).
__global__ __launch_bounds__(256) void k_gather_xy(const int *__restrict__ perm,
                                                   const double *__restrict__ x,
                                                   const double *__restrict__ y, int n,
                                                   double *__restrict__ xs,
                                                   double *__restrict__ ys, unsigned *err) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned j = (unsigned)perm[i];
        if (j >= (unsigned)n) {
            atomicOr(err, DEVERR_BOUNDS);
            continue;
        }
        xs[i] = __ldg(x + j);
        ys[i] = __ldg(y + j);
    }
}

// Late values, once they are in: v in sorted order (the one gather left after their arrival).
__global__ __launch_bounds__(256) void k_gather_v(const int *__restrict__ perm,
                                                  const double *__restrict__ v, int n,
                                                  double *__restrict__ vs) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned j = (unsigned)perm[i];
        if (j < (unsigned)n) vs[i] = __ldg(v + j);
    }
}

// Sorted keys and permutation from the sorted items.
__global__ __launch_bounds__(256) void k_items_split(const unsigned long long *__restrict__ items,
                                                     int n, int *__restrict__ keys,
                                                     int *__restrict__ perm) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long it = items[i];
        keys[i] = (int)(it >> 32);
        perm[i] = (int)(unsigned)it;
    }
}

// The allocation-free sort's gather: the sorted items sit in xs (as 8-byte words); each thread
// reads item i and then overwrites xs[i] with the source's x, so no other buffer is needed.
__global__ __launch_bounds__(256) void k_gather_items_inplace(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ v, int n,
    int *__restrict__ keys, int *__restrict__ perm, double *xs, double *__restrict__ ys,
    double *__restrict__ vs, unsigned *err) {
    unsigned long long *items = reinterpret_cast<unsigned long long *>(xs);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long it = items[i];
        const unsigned j = (unsigned)it;
        if (j >= (unsigned)n) {
            atomicOr(err, DEVERR_BOUNDS);
            continue;
        }
        keys[i] = (int)(it >> 32);
        perm[i] = (int)j;
        xs[i] = x[j];
        ys[i] = y[j];
        vs[i] = v[j];
    }
}

// ---------------------------------------------------------------------------- small sorts
// Up to SMALL_SORT sources (or targets) are sorted by one block, in one launch: bounding square,
// keys, an LSD radix sort of the items (key << 32 | index) held in shared memory, and the
// gather.  It is bound by the latency of its phases, about 6 us for 4096 items and 15 us for
// 16,384, where the eight launches of the general sort take 65 us whatever the size; past 16K
// items (128 KB of shared memory) one SM would be the slower one.  Same keys, order and values:
// ties keep input order in both.
constexpr int SMALL_THREADS = 1024;
constexpr int SMALL_WARPS = SMALL_THREADS / 32;
constexpr int SMALL_SORT = 16 * SMALL_THREADS;
constexpr int SMALL_ROW = RS_RADIX + 1;   // padded: a digit's 32 warp counts in distinct banks

template <int ITEMS>
constexpr size_t small_smem() {
    return sizeof(unsigned long long) * SMALL_THREADS * ITEMS + sizeof(int) * SMALL_WARPS * SMALL_ROW;
}

// Sorts the block's items by their upper 32 bits; warp w holds items [w, w + 1) * 32 ITEMS of the
// input order in `item`; the sorted items are left in s_items.
template <int ITEMS>
__device__ __forceinline__ void block_sort_items(unsigned long long (&item)[ITEMS],
                                                 unsigned long long *s_items, int *s_hist) {
    __shared__ int s_total[RS_RADIX];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const int first = warp * 32 * ITEMS + lane;
    const unsigned lt = lanemask_lt();
    int *hist = s_hist + warp * SMALL_ROW;
    for (int shift = 32; shift < 64; shift += 8) {
        if (shift > 32)
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) item[k] = s_items[first + 32 * k];
        for (int i = lane; i < RS_RADIX; i += 32) hist[i] = 0;
        __syncwarp();
        int rank[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int d = (int)(item[k] >> shift) & 0xFF;
            const unsigned peers = digit_peers(FULL_MASK, d);
            const int old = hist[d];
            __syncwarp();
            if ((peers & lt) == 0) hist[d] = old + __popc(peers);
            __syncwarp();
            rank[k] = old + __popc(peers & lt);
        }
        __syncthreads();   // (also: every item has been read)
        // each warp scans the warp counts of 8 digits, lane = warp
#pragma unroll
        for (int q = 0; q < RS_RADIX / SMALL_WARPS; ++q) {
            const int d = warp * (RS_RADIX / SMALL_WARPS) + q;
            const int v = s_hist[lane * SMALL_ROW + d];
            int inc = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL_MASK, inc, o);
                if (lane >= o) inc += t;
            }
            s_hist[lane * SMALL_ROW + d] = inc - v;
            if (lane == 31) s_total[d] = inc;
        }
        __syncthreads();
        const int tot = threadIdx.x < RS_RADIX ? s_total[threadIdx.x] : 0;
        const int start = block_exclusive_scan(tot, nullptr);
        if (threadIdx.x < RS_RADIX) s_total[threadIdx.x] = start;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int d = (int)(item[k] >> shift) & 0xFF;
            s_items[s_total[d] + hist[d] + rank[k]] = item[k];
        }
        __syncthreads();
    }
}

// Block 0, sources: frame, sorted keys, permutation, x and y, and v where it is there (null: late
// values).  Block 1 (when launched), targets: the permutation alone, in the frame that it forms from
// the sources like block 0, so that the two sorts of a small solve run side by side.
template <int ITEMS>
__global__ __launch_bounds__(SMALL_THREADS) void k_sort_small(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ v, int n,
    Frame *frame, int *__restrict__ keys, int *__restrict__ perm, double *__restrict__ xs,
    double *__restrict__ ys, double *__restrict__ vs, const double *__restrict__ xt,
    const double *__restrict__ yt, int nt, int *__restrict__ tperm, int *wide) {
    extern __shared__ __align__(16) unsigned long long small_dyn[];
    unsigned long long *s_items = small_dyn;
    int *s_hist = reinterpret_cast<int *>(s_items + SMALL_THREADS * ITEMS);
    __shared__ double4 s_ext[SMALL_WARPS];
    __shared__ Frame s_frame;
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    // extrema as k_bbox
    double xmi = 1e13, xma = 0, ymi = 1e13, yma = 0;
    for (int i = threadIdx.x; i < n; i += SMALL_THREADS) {
        const double xv = x[i], yv = y[i];
        xmi = fmin(xmi, xv);
        xma = fmax(xma, xv);
        ymi = fmin(ymi, yv);
        yma = fmax(yma, yv);
    }
    warp_minmax(xmi, xma, ymi, yma);
    if (lane == 0) s_ext[warp] = make_double4(xmi, xma, ymi, yma);
    __syncthreads();
    if (warp == 0) {
        const double4 r = s_ext[lane];
        xmi = r.x; xma = r.y; ymi = r.z; yma = r.w;
        warp_minmax(xmi, xma, ymi, yma);
        if (lane == 0) {
            s_frame = frame_of(make_double4(xmi, xma, ymi, yma));
            if (blockIdx.x == 0) *frame = s_frame;
        }
    }
    __syncthreads();
    const Frame f = s_frame;
    const bool targets = blockIdx.x == 1;
    unsigned long long item[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = warp * 32 * ITEMS + 32 * k + lane;
        // past the end: after every key, and after equal ones (they come last in input order)
        unsigned key = 0xffffffffu;
        if (targets) {
            if (i < nt) {
                const double xi = xt[i], yi = yt[i];
                key = (unsigned)target_key(xi, yi, f);
                if (target_wide(xi, yi, f)) atomicOr(wide, 1);
            }
        } else if (i < n) {
            key = (unsigned)morton_key(x[i], y[i], f);
        }
        item[k] = ((unsigned long long)key << 32) | (unsigned)i;
    }
    block_sort_items<ITEMS>(item, s_items, s_hist);
    if (targets) {
        for (int i = threadIdx.x; i < nt; i += SMALL_THREADS) tperm[i] = (int)(unsigned)s_items[i];
        return;
    }
    for (int i = threadIdx.x; i < n; i += SMALL_THREADS) {
        const unsigned long long it = s_items[i];
        const unsigned j = (unsigned)it;
        keys[i] = (int)(it >> 32);
        perm[i] = (int)j;
        xs[i] = x[j];
        ys[i] = y[j];
        if (v) vs[i] = v[j];
    }
}

// Targets by themselves (the sources sorted before, by whichever sort): the permutation alone.
template <int ITEMS>
__global__ __launch_bounds__(SMALL_THREADS) void k_sort_small_targets(
    const double *__restrict__ x, const double *__restrict__ y, int n,
    const Frame *__restrict__ frame, int *__restrict__ perm, int *wide) {
    extern __shared__ __align__(16) unsigned long long small_dyn[];
    unsigned long long *s_items = small_dyn;
    int *s_hist = reinterpret_cast<int *>(s_items + SMALL_THREADS * ITEMS);
    pdl_begin();
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const Frame f = *frame;
    unsigned long long item[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = warp * 32 * ITEMS + 32 * k + lane;
        unsigned key = 0xffffffffu;
        if (i < n) {
            const double xi = x[i], yi = y[i];
            key = (unsigned)target_key(xi, yi, f);
            if (target_wide(xi, yi, f)) atomicOr(wide, 1);
        }
        item[k] = ((unsigned long long)key << 32) | (unsigned)i;
    }
    block_sort_items<ITEMS>(item, s_items, s_hist);
    for (int i = threadIdx.x; i < n; i += SMALL_THREADS) perm[i] = (int)(unsigned)s_items[i];
}

template <int ITEMS>
static int sort_small(Context &c, const double *x, const double *y, const double *v, int n,
                      Frame *frame, int *keys, int *perm, double *xs, double *ys, double *vs,
                      const double *xt, const double *yt, int nt, int *tperm) {
    k_sort_small<ITEMS><<<tperm ? 2 : 1, SMALL_THREADS, small_smem<ITEMS>(), c.stream>>>(
        x, y, v, n, frame, keys, perm, xs, ys, vs, xt, yt, nt, tperm,
        c.ctrl.meta + META_WIDE);
    TC_KERNEL_CHECK();
    return TC_OK;
}

template <int ITEMS>
static int sort_small_targets(Context &c, const double *x, const double *y, int n, int *perm) {
    TC_CUDA_TRY(launch_pdl(c.launch_overlap && c.single, k_sort_small_targets<ITEMS>, 1,
                           SMALL_THREADS, small_smem<ITEMS>(), c.stream, x, y, n,
                           (const Frame *)slot_ptr<Frame>(c, S_FRAME), perm,
                           c.ctrl.meta + META_WIDE));
    TC_KERNEL_CHECK();
    return TC_OK;
}

static int grid_for(int n, int threads, int per_sm = 8) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long g = ((long long)n + threads - 1) / threads;
    long long cap = (long long)sms * per_sm;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

int radix_sort_pairs(Context &c, const int *keys_in, const int *vals_in, int n, int nbits,
                     int *keys_a, int *vals_a, int *keys_b, int *vals_b, int **keys_out,
                     int **vals_out) {
    const bool ovl = c.launch_overlap;   // launch_pdl chains (tc_set_launch_overlap)
    if (n >= (1 << 30)) {
        set_error(TC_ERR_INVALID, "radix sort supports fewer than 2^30 keys (got %d)", n);
        return TC_ERR_INVALID;
    }
    const int npasses = (nbits + 7) / 8;
    const int ntiles = (n + RS_TILE - 1) / RS_TILE;
    int *hist = c.ctrl.t_hist, *counter = c.ctrl.t_tile_ctr, *offsets = c.ctrl.t_offsets;
    unsigned *status = c.ctrl.t_status;   // (cleared at the solve's start)
    // the kernels follow each other, and the keys' kernel, directly (launch_pdl)
    TC_CUDA_TRY(launch_pdl(ovl, k_hist, grid_for(n, 256, 4), 256, 0, c.stream, keys_in, n, npasses,
                           hist));
    TC_KERNEL_CHECK();
    TC_CUDA_TRY(launch_pdl(ovl, k_hist_scan, npasses, RS_RADIX, 0, c.stream, (const int *)hist,
                           offsets));
    TC_KERNEL_CHECK();
    unsigned *err = c.ctrl.err;

    const int *ki = keys_in, *vi = vals_in;
    int *ko = keys_a, *vo = vals_a;
    for (int p = 0; p < npasses; ++p) {
        TC_CUDA_TRY(launch_pdl(ovl, k_onesweep, ntiles, RS_THREADS, 0, c.stream, ki, vi, ko, vo, n,
                               8 * p, (const int *)(offsets + p * RS_RADIX),
                               status + (size_t)p * ntiles * RS_RADIX, counter + p, err));
        TC_KERNEL_CHECK();
        ki = ko;
        vi = vo;
        if (ko == keys_a) { ko = keys_b; vo = vals_b; }
        else { ko = keys_a; vo = vals_a; }
    }
    *keys_out = const_cast<int *>(ki);
    *vals_out = const_cast<int *>(vi);
    return TC_OK;
}

// ---------------------------------------------------------------------------- scan
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__global__ __launch_bounds__(SCAN_THREADS) void k_scan_reduce(const int *__restrict__ in, int n,
                                                             int *__restrict__ block_sums) {
    pdl_begin();
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i)
        if (base + i < n) s += in[base + i];
    int total;
    block_exclusive_scan(s, &total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ __launch_bounds__(SCAN_THREADS) void k_scan_blocks(int *block_sums, int nb,
                                                             int *out_total, int nparts,
                                                             volatile unsigned *host,
                                                             const int *meta) {
    pdl_begin();
    // one CTA: each thread scans a contiguous chunk of the block sums
    const int per = (nb + SCAN_THREADS - 1) / SCAN_THREADS;
    const int b0 = threadIdx.x * per;
    int s = 0;
    for (int i = 0; i < per; ++i)
        if (b0 + i < nb) s += block_sums[b0 + i];
    int total;
    int run = block_exclusive_scan(s, &total);
    for (int i = 0; i < per; ++i)
        if (b0 + i < nb) {
            const int v = block_sums[b0 + i];
            block_sums[b0 + i] = run;
            run += v;
        }
    if (threadIdx.x == 0) {
        *out_total = total;
        if (host) host[nparts - 1] = (unsigned)total;
    }
    if (host && threadIdx.x < 4) host[nparts + threadIdx.x] = (unsigned)meta[threadIdx.x];
}

__global__ __launch_bounds__(SCAN_THREADS) void k_scan_apply(const int *__restrict__ in, int n,
                                                            const int *__restrict__ block_offs,
                                                            int *__restrict__ out, int part,
                                                            volatile unsigned *host) {
    pdl_begin();
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
        v[i] = base + i < n ? in[base + i] : 0;
        s += v[i];
    }
    int run = block_exclusive_scan(s, nullptr) + block_offs[blockIdx.x];
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i)
        if (base + i < n) {
            out[base + i] = run;
            if (host && base + i > 0 && (base + i) % part == 0)
                host[(base + i) / part - 1] = (unsigned)run;
            run += v[i];
        }
}

// The whole scan in one block, a tile after another, for short inputs: a tile takes about 2 us,
// the three launches about 8.
constexpr int SCAN_SMALL = 4 * SCAN_TILE;

__global__ __launch_bounds__(SCAN_THREADS) void k_scan_small(const int *__restrict__ in, int n,
                                                            int *__restrict__ out, int part,
                                                            volatile unsigned *host,
                                                            const int *meta) {
    pdl_begin();
    int carry = 0;
    for (int t0 = 0; t0 < n; t0 += SCAN_TILE) {
        const int base = t0 + threadIdx.x * SCAN_ITEMS;
        int v[SCAN_ITEMS];
        int s = 0, total;
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i) {
            v[i] = base + i < n ? in[base + i] : 0;
            s += v[i];
        }
        int run = carry + block_exclusive_scan(s, &total);
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i)
            if (base + i < n) {
                out[base + i] = run;
                if (host && base + i > 0 && (base + i) % part == 0)
                    host[(base + i) / part - 1] = (unsigned)run;
                run += v[i];
            }
        carry += total;
    }
    if (threadIdx.x == 0) {
        out[n] = carry;
        if (host) host[n / part - 1] = (unsigned)carry;
    }
    if (host && threadIdx.x < 4) host[n / part + threadIdx.x] = (unsigned)meta[threadIdx.x];
}

int exclusive_scan(Context &c, const int *d_in, int *d_out, int n, int part, unsigned *host,
                   const int *meta) {
    const bool ovl = c.launch_overlap;   // launch_pdl chains (tc_set_launch_overlap)
    if (n > 0 && n <= SCAN_SMALL) {
        TC_CUDA_TRY(launch_pdl(ovl, k_scan_small, 1, SCAN_THREADS, 0, c.stream, d_in, n, d_out,
                               part, (volatile unsigned *)host, meta));
        TC_KERNEL_CHECK();
        return TC_OK;
    }
    const int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    int *bs;
    int rc;
    if ((rc = ensure(c, S_SCAN_BLOCKS, (size_t)nb + 1, &bs))) return rc;
    if (n == 0) {
        TC_CUDA_TRY(cudaMemsetAsync(d_out, 0, sizeof(int), c.stream));
        return TC_OK;
    }
    TC_CUDA_TRY(launch_pdl(ovl, k_scan_reduce, nb, SCAN_THREADS, 0, c.stream, d_in, n, bs));
    TC_KERNEL_CHECK();
    TC_CUDA_TRY(launch_pdl(ovl, k_scan_blocks, 1, SCAN_THREADS, 0, c.stream, bs, nb, d_out + n,
                           part > 0 ? n / part : 0, (volatile unsigned *)host, meta));
    TC_KERNEL_CHECK();
    TC_CUDA_TRY(launch_pdl(ovl, k_scan_apply, nb, SCAN_THREADS, 0, c.stream, d_in, n,
                           (const int *)bs, d_out, part, (volatile unsigned *)host));
    TC_KERNEL_CHECK();
    return TC_OK;
}

// ---------------------------------------------------------------------------- drivers
// histograms and their scans: the four radix digits, then the buckets of the records
constexpr int NHIST = RS_MAX_PASSES + 1;

int ctrl_prepare(Context &c, int n, int m) {
    const size_t words_s = (size_t)RS_MAX_PASSES * sort_tiles(n) * RS_RADIX;
    const size_t words_t = (size_t)RS_MAX_PASSES * ((m + RS_TILE - 1) / RS_TILE) * RS_RADIX;
    const size_t words_l = tree_list_tiles(n);
    unsigned *base = nullptr;
    Ctrl k = {};
    size_t total = 0, cleared = 0;
    for (int pass = 0; pass < 2; ++pass) {   // sizes, then pointers
        size_t at = 0;
        auto take = [&](auto *&p, size_t words) {
            p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at);
            at += (words + 3) & ~(size_t)3;   // 16-byte steps
        };
        take(k.err, 16);
        take(k.stats, 2 * STAT_SLOTS);
        take(k.bbox_done, 1);
        take(k.tile_ctr, RS_MAX_PASSES);
        take(k.bucket_fill, NB_BUCKETS);
        take(k.nlist, 1);
        take(k.tl_ctr, 1);
        take(k.meta, 4);
        take(k.near_ctr, 1);
        take(k.far_ctr, FORCE_CHUNKS);
        take(k.e2l_ctr, 1);
        take(k.task_fill, TASK_BINS * FORCE_CHUNKS);
        take(k.near_fill, TASK_BINS);
        take(k.t_tile_ctr, RS_MAX_PASSES);
        take(k.hist, NHIST * RS_RADIX);
        take(k.t_hist, RS_MAX_PASSES * RS_RADIX);
        take(k.tl_status, words_l);
        take(k.status, words_s);
        take(k.t_status, words_t);
        cleared = at;
        take(k.offsets, NHIST * RS_RADIX);
        take(k.t_offsets, RS_MAX_PASSES * RS_RADIX);
        take(k.sink, RS_RADIX);
        total = at;
        if (pass == 0)
            if (int rc = ensure(c, S_CTRL, total, &base)) return rc;
    }
    c.ctrl = k;
    TC_CUDA_TRY(cudaMemsetAsync(base, 0, cleared * sizeof(unsigned), c.stream));
    return TC_OK;
}

// The order of a solve's targets, on the auxiliary stream from where the sources' frame is on the
// main one (all that it needs): beside the rest of the source sort and the tree build.  After the
// tree it delayed the lists and with them the evaluation: FP64 solves of 64K sources and targets
// 386 -> 356 us, 131K 852 -> 819, 4M 13.19 -> 13.11 ms; mixed, 700,001 1470 -> 1430 us.
static int targets_beside(Context &c, const double *xt, const double *yt, int m) {
    if (!xt || m <= 0) return TC_OK;
    TC_CUDA_TRY(stream_after(c, c.aux, c.stream, c.ev_fork));
    AuxScope on_aux(c);
    const int rc = sort_targets(c, xt, yt, m, &c.tperm);
    if (rc == TC_OK) c.targets_sorted = true;
    return rc;
}

int sort_sources(Context &c, const double *x, const double *y, const double *v, int n,
                 cudaEvent_t values_ready, const double *xt, const double *yt, int m) {
    const bool ovl = c.launch_overlap;   // launch_pdl chains (tc_set_launch_overlap)
    int rc;
    c.targets_sorted = false;
    c.late_ready = nullptr;   // a late-value sort of an earlier call that failed midway
    double *xs, *ys, *vs;
    int *keys, *perm;
    Frame *frame;
    double4 *partials;
    if ((rc = ensure(c, S_XS, n, &xs)) || (rc = ensure(c, S_YS, n, &ys)) ||
        (rc = ensure(c, S_VS, n, &vs)) || (rc = ensure(c, S_KEYS, n, &keys)) ||
        (rc = ensure(c, S_PERM, n, &perm)))
        return rc;
    // frame and bbox partials share one small buffer
    const int gb = grid_for(n, BBOX_THREADS, 8);
    if ((rc = ensure(c, S_FRAME, sizeof(Frame) + sizeof(double4) * gb + 64, (char **)&frame)))
        return rc;
    partials = reinterpret_cast<double4 *>(reinterpret_cast<char *>(frame) + 64);
    unsigned *done = c.ctrl.bbox_done;
    // (the stalled look-back of the test setting is the general sort's)
    if (n <= SMALL_SORT && c.test_stall != TC_STALL_SORT) {
        const double *v_now = values_ready ? nullptr : v;
        // (not this sort's, but the list builds' scratch: list_scratch)
        double2 *rec;
        if ((rc = ensure(c, S_REC, 2 * (size_t)n, &rec))) return rc;
        // the targets beside them, where they are there already and as few (solves on one stream):
        // 4096 sources and targets FP64 162 -> 142 us, mixed 221 -> 201 us
        int *tperm = nullptr;
        if (xt && c.single && m > 0 && m <= SMALL_SORT) {
            if ((rc = ensure(c, S_TPERM, m, &tperm))) return rc;
            c.tperm = tperm;
            c.targets_sorted = true;
        }
        rc = std::max(n, tperm ? m : 0) <= 4 * SMALL_THREADS
                 ? sort_small<4>(c, x, y, v_now, n, frame, keys, perm, xs, ys, vs, xt, yt, m, tperm)
                 : sort_small<16>(c, x, y, v_now, n, frame, keys, perm, xs, ys, vs, xt, yt, m, tperm);
        if (rc || (!c.single && (rc = targets_beside(c, xt, yt, m)))) return rc;
        c.nsrc = n;
        if (values_ready) {
            c.late_x = c.late_y = nullptr;   // x and y are sorted; v in finish_sources
            c.late_v = v;
            c.late_ready = values_ready;
        }
        return TC_OK;
    }

    // four 8-bit passes over the (key, index) items, then one gather of the records
    if (n >= (1 << 30)) {
        set_error(TC_ERR_INVALID, "too many sources for the radix sort (%d)", n);
        return TC_ERR_INVALID;
    }
    unsigned long long *items_a, *items_b;
    double2 *rec;
    const int npasses = (2 * LMAX + 7) / 8;
    const int ntiles = sort_tiles(n);
    if ((rc = ensure(c, S_ITEMS_A, n, &items_a)) || (rc = ensure(c, S_ITEMS_B, n, &items_b)) ||
        (rc = ensure(c, S_REC, 2 * (size_t)n, &rec)))
        return rc;
    // every counter is cleared at the solve's start (ctrl_prepare), so that the sort's kernels
    // follow each other directly on the stream (launch_pdl)
    int *hist = c.ctrl.hist, *offsets = c.ctrl.offsets, *counter = c.ctrl.tile_ctr;
    int *bucket_fill = c.ctrl.bucket_fill;
    unsigned *status = c.ctrl.status, *sink = c.ctrl.sink;
    k_bbox<<<gb, BBOX_THREADS, 0, c.stream>>>(x, y, n, partials, done, frame);
    TC_KERNEL_CHECK();
    if ((rc = targets_beside(c, xt, yt, m))) return rc;
    // resident values: the records are written by the first pass, in buckets (see FirstPass);
    // values that arrive later: items in input order; x, y, v gathered by the permutation
    // in finish_sources
    const bool bucketed = values_ready == nullptr;
    if (bucketed)
        TC_CUDA_TRY(launch_pdl(ovl, k_key_hist, grid_for(n, 256, 8), 256, 0, c.stream, x, y, n,
                               (const Frame *)frame, npasses, hist));
    else
        TC_CUDA_TRY(launch_pdl(ovl, k_keys_pack, grid_for(n, 256, 8), 256, 0, c.stream, x, y, n,
                               (const Frame *)frame, items_a, npasses, hist));
    TC_KERNEL_CHECK();
    TC_CUDA_TRY(launch_pdl(ovl, k_hist_scan, NHIST, RS_RADIX, 0, c.stream, (const int *)hist,
                           offsets));
    TC_KERNEL_CHECK();
    unsigned *err = c.ctrl.err;
    const FirstPass fp = {x, y, v, frame, rec, offsets + RS_MAX_PASSES * RS_RADIX, bucket_fill};
    static_assert((2 * LMAX + 7) / 8 % 2 == 0, "an even number of passes ends in items_a");
    for (int p = 0; p < npasses; ++p) {
        const bool odd = p & 1;
        const int stall = p == 0 && c.test_stall == TC_STALL_SORT ? 0 : -1;
        auto pass_of = [&](auto tile) {
            constexpr int ITEMS = decltype(tile)::value / PS_THREADS;
            if (p > 0) return k_onesweep_items<ITEMS, false>;
            if (stall >= 0)
                return bucketed ? k_onesweep_items<ITEMS, true, true>
                                : k_onesweep_items<ITEMS, false, true>;
            return bucketed ? k_onesweep_items<ITEMS, true> : k_onesweep_items<ITEMS, false>;
        };
        auto pass = sort_tile(n) == PS_TILE ? pass_of(std::integral_constant<int, PS_TILE>{})
                                            : pass_of(std::integral_constant<int, PS_SMALL_TILE>{});
        TC_CUDA_TRY(launch_pdl(ovl, pass, ntiles, PS_THREADS, 0, c.stream,
                               (const unsigned long long *)(odd ? items_b : items_a),
                               odd ? items_a : items_b, n, 32 + 8 * p,
                               (const int *)(offsets + p * RS_RADIX),
                               status + (size_t)p * ntiles * RS_RADIX, counter + p, err,
                               c.spin_limit, stall, sink, fp));
        TC_KERNEL_CHECK();
    }
    c.nsrc = n;
    // a test stall leaves the passes' output unordered: report it before anything reads it
    if (c.test_stall == TC_STALL_SORT && (rc = check_device_errors(c, "source sort"))) return rc;
    if (values_ready) {
        // the keys now (the tree needs nothing else); x, y, v in finish_sources
        TC_CUDA_TRY(launch_pdl(ovl, k_items_split, grid_for(n, 256, 8), 256, 0, c.stream,
                               (const unsigned long long *)items_a, n, keys, perm));
        TC_KERNEL_CHECK();
        c.late_x = x;
        c.late_y = y;
        c.late_v = v;
        c.late_ready = values_ready;
        return TC_OK;
    }
    // a window of the sorted order in flight at a time: its records come from a compact range of
    // buckets, which stays in L2.  The grid is what is resident (2 CTAs per SM): with twice that,
    // half of the stripes ran after the others, and the buckets were read twice (16M sheet, sort
    // phase 1163 -> 1110 us; 1, 3 CTAs or half-size batches: 1190-1240).  One 32-byte load per
    // record instead of two of 16 bytes: the random loads are bound by the L1 tag lookups
    TC_CUDA_TRY(launch_pdl(ovl, k_gather_sources, grid_for(n, GS_THREADS * GS_ITEMS, 2),
                           GS_THREADS, 0, c.stream, (const unsigned long long *)items_a,
                           (const double2 *)rec, n, keys, perm, xs, ys, vs, err));
    TC_KERNEL_CHECK();
    return TC_OK;
}

int finish_sources(Context &c) {
    if (!c.late_ready) return TC_OK;
    const int n = c.nsrc;
    const int *perm = slot_ptr<int>(c, S_PERM);
    if (c.late_x) {
        k_gather_xy<<<grid_for(n, 256, 8), 256, 0, c.stream>>>(perm, c.late_x, c.late_y, n,
                                                              slot_ptr<double>(c, S_XS),
                                                              slot_ptr<double>(c, S_YS),
                                                              c.ctrl.err);
        TC_KERNEL_CHECK();
    }
    TC_CUDA_TRY(cudaStreamWaitEvent(c.stream, c.late_ready, 0));
    c.late_ready = nullptr;
    k_gather_v<<<grid_for(n, 256, 8), 256, 0, c.stream>>>(perm, c.late_v, n,
                                                         slot_ptr<double>(c, S_VS));
    TC_KERNEL_CHECK();
    return TC_OK;
}



// The targets' Morton order in the sources' frame: *perm is one of the buffers.
int sort_targets(Context &c, const double *xt, const double *yt, int m, int **perm) {
    int *tkeys, *tperm, *tkeys2, *tperm2, rc, *ko;
    if ((rc = ensure(c, S_TPERM, m, &tperm))) return rc;
    if (m <= SMALL_SORT) {
        *perm = tperm;
        return m <= 4 * SMALL_THREADS ? sort_small_targets<4>(c, xt, yt, m, tperm)
                                      : sort_small_targets<16>(c, xt, yt, m, tperm);
    }
    if ((rc = ensure(c, S_TKEYS, m, &tkeys)) || (rc = ensure(c, S_TKEYS2, m, &tkeys2)) ||
        (rc = ensure(c, S_TPERM2, m, &tperm2)))
        return rc;
    k_target_keys<<<grid_for(m, 256), 256, 0, c.stream>>>(xt, yt, m, slot_ptr<Frame>(c, S_FRAME),
                                                          tkeys, c.ctrl.meta + META_WIDE);
    TC_KERNEL_CHECK();
    return radix_sort_pairs(c, tkeys, nullptr, m, 2 * LMAX, tkeys2, tperm2, tkeys, tperm, &ko, perm);
}

// ---------------------------------------------------------------------------- allocation-free
// Source sort for callers that cannot allocate device memory, on the kernels the host entry
// points run (k_bbox, k_keys_pack, four k_onesweep_items passes).  The caller's output arrays
// double as the passes' ping-pong buffers: the 8-byte items live in xsorted and ysorted until
// the last pass, and the gather then overwrites them in place.  Everything else -- the
// per-tile look-back words, the digit histograms and their scans, the tile counters, the
// bounding-box partials and the error word -- lives in one static device array of fixed size,
// so a call makes no cudaMalloc/cudaFree and no other allocating call.
constexpr int NOALLOC_MAX_SOURCES = 1 << 20;
constexpr int NA_MAX_TILES = (NOALLOC_MAX_SOURCES + PS_TILE - 1) / PS_TILE;
constexpr int NA_MAX_BBOX_BLOCKS = 4096;
constexpr size_t NA_OFF_STATUS = 0;
constexpr size_t NA_OFF_HIST =
    NA_OFF_STATUS + sizeof(unsigned) * RS_MAX_PASSES * NA_MAX_TILES * RS_RADIX;
constexpr size_t NA_OFF_CTR = NA_OFF_HIST + sizeof(int) * 2 * RS_MAX_PASSES * RS_RADIX;
constexpr size_t NA_OFF_ERR = NA_OFF_CTR + 256;
constexpr size_t NA_OFF_DONE = NA_OFF_ERR + 256;
constexpr size_t NA_OFF_PARTIALS = NA_OFF_DONE + 256;
constexpr size_t NA_BYTES = NA_OFF_PARTIALS + sizeof(double4) * NA_MAX_BBOX_BLOCKS;  // ~1.5 MB

// One copy per device that loads the library, held until the process exits.  In host code
// the name is only a host-side handle: kernels get the device address from
// cudaGetSymbolAddress (noalloc_scratch_base), never the symbol itself.
static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

static unsigned char *noalloc_scratch_base(int device) {
    constexpr int MAX_DEVICES = 64;
    static std::mutex mu;
    static void *addr[MAX_DEVICES] = {};
    if (device < 0 || device >= MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[device]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) {
            set_error(TC_ERR_CUDA, "tc_sort_sources_noalloc: cudaGetSymbolAddress failed: %s",
                      cudaGetErrorString(e));
            return nullptr;
        }
        addr[device] = p;
    }
    return static_cast<unsigned char *>(addr[device]);
}

int prepare_sort() {
    int rc;
    if ((rc = allow_shared((const void *)k_sort_small<4>, small_smem<4>())) ||
        (rc = allow_shared((const void *)k_sort_small<16>, small_smem<16>())) ||
        (rc = allow_shared((const void *)k_sort_small_targets<4>, small_smem<4>())) ||
        (rc = allow_shared((const void *)k_sort_small_targets<16>, small_smem<16>())))
        return rc;
    return TC_OK;
}

void kernels_sort(KernelList &v) {
    v.insert(v.end(), {(const void *)k_bbox, (const void *)k_target_keys,
                       (const void *)k_gather_items_inplace, (const void *)k_hist,
                       (const void *)k_hist_scan,
                       (const void *)k_onesweep, (const void *)k_keys_pack,
                       (const void *)k_onesweep_items<12, true>,
                       (const void *)k_onesweep_items<12, false>, (const void *)k_key_hist,
                       (const void *)k_onesweep_items<12, true, true>,
                       (const void *)k_onesweep_items<12, false, true>,
                       (const void *)k_onesweep_items<8, true>,
                       (const void *)k_onesweep_items<8, false>,
                       (const void *)k_onesweep_items<8, true, true>,
                       (const void *)k_onesweep_items<8, false, true>,
                       (const void *)k_gather_sources, (const void *)k_gather_xy,
                       (const void *)k_gather_v, (const void *)k_items_split,
                       (const void *)k_scan_reduce, (const void *)k_scan_blocks,
                       (const void *)k_scan_apply, (const void *)k_scan_small,
                       (const void *)k_sort_small<4>, (const void *)k_sort_small<16>,
                       (const void *)k_sort_small_targets<4>,
                       (const void *)k_sort_small_targets<16>});
}

}  // namespace tc

extern "C" TC_API int tc_sort_sources_noalloc(const double *xsources, const double *ysources,
                                              const double *sourcevalues, int nsources,
                                              int *keys, int *perm, double *xsorted,
                                              double *ysorted, double *vsorted, double *frame,
                                              void *cuda_stream) {
    using namespace tc;
    set_error(TC_OK, "");
    const int n = nsources;
    if (n < 0 || n > NOALLOC_MAX_SOURCES) {
        set_error(TC_ERR_INVALID,
                  "tc_sort_sources_noalloc: nsources = %d is outside [0, %d], the size of its "
                  "fixed scratch array", n, NOALLOC_MAX_SOURCES);
        return TC_ERR_INVALID;
    }
    if (n == 0) return TC_OK;
    if (!xsources || !ysources || !sourcevalues || !keys || !perm || !xsorted || !ysorted ||
        !vsorted || !frame) {
        set_error(TC_ERR_INVALID, "tc_sort_sources_noalloc: NULL array argument");
        return TC_ERR_INVALID;
    }
    int dev = 0;
    TC_CUDA_TRY(cudaGetDevice(&dev));
    unsigned char *base = noalloc_scratch_base(dev);
    if (!base) {
        if (treecode_last_status() == TC_OK)
            set_error(TC_ERR_INVALID, "tc_sort_sources_noalloc: device %d not supported", dev);
        return treecode_last_status();
    }
    cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
    unsigned *status = reinterpret_cast<unsigned *>(base + NA_OFF_STATUS);
    int *hist = reinterpret_cast<int *>(base + NA_OFF_HIST);
    int *offsets = hist + RS_MAX_PASSES * RS_RADIX;
    int *counter = reinterpret_cast<int *>(base + NA_OFF_CTR);
    unsigned *err = reinterpret_cast<unsigned *>(base + NA_OFF_ERR);
    unsigned *done = reinterpret_cast<unsigned *>(base + NA_OFF_DONE);
    double4 *partials = reinterpret_cast<double4 *>(base + NA_OFF_PARTIALS);
    Frame *fr = reinterpret_cast<Frame *>(frame);
    // the passes' ping-pong buffers: the caller's xsorted / ysorted, as 8-byte items
    unsigned long long *items_a = reinterpret_cast<unsigned long long *>(xsorted);
    unsigned long long *items_b = reinterpret_cast<unsigned long long *>(ysorted);

    // The array keeps the previous call's contents: clear what has to start at zero.
    const int npasses = (2 * LMAX + 7) / 8;
    const int ntiles = (n + PS_TILE - 1) / PS_TILE;
    TC_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(unsigned), s));
    TC_CUDA_TRY(cudaMemsetAsync(done, 0, sizeof(unsigned), s));
    TC_CUDA_TRY(cudaMemsetAsync(hist, 0, sizeof(int) * RS_MAX_PASSES * RS_RADIX, s));
    TC_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int) * RS_MAX_PASSES, s));
    TC_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(unsigned) * (size_t)npasses * ntiles * RS_RADIX, s));

    const int gb = std::min(grid_for(n, BBOX_THREADS, 8), NA_MAX_BBOX_BLOCKS);
    k_bbox<<<gb, BBOX_THREADS, 0, s>>>(xsources, ysources, n, partials, done, fr);
    TC_KERNEL_CHECK();
    k_keys_pack<<<grid_for(n, 256, 8), 256, 0, s>>>(xsources, ysources, n, fr, items_a, npasses,
                                                    hist);
    TC_KERNEL_CHECK();
    k_hist_scan<<<npasses, RS_RADIX, 0, s>>>(hist, offsets);
    TC_KERNEL_CHECK();
    static_assert((2 * LMAX + 7) / 8 % 2 == 0, "an even number of passes ends in items_a");
    for (int p = 0; p < npasses; ++p) {
        const bool odd = p & 1;
        k_onesweep_items<12, false><<<ntiles, PS_THREADS, 0, s>>>(
            odd ? items_b : items_a, odd ? items_a : items_b, n, 32 + 8 * p,
            offsets + p * RS_RADIX, status + (size_t)p * ntiles * RS_RADIX, counter + p, err,
            RS_SPIN_LIMIT, -1, nullptr, FirstPass{});
        TC_KERNEL_CHECK();
    }
    k_gather_items_inplace<<<grid_for(n, 256), 256, 0, s>>>(xsources, ysources, sourcevalues, n,
                                                             keys, perm, xsorted, ysorted,
                                                             vsorted, err);
    TC_KERNEL_CHECK();
    unsigned h_err = 0;
    TC_CUDA_TRY(cudaMemcpyAsync(&h_err, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    TC_CUDA_TRY(cudaStreamSynchronize(s));
    if (h_err) {
        set_error(h_err & DEVERR_SPIN_LIMIT ? TC_ERR_TIMEOUT : TC_ERR_CUDA,
                  "tc_sort_sources_noalloc: device error flags 0x%x", h_err);
        return treecode_last_status();
    }
    return TC_OK;
}
