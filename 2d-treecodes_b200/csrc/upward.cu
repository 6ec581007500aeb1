// upward.cu -- the upward pass, in two parts.
//
// Moments (what the traversals read): k_leaf_setup_warp (a warp per node) or k_leaf_setup (four
// threads per node, for many nodes) runs the leaf setup with the reference's four strided accumulators (drivers/upward.cpp:61-93,
// kernels/upward-common.ispc:13-57); k_moments_level / k_moments_top then form every inner
// node's mass, weights, com and radius level by level, deepest first (upward.cpp:95-218).
// Expansions: k_leaf_p2e (one warp per leaf, lanes over sources, FP32 lane sums in the
// mixed-precision form; kernels/upward-kernels.m4:18-93), then E2E deepest level first
// (upward-kernels.m4:95-149): k_upward_wide (four threads per inner node, one per child) on wide
// levels, k_upward_level (warp per inner node) on narrow ones, k_upward_top (one block) on the
// small top levels.  Inner node r of level l is addressed structurally (its children are
// off[l+1] + 4r .. +3, its id is their cell's parent), so the E2E does not depend on the child
// pointers that the moments pass may rewrite.  The two parts are separate so that the
// interaction lists can be built on another stream while the expansions are formed.
//
// Bit-exact restatements (decisions of the traversals depend on these values):
//  * leaf mass / |v| weights / weighted sums: four strided lane accumulators, reduced as
//    (l0 + l1) + (l2 + l3); a lane whose own weight sum is zero measures the radius about the
//    origin (upward-common.ispc:44-45 tests the varying wsum);
//  * leaf com = wx/w, or the cell centre fma(0.5, h, fma(cx, h, xmin)) when w == 0;
//  * parent sums over children as (c0 + c3) + (c1 + c2): the reference's source adds c0..c3 in
//    sequence (upward.cpp:105-115), and this is the reassociation g++ -O3 --fast-math (the
//    reference's release flags) makes of that loop in the compiled driver the parity tests
//    run against; a build of the reference without fast-math would sum in sequence;
//  * parent radius min(max_c (sqrt(fma(rx, rx, ry*ry)) + r_c), (double)1.4143f * ext / 2^l)
//    over children with nonzero weight;
//  * when all four children are negligible (|w| < 1.1e-16) the parent's expansion is zeroed and
//    the child that arrives last becomes an empty leaf (upward.cpp:173-180).  Which child that
//    is depends on the reference's OpenMP task timing; below the task threshold (5000 sources
//    per cell, upward.cpp:271) its subtrees complete in child order, so it is child 3, which is
//    what this code always picks (the oracle fixtures take that serial path); with exactly
//    three negligible children the remaining
//    child's coefficients are copied unshifted (upward.cpp:182-188).
// The expansion coefficients themselves are sums whose order is free (the parity gate on them
// is a relative tolerance), so P2E and E2E use whatever order suits the GPU.
//
// Expansion layout: exps[node][0][k] real parts, exps[node][1][k] imaginary parts, k < ORDER.
#include <algorithm>
#include <type_traits>

#include "tc_internal.h"
#include "tc_math.cuh"

namespace tc {

__constant__ BinomTable c_binom_up = make_binom_table();   // uniform indices only
__device__ const BinomTable g_binom_up = make_binom_table();   // per-lane indices

constexpr int UP_WARPS = 4;          // warps per block of the leaf and per-level merge kernels
constexpr int UP_TOP_WARPS = 16;     // warps of the single-block launch over the top levels
// A level this small joins the single-block launch.  One SM reads the children of 64 nodes no
// faster than a launch over several takes (a launch follows in ~2.5 us): 64 -> 16 took ~8 us off
// the upward phase of solves of 64K to 1M sources, and nothing off the smallest.
constexpr int UP_TOP_MAX_NODES = 16;
constexpr int UP_WIDE_MIN_NODES = 2048;  // a level with this many inner nodes: k_upward_wide


__device__ __forceinline__ bool is_leaf(int2 rg, int4 cl, int leafcap) {
    return (rg.y - rg.x <= leafcap) || cl.x == LMAX;
}

// ------------------------------------------------------------------------------ leaves
// A leaf's moments from its sums: com (upward.cpp:71-72; x0 = fma(cx, h, xmin) as in build_tree).
__device__ __forceinline__ void leaf_record(int node, int4 cl, double msum, double wsum,
                                            double xsum, double ysum, double r2, TNode *tnode,
                                            double *mass, double *wgt, double *wxs, double *wys,
                                            const Frame *__restrict__ frame) {
    double xcom, ycom;
    if (wsum != 0) {
        xcom = __ddiv_rn(xsum, wsum);
        ycom = __ddiv_rn(ysum, wsum);
    } else {
        const Frame f = *frame;
        const double h = __ddiv_rn(f.ext, (double)(1 << cl.x));
        xcom = __fma_rn(0.5, h, __fma_rn((double)cl.y, h, f.xmin));
        ycom = __fma_rn(0.5, h, __fma_rn((double)cl.z, h, f.ymin));
    }
    tnode[node].xcom = xcom;
    tnode[node].ycom = ycom;
    tnode[node].r = __dsqrt_rn(r2);
    mass[node] = msum;
    wgt[node] = wsum;
    wxs[node] = xsum;
    wys[node] = ysum;
}

// k_leaf_setup: lane quad per node (4 threads each, in the order of the node ids).  Only the
// quads of leaves do work; the others still take part in the quad shuffles.
__global__ __launch_bounds__(256) void k_leaf_setup(
    int nnodes, int nsrc, int leafcap, const double *__restrict__ xs, const double *__restrict__ ys,
    const double *__restrict__ vs, const int2 *__restrict__ range, const int4 *__restrict__ cell,
    TNode *tnode, double *mass, double *wgt, double *wxs, double *wys,
    const Frame *__restrict__ frame, unsigned *err) {
    pdl_begin();
    const int lane = lane_id(), q = lane & 3, qbase = lane & ~3;
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int node = (int)(tid >> 2);
    bool act = false;
    int s = 0, e = 0;
    int4 cl = {0, 0, 0, 0};
    if (node < nnodes) {
        const int2 rg = range[node];
        cl = cell[node];
        if (is_leaf(rg, cl, leafcap)) {
            if (rg.x < 0 || rg.y < rg.x || rg.y > nsrc || cl.w >= nnodes || cl.x < 0 || cl.x > LMAX) {
                if (q == 0) atomicOr(err, DEVERR_BOUNDS);
            } else {
                act = true;
                s = rg.x;
                e = rg.y;
            }
        }
    }
    // four strided accumulators: element i goes to lane (i - s) % 4 (upward-common.ispc:24-42)
    double ms = 0, ws = 0, wxl = 0, wyl = 0;
    if (act)
#pragma unroll 8
        for (int j = s + q; j < e; j += 4) {
            const double x = __ldg(xs + j), y = __ldg(ys + j), m = __ldg(vs + j);
            const double w = fabs(m);
            ms = __dadd_rn(ms, m);
            ws = __dadd_rn(ws, w);
            wxl = __dadd_rn(wxl, __dmul_rn(x, w));
            wyl = __dadd_rn(wyl, __dmul_rn(y, w));
        }
    // (l0 + l1) + (l2 + l3) within the quad, broadcast to its four lanes
    auto reduce4 = [&](double v) {
        const double a = __dadd_rn(v, __shfl_down_sync(FULL_MASK, v, 1));
        return __shfl_sync(FULL_MASK, __dadd_rn(a, __shfl_down_sync(FULL_MASK, a, 2)), qbase);
    };
    const double msum = reduce4(ms), wsum = reduce4(ws), xsum = reduce4(wxl), ysum = reduce4(wyl);
    // radius about the per-lane centre (upward-common.ispc:44-56)
    double r2 = 0;
    if (act) {
        const double lx = ws != 0 ? __ddiv_rn(xsum, wsum) : 0.0;
        const double ly = ws != 0 ? __ddiv_rn(ysum, wsum) : 0.0;
#pragma unroll 8
        for (int j = s + q; j < e; j += 4) {
            const double xr = __dsub_rn(__ldg(xs + j), lx), yr = __dsub_rn(__ldg(ys + j), ly);
            r2 = fmax(r2, __dadd_rn(__dmul_rn(xr, xr), __dmul_rn(yr, yr)));
        }
    }
    r2 = fmax(r2, __shfl_xor_sync(FULL_MASK, r2, 1));
    r2 = fmax(r2, __shfl_xor_sync(FULL_MASK, r2, 2));
    if (act && q == 0) {
        leaf_record(node, cl, msum, wsum, xsum, ysum, r2, tnode, mass, wgt, wxs, wys, frame);
    }
}

// The same for fewer nodes: a warp per node.  Few leaves of up to 512 sources are bound by the
// latency of a lane's serial loads; here the warp loads LS_BATCH sources at a time, coalesced,
// leaves v, |v|, x|v|, y|v| in shared memory, and 16 lanes run the 16 chains (four per quantity) of
// the same sums.  The radius is a maximum, so all 32 lanes take part, each about the centre of the
// chain that its sources belong to.  Solves of 4096 sources: potential 172 -> 164 us, force 171 ->
// 164; potential 64K 412 -> 390, 700,001 mixed 1522 -> 1490; force 1M mixed 1044 -> 1030 us.
// The quads do with 0.4 of the instructions and waits per leaf, which counts once the nodes are
// many times the resident warps: equal at 60,000 and 120,000 nodes, at 236,000 (16M sheet) the
// warp form takes 143 us for the quads' 121.
constexpr int LS_WARPS = 4;
constexpr int LS_BATCH = 128;
constexpr int LS_ROW = LS_BATCH + 4;   // padded: the 16 chains' operands in distinct banks
constexpr int LS_U = LS_BATCH / 32;
constexpr int LS_QUAD_NODES = 1 << 16;   // from here on, a quad per node

__global__ __launch_bounds__(LS_WARPS * 32) void k_leaf_setup_warp(
    int nnodes, int nsrc, int leafcap, const double *__restrict__ xs, const double *__restrict__ ys,
    const double *__restrict__ vs, const int2 *__restrict__ range, const int4 *__restrict__ cell,
    TNode *tnode, double *mass, double *wgt, double *wxs, double *wys,
    const Frame *__restrict__ frame, unsigned *err) {
    __shared__ double s_val[LS_WARPS][4][LS_ROW];
    pdl_begin();
    const int lane = lane_id(), q = lane & 3, warp = threadIdx.x >> 5;
    const int node = blockIdx.x * LS_WARPS + warp;
    if (node >= nnodes) return;
    const int2 rg = range[node];
    const int4 cl = cell[node];
    if (!is_leaf(rg, cl, leafcap)) return;
    if (rg.x < 0 || rg.y < rg.x || rg.y > nsrc || cl.w >= nnodes || cl.x < 0 || cl.x > LMAX) {
        if (lane == 0) atomicOr(err, DEVERR_BOUNDS);
        return;
    }
    const int s = rg.x, e = rg.y;
    double(&val)[4][LS_ROW] = s_val[warp];
    // lane 4 c + q holds chain q of quantity c (lanes 16-31 idle); past the end zeros are added,
    // which change no sum
    const double *chain = &val[(lane >> 2) & 3][q];
    double sum = 0;
    double x[LS_U], y[LS_U];
    for (int base = s; base < e; base += LS_BATCH) {
        double m[LS_U];
#pragma unroll
        for (int u = 0; u < LS_U; ++u) {
            const int j = base + 32 * u + lane;
            const bool ok = j < e;
            x[u] = ok ? __ldg(xs + j) : 0.0;
            y[u] = ok ? __ldg(ys + j) : 0.0;
            m[u] = ok ? __ldg(vs + j) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < LS_U; ++u) {
            const double w = fabs(m[u]);
            val[0][32 * u + lane] = m[u];
            val[1][32 * u + lane] = w;
            val[2][32 * u + lane] = __dmul_rn(x[u], w);
            val[3][32 * u + lane] = __dmul_rn(y[u], w);
        }
        __syncwarp();
        if (lane < 16) {
            const int n = (min(LS_BATCH, e - base) + 3) & ~3;
#pragma unroll 8
            for (int i = 0; i < n; i += 4) sum = __dadd_rn(sum, chain[i]);
        }
    }
    __syncwarp();
    // (l0 + l1) + (l2 + l3) of each quantity, broadcast
    const double pair = __dadd_rn(sum, __shfl_down_sync(FULL_MASK, sum, 1));
    const double quad = __dadd_rn(pair, __shfl_down_sync(FULL_MASK, pair, 2));
    const double msum = __shfl_sync(FULL_MASK, quad, 0), wsum = __shfl_sync(FULL_MASK, quad, 4),
                 xsum = __shfl_sync(FULL_MASK, quad, 8), ysum = __shfl_sync(FULL_MASK, quad, 12);
    const double ws = __shfl_sync(FULL_MASK, sum, 4 + q);
    const double lx = ws != 0 ? __ddiv_rn(xsum, wsum) : 0.0;
    const double ly = ws != 0 ? __ddiv_rn(ysum, wsum) : 0.0;
    double r2 = 0;
    auto reach = [&](double xj, double yj) {
        const double xr = __dsub_rn(xj, lx), yr = __dsub_rn(yj, ly);
        r2 = fmax(r2, __dadd_rn(__dmul_rn(xr, xr), __dmul_rn(yr, yr)));
    };
    if (e - s <= LS_BATCH) {   // still in registers
#pragma unroll
        for (int u = 0; u < LS_U; ++u)
            if (s + 32 * u + lane < e) reach(x[u], y[u]);
    } else {
#pragma unroll 8
        for (int j = s + lane; j < e; j += 32) reach(__ldg(xs + j), __ldg(ys + j));
    }
    for (int o = 1; o < 32; o <<= 1) r2 = fmax(r2, __shfl_xor_sync(FULL_MASK, r2, o));
    if (lane == 0)
        leaf_record(node, cl, msum, wsum, xsum, ysum, r2, tnode, mass, wgt, wxs, wys, frame);
}

// k_leaf_p2e: a_n = -1/(n+1) sum_i v_i (z_i - c)^(n+1), one warp per leaf, lanes over sources
// with the P coefficients in registers; the 32 partial sums of each coefficient meet in shared
// memory, transposed, and are added there in parts by all lanes (LEAF_PARTS).
template <int P, class T = double>
struct alignas(16) LeafShared {
    T v[32][2 * P + 1];
};

template <int P, bool MIXED>
constexpr size_t leaf_bytes() {
    return UP_WARPS * sizeof(LeafShared<P, typename std::conditional<MIXED, float, double>::type>);
}

// The 2 P columns of 32 rows are cut in PARTS each, so that all lanes take the same number of cut
// columns (P = 24: 96, three of 16 rows each; P = 12: 96, three of 8 rows).  The mixed form is
// bound by the conversions of these sums: with one lane per coefficient, both its columns and
// lanes from P on idle, 64 a lane instead of 48.  16M sheet: upward phase mixed 592 -> 580 us, FP64
// 675 -> 664.
template <int P>
constexpr int LEAF_PARTS = P % 16 == 0 ? 1 : P % 8 == 0 ? 2 : P % 4 == 0 ? 4 : P % 2 == 0 ? 8 : 16;


// MIXED: the mixed-precision form accumulates in FP32 on offsets scaled by R, the power of two
// at or above the cell's half-diagonal (every source of the leaf lies in its cell, and so does
// the com, so |z / R| <= 1 and no power under- or overflows).  Each lane sums at most
// leafcap/32 terms in FP32; the 32 lane sums are added in FP64 and rescaled by R^(n+1) exactly.
template <int P, bool MIXED>
__global__ __launch_bounds__(UP_WARPS * 32, MIXED ? 4 : 3) void k_leaf_p2e(
    int nnodes, int nsrc, int leafcap, const double *__restrict__ xs, const double *__restrict__ ys,
    const double *__restrict__ vs, const int2 *__restrict__ range, const int4 *__restrict__ cell,
    const TNode *__restrict__ tnode, double *exps, const Frame *__restrict__ frame) {
    pdl_begin();
    using acc_t = typename std::conditional<MIXED, float, double>::type;
    constexpr int PARTS = LEAF_PARTS<P>, TASKS = 2 * P * PARTS / 32, ROWS = 32 / PARTS;
    static_assert(ROWS % 2 == 0 && sizeof(LeafShared<P, acc_t>) >= 32 * TASKS * sizeof(double));
    constexpr int U = MIXED ? 4 : (P > 16 ? 6 : 4);   // sources per lane in flight
    extern __shared__ __align__(16) unsigned char leaf_smem[];
    LeafShared<P, acc_t> &sh = reinterpret_cast<LeafShared<P, acc_t> *>(leaf_smem)[threadIdx.x >> 5];
    const int lane = lane_id();
    const double ext = frame->ext;
    const int stride = gridDim.x * UP_WARPS;
    int next = blockIdx.x * UP_WARPS + (threadIdx.x >> 5);
    // the next node's record is loaded while the current leaf is expanded
    int2 nrg = {0, 0};
    int4 ncl = {0, 0, 0, 0};
    double ncx = 0, ncy = 0;
    // (the com only for leaves: the parents' moments may be written meanwhile)
    if (next < nnodes) {
        nrg = range[next];
        ncl = cell[next];
        if (is_leaf(nrg, ncl, leafcap)) {
            ncx = tnode[next].xcom;
            ncy = tnode[next].ycom;
        }
    }
    while (next < nnodes) {
        const int node = next;
        const int2 rg = nrg;
        const int4 cl = ncl;
        const double cx = ncx, cy = ncy;
        next += stride;
        if (next < nnodes) {
            nrg = range[next];
            ncl = cell[next];
            if (is_leaf(nrg, ncl, leafcap)) {
                ncx = tnode[next].xcom;
                ncy = tnode[next].ycom;
            }
        }
        if (!is_leaf(rg, cl, leafcap) || rg.x < 0 || rg.y < rg.x || rg.y > nsrc) continue;
        int e = 0;   // R = 2^e (mixed form)
        if (MIXED) frexp(1.4142135623730951 * (1.0 + 1e-12) * ldexp(ext, -cl.x), &e);
        const double inv_r = MIXED ? ldexp(1.0, -e) : 1.0;
        acc_t ar[P], ai[P];
#pragma unroll
        for (int n = 0; n < P; ++n) ar[n] = ai[n] = acc_t(0);
        // mixed form: the powers in consecutive pairs (v z^(n+1), v z^(n+2)) held in f32x2
        // lanes and advanced by z^2, so one paired instruction does the work of two
        float2 ar2[P / 2], ai2[P / 2];
        if constexpr (MIXED) {
#pragma unroll
            for (int n = 0; n < P / 2; ++n) ar2[n] = ai2[n] = make_float2(0.f, 0.f);
        }
        for (int base = rg.x; base < rg.y; base += 32 * U) {
            const int nu = min(U, (rg.y - base + 31) >> 5);   // warp-uniform
            acc_t zr[U], zi[U], v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = base + 32 * u + lane;
                const bool ok = u < nu && j < rg.y;
                zr[u] = ok ? acc_t((__ldg(xs + j) - cx) * inv_r) : acc_t(0);
                zi[u] = ok ? acc_t((__ldg(ys + j) - cy) * inv_r) : acc_t(0);
                v[u] = ok ? acc_t(__ldg(vs + j)) : acc_t(0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (u >= nu) break;
                if constexpr (MIXED) {
                    const float p1r = v[u] * zr[u], p1i = v[u] * zi[u];
                    const float p2r = fmaf(p1r, zr[u], -p1i * zi[u]);
                    const float p2i = fmaf(p1r, zi[u], p1i * zr[u]);
                    const float z2r = fmaf(zr[u], zr[u], -zi[u] * zi[u]);
                    const float z2i = 2.f * zr[u] * zi[u];
                    const float2 z2r2 = make_float2(z2r, z2r), z2i2 = make_float2(z2i, z2i);
                    const float2 nz2i2 = make_float2(-z2i, -z2i);
                    float2 re2 = make_float2(p1r, p2r), im2 = make_float2(p1i, p2i);
#pragma unroll
                    for (int n = 0; n < P / 2; ++n) {
                        ar2[n] = __fadd2_rn(ar2[n], re2);
                        ai2[n] = __fadd2_rn(ai2[n], im2);
                        if (n + 1 < P / 2) {
                            const float2 nre = __ffma2_rn(re2, z2r2, __fmul2_rn(im2, nz2i2));
                            im2 = __ffma2_rn(re2, z2i2, __fmul2_rn(im2, z2r2));
                            re2 = nre;
                        }
                    }
                } else {
                    acc_t pr = v[u] * zr[u], pim = v[u] * zi[u];
#pragma unroll
                    for (int n = 0; n < P; ++n) {
                        ar[n] += pr;
                        ai[n] += pim;
                        const acc_t tr = fma(pr, zr[u], -pim * zi[u]);
                        pim = fma(pr, zi[u], pim * zr[u]);
                        pr = tr;
                    }
                }
            }
        }
        if constexpr (MIXED) {
#pragma unroll
            for (int n = 0; n < P / 2; ++n) {
                ar[2 * n] = ar2[n].x;
                ar[2 * n + 1] = ar2[n].y;
                ai[2 * n] = ai2[n].x;
                ai[2 * n + 1] = ai2[n].y;
            }
        }
        __syncwarp();
#pragma unroll
        for (int n = 0; n < P; ++n) {
            sh.v[lane][n] = ar[n];
            sh.v[lane][P + n] = ai[n];
        }
        __syncwarp();
        double part[TASKS];
#pragma unroll
        for (int k = 0; k < TASKS; ++k) {
            const int t = 32 * k + lane;
            const acc_t *col = &sh.v[t / (2 * P) * ROWS][t % (2 * P)];
            double s0 = 0, s1 = 0;
#pragma unroll 8
            for (int i = 0; i < ROWS; i += 2) {
                s0 += (double)col[i * (2 * P + 1)];
                s1 += (double)col[(i + 1) * (2 * P + 1)];
            }
            part[k] = s0 + s1;
        }
        __syncwarp();
        double *parts = reinterpret_cast<double *>(&sh);
#pragma unroll
        for (int k = 0; k < TASKS; ++k) parts[32 * k + lane] = part[k];
        __syncwarp();
        if (lane < P) {
            double sr = parts[lane], si = parts[P + lane];
#pragma unroll
            for (int h = 1; h < PARTS; ++h) {
                sr += parts[h * 2 * P + lane];
                si += parts[h * 2 * P + P + lane];
            }
            double fac = -1.0 / (lane + 1);
            if (MIXED) fac = ldexp(fac, e * (lane + 1));
            double *ex = exps + (size_t)node * 2 * P;
            ex[lane] = sr * fac;
            ex[P + lane] = si * fac;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------ moments
// Parent moments, bit-exact (upward.cpp:95-218): sums over the children as (c0 + c3) + (c1 + c2),
// com = wx / w, radius min(max_c |com - com_c| + r_c over weighted children, (double)1.4143f ext
// / 2^l); when all four children are negligible child 3 becomes an empty leaf.  These are what
// the traversals read; they run level by level before any expansion work, so that the
// interaction lists can be built while the expansions are still being formed.
// Inner node r of level l owns the children off[l+1] + 4r .. +3 and is their common parent
// cell[off[l+1] + 4r].w.
__device__ __forceinline__ void parent_moments(int l, int cb, int parent, double ext,
                                               TNode *tnode, double *mass, double *wgt,
                                               double *wxs, double *wys) {
    double cm[4], cw[4], cwx[4], cwy[4], cxc[4], cyc[4], cr[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        cm[c] = mass[cb + c];
        cw[c] = wgt[cb + c];
        cwx[c] = wxs[cb + c];
        cwy[c] = wys[cb + c];
        cxc[c] = tnode[cb + c].xcom;
        cyc[c] = tnode[cb + c].ycom;
        cr[c] = tnode[cb + c].r;
    }
    const double pm = __dadd_rn(__dadd_rn(cm[0], cm[3]), __dadd_rn(cm[1], cm[2]));
    const double pw = __dadd_rn(__dadd_rn(cw[0], cw[3]), __dadd_rn(cw[1], cw[2]));
    const double pwx = __dadd_rn(__dadd_rn(cwx[0], cwx[3]), __dadd_rn(cwx[1], cwx[2]));
    const double pwy = __dadd_rn(__dadd_rn(cwy[0], cwy[3]), __dadd_rn(cwy[1], cwy[2]));
    const double px = __ddiv_rn(pwx, pw), py = __ddiv_rn(pwy, pw);
    double rr = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (cw[c] != 0) {
            const double rx = __dsub_rn(px, cxc[c]), ry = __dsub_rn(py, cyc[c]);
            const double cand = __dadd_rn(__dsqrt_rn(__fma_rn(rx, rx, __dmul_rn(ry, ry))), cr[c]);
            rr = cand > rr ? cand : rr;
        }
    const double cap = __ddiv_rn(__dmul_rn((double)1.4143f, ext), (double)(1 << l));
    int zcount = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) zcount += fabs(cw[c]) < 1.1e-16;
    tnode[parent].xcom = px;
    tnode[parent].ycom = py;
    tnode[parent].r = cap < rr ? cap : rr;
    mass[parent] = pm;
    wgt[parent] = pw;
    wxs[parent] = pwx;
    wys[parent] = pwy;
    if (zcount == 4) {
        tnode[cb + 3].child = -1;
        tnode[cb + 3].count = 0;
    }
}

// Inner node r of the level whose nodes are [lo, mid): its children from cb on, and its id.
__device__ __forceinline__ bool inner_node(int r, int lo, int mid, int nnodes,
                                           const int4 *__restrict__ cell, int &cb, int &parent,
                                           unsigned *err) {
    cb = mid + 4 * r;
    parent = cb + 4 <= nnodes ? cell[cb].w : -1;
    if (parent < lo || parent >= mid) {
        atomicOr(err, DEVERR_TREE);
        return false;
    }
    return true;
}

// one level, one thread per inner node
__global__ __launch_bounds__(256) void k_moments_level(int l, LevelOffsets lo, int nnodes,
                                                       const int4 *__restrict__ cell, TNode *tnode,
                                                       double *mass, double *wgt, double *wxs,
                                                       double *wys, const Frame *__restrict__ frame,
                                                       unsigned *err) {
    // the tree and the frame are complete; the children's moments from pdl_begin on
    const int r = blockIdx.x * blockDim.x + threadIdx.x;   // (a thread per inner node)
    const double ext = frame->ext;
    int cb = 0, parent = 0;
    const bool ok = r < (lo.off[l + 2] - lo.off[l + 1]) / 4 &&
                    inner_node(r, lo.off[l], lo.off[l + 1], nnodes, cell, cb, parent, err);
    pdl_begin();
    if (ok) parent_moments(l, cb, parent, ext, tnode, mass, wgt, wxs, wys);
}

// levels ltop .. 0 in one block, a block barrier between levels
// Levels with at most this many inner nodes: one block.  With 1024 the single SM's share of the
// L2 bandwidth bound it (28 words a node: 43 us on the 16M sheet); at 64 the wide levels get
// launches of their own: the upward phase of a 300K-source solve 127 -> 102 us.
constexpr int MOM_TOP_MAX = 64;
__global__ __launch_bounds__(MOM_TOP_MAX) void k_moments_top(int ltop, LevelOffsets lo, int nnodes,
                                                      const int4 *__restrict__ cell, TNode *tnode,
                                                      double *mass, double *wgt, double *wxs,
                                                      double *wys, const Frame *__restrict__ frame,
                                                      unsigned *err) {
    pdl_begin();
    const double ext = frame->ext;
    for (int l = ltop; l >= 0; --l) {
        const int ninner = (lo.off[l + 2] - lo.off[l + 1]) / 4;
        for (int r = threadIdx.x; r < ninner; r += blockDim.x) {
            int cb, parent;
            if (inner_node(r, lo.off[l], lo.off[l + 1], nnodes, cell, cb, parent, err))
                parent_moments(l, cb, parent, ext, tnode, mass, wgt, wxs, wys);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------ merge (E2E)
// b_l = sum_c z0^l [ -m_c/l + sum_{k=1..l} C(l-1,k-1) a_{c,k-1} z0^-k ],  z0 = child com - parent
// com (upward-kernels.m4:95-149).  All four children are shifted unless three or four of them
// are negligible: four -> the parent's expansion is zero; three -> the remaining child's
// coefficients are copied unshifted (upward.cpp:173-188).
// Narrow levels: a warp per inner node; lane l-1 (l = 1..P) owns coefficient l of the parent
// for all four children, with the binomials C(l-1, k-1) (zero for k > l) from a block-shared
// table, row k.
template <int P>
struct MergeShared {
    cplx coef[4][P];   // a_{c,k-1} z0_c^-k, k = 1..P
};

template <int P>
struct BinomRows {
    double b[P][32];   // b[k][lane] = C(lane, k) for k <= lane < P, else 0
};

template <int P>
__device__ __forceinline__ void fill_binom_rows(BinomRows<P> &t) {
    for (int i = threadIdx.x; i < P * 32; i += blockDim.x) {
        const int k = i / 32, l = i % 32;
        t.b[k][l] = (l < P && k <= l) ? g_binom_up.c[l][k] : 0.0;
    }
}

// What a merge needs besides the children's coefficients: their moments, which every E2E kernel
// finds complete (a kernel starts only once the one before it has seen its own predecessor
// complete, and the moments are older than any E2E kernel), and the powers z0_c^-l of this
// lane's l.  An E2E kernel forms the first node's before it waits for the level below
// (pdl_begin): the loads, the reciprocals and the powers are most of a narrow level's latency.
// Upward phase of a 256K-source solve 84 -> 75 us, 1M 149 -> 137.
struct MergeGeom {
    int cb, parent, zcount, nz;
    bool ok;
    double cm[4];
    cplx zl[4];
};

template <int P>
__device__ __forceinline__ void merge_geom(MergeGeom &g, int r, int lo, int mid,
                                           int nnodes, const int4 *__restrict__ cell,
                                           const TNode *tnode, const double *mass,
                                           const double *wgt, unsigned *err) {
    const int lane = lane_id();
    int cb = 0, parent = 0;
    bool ok = true;
    if (lane == 0) ok = inner_node(r, lo, mid, nnodes, cell, cb, parent, err);
    g.ok = __shfl_sync(FULL_MASK, ok, 0);
    g.cb = __shfl_sync(FULL_MASK, cb, 0);
    g.parent = __shfl_sync(FULL_MASK, parent, 0);
    if (!g.ok) return;
    g.zcount = 0;
    double cw[4], cxc[4], cyc[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        g.cm[c] = mass[g.cb + c];
        cw[c] = wgt[g.cb + c];
        cxc[c] = tnode[g.cb + c].xcom;
        cyc[c] = tnode[g.cb + c].ycom;
    }
    const double px = tnode[g.parent].xcom, py = tnode[g.parent].ycom;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const bool negl = fabs(cw[c]) < 1.1e-16;
        g.zcount += negl;
        g.nz = negl ? g.nz : c;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {   // (unused with three or four negligible children)
        const double x0 = cxc[c] - px, y0 = cyc[c] - py;
        const double iz = rcp_any(x0 * x0 + y0 * y0);
        g.zl[c] = cpow_int({x0 * iz, -y0 * iz}, lane < P ? lane + 1 : 1);
    }
}

template <int P>
__device__ __forceinline__ void merge_node(const MergeGeom &g, double *exps,
                                           const BinomRows<P> &bt, MergeShared<P> &sh) {
    const int lane = lane_id();
    // this lane's coefficient of each child
    double er[4] = {0, 0, 0, 0}, ei[4] = {0, 0, 0, 0};
    if (lane < P)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double *ex = exps + (size_t)(g.cb + c) * 2 * P;
            er[c] = ex[lane];
            ei[c] = ex[P + lane];
        }
    double *dst = exps + (size_t)g.parent * 2 * P;
    if (g.zcount == 4) {
        for (int k = lane; k < 2 * P; k += 32) dst[k] = 0.0;
    } else if (g.zcount == 3) {
        double sr = 0, si = 0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sr = c == g.nz ? er[c] : sr;
            si = c == g.nz ? ei[c] : si;
        }
        if (lane < P) {
            dst[lane] = sr;
            dst[P + lane] = si;
        }
    } else {
        const int l = lane + 1;
        __syncwarp();
        if (lane < P)
#pragma unroll
            for (int c = 0; c < 4; ++c) sh.coef[c][lane] = cmul({er[c], ei[c]}, g.zl[c]);
        __syncwarp();
        if (lane < P) {
            const double minv = -1.0 / l;
            double tr[4], ti[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                tr[c] = l == 1 ? -g.cm[c] : g.cm[c] * minv;
                ti[c] = 0.0;
            }
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const double b = bt.b[k][lane];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const cplx a = sh.coef[c][k];
                    tr[c] = fma(b, a.re, tr[c]);
                    ti[c] = fma(b, a.im, ti[c]);
                }
            }
            // z0^l = 1 / z0^-l
            double sr[4], si[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double invz2 = g.zl[c].re * g.zl[c].re + g.zl[c].im * g.zl[c].im;
                const double inv = invz2 != 0 ? 1.0 / invz2 : 0.0;
                const double rz = g.zl[c].re * inv, iz = -g.zl[c].im * inv;
                sr[c] = tr[c] * rz - ti[c] * iz;
                si[c] = tr[c] * iz + ti[c] * rz;
            }
            dst[lane] = (sr[0] + sr[1]) + (sr[2] + sr[3]);
            dst[P + lane] = (si[0] + si[1]) + (si[2] + si[3]);
        }
    }
    __syncwarp();
}

// One level, one warp per inner node.
template <int P>
__global__ __launch_bounds__(UP_WARPS * 32, 5) void k_upward_level(
    int l, LevelOffsets lo, int nnodes, const int4 *__restrict__ cell, const TNode *tnode,
    const double *mass, const double *wgt, double *exps, unsigned *err) {
    __shared__ MergeShared<P> shared[UP_WARPS];
    __shared__ BinomRows<P> bt;
    fill_binom_rows<P>(bt);
    __syncthreads();
    MergeShared<P> &sh = shared[threadIdx.x >> 5];
    // (read once: parameters read on both sides of pdl_begin were copied to local memory)
    const int first = lo.off[l], mid = lo.off[l + 1], ninner = (lo.off[l + 2] - mid) / 4;
    int r = blockIdx.x * UP_WARPS + (threadIdx.x >> 5);
    MergeGeom g = {};
    if (r < ninner) merge_geom<P>(g, r, first, mid, nnodes, cell, tnode, mass, wgt, err);
    pdl_begin();   // the coefficients of the level below are complete from here on
    while (r < ninner) {
        if (g.ok) merge_node<P>(g, exps, bt, sh);
        r += gridDim.x * UP_WARPS;
        if (r < ninner) merge_geom<P>(g, r, first, mid, nnodes, cell, tnode, mass, wgt, err);
    }
}

// Wide levels, four threads per inner node (thread 4j + c shifts child c of the warp's j-th
// node): 8 inner nodes per warp.  The warp's 32 children are consecutive (children of inner
// node r are off[l+1] + 4r .. +3), so their coefficients are staged with coalesced loads; each
// thread then holds its own child's scaled coefficients in registers, forms that child's
// contribution to every coefficient of the parent with the binomial sums fully unrolled
// (uniform constant-bank operands), and the four contributions are added through shared
// memory.  A thread per node (all four children, the parent's coefficients accumulated in
// shared memory) held 250 registers and 38 KB of shared memory per warp, 5 warps per SM; this
// form holds 168 and 12.5 KB, 12 warps per SM.
constexpr int UP_WIDE_MIN_BLOCKS = 12;
template <int P>
struct WideShared {
    double c[32][2 * P + 1];   // row t: thread t's child coefficients, then its contribution
};

template <int P>
__global__ __launch_bounds__(32, UP_WIDE_MIN_BLOCKS) void k_upward_wide(
    int l, LevelOffsets lo, int nnodes, const int4 *__restrict__ cell, const TNode *tnode,
    const double *mass, const double *wgt, double *exps, unsigned *err) {
    pdl_begin();
    __shared__ WideShared<P> st;
    const int lane = lane_id(), j = lane >> 2, c = lane & 3;
    const int cbase = lo.off[l + 1];
    const int ninner = (lo.off[l + 2] - cbase) / 4;
    for (int r0 = blockIdx.x * 8; r0 < ninner; r0 += gridDim.x * 8) {
        const int r = r0 + j;
        const int cb = cbase + 4 * r;
        bool act = r < ninner;
        int parent = -1;
        if (act) {
            parent = cell[cb].w;
            if (parent < lo.off[l] || parent >= lo.off[l + 1] || cb + 4 > nnodes) {
                atomicOr(err, DEVERR_TREE);
                act = false;
            }
        }
        const int id = act ? cb + c : 0;
        const double m = mass[id], w = wgt[id];
        const double cx = tnode[id].xcom, cy = tnode[id].ycom;
        const double px = act ? tnode[parent].xcom : 0.0, py = act ? tnode[parent].ycom : 0.0;
        // the node's negligible children (its four threads' bits of the ballot)
        const unsigned negl = __ballot_sync(FULL_MASK, act && fabs(w) < 1.1e-16);
        const unsigned g = (negl >> (4 * j)) & 0xFu;
        const int zcount = __popc(g);
        const int nz = 31 - __clz((~g & 0xFu) | 1u);   // the last non-negligible child
        const bool shift = act && zcount <= 2;
        const bool copy = act && zcount == 3 && c == nz;
        // the warp's 32 children, coalesced (zeros past the level)
        __syncwarp();
        {
            const size_t first = (size_t)(cbase + 4 * r0) * 2 * P;
            const int nchild = min(32, 4 * (ninner - r0));
            for (int idx = lane; idx < 32 * 2 * P; idx += 32) {
                const int ch = idx / (2 * P), t = idx - ch * (2 * P);
                st.c[ch][t] = ch < nchild ? exps[first + idx] : 0.0;
            }
        }
        __syncwarp();
        // C_k = a_{k-1} z0^-k of this thread's child
        const double x0 = cx - px, y0 = cy - py;
        double cr[P], ci[P];
        {
            const double r2z0 = x0 * x0 + y0 * y0;
            const cplx zinv = shift ? cplx{x0 / r2z0, -y0 / r2z0} : cplx{0.0, 0.0};
            cplx zp = zinv;
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const cplx v = cmul({st.c[lane][k], st.c[lane][P + k]}, zp);
                cr[k] = v.re;
                ci[k] = v.im;
                zp = cmul(zp, zinv);
            }
        }
        // this child's part of parent coefficient L: z0^L (-m/L + sum_{k<=L} C(L-1, k-1) C_k)
        const cplx z0 = {x0, y0};
        cplx zl = z0;
#pragma unroll
        for (int L = 1; L <= P; ++L) {
            double tr = L == 1 ? -m : m * (-1.0 / L), ti = 0.0;
#pragma unroll
            for (int k = 1; k <= L; ++k) {
                const double b = c_binom_up.c[L - 1][k - 1];
                tr = fma(b, cr[k - 1], tr);
                ti = fma(b, ci[k - 1], ti);
            }
            const cplx o = cmul({tr, ti}, zl);
            zl = cmul(zl, z0);
            // three negligible children: the fourth's coefficients unshifted; four: zero
            const double a_re = st.c[lane][L - 1], a_im = st.c[lane][P + L - 1];
            st.c[lane][L - 1] = shift ? o.re : (copy ? a_re : 0.0);
            st.c[lane][P + L - 1] = shift ? o.im : (copy ? a_im : 0.0);
        }
        __syncwarp();
        // the parent's coefficients t = c, c + 4, ...: its four children's parts in order
        if (act)
            for (int t = c; t < 2 * P; t += 4)
                exps[(size_t)parent * 2 * P + t] =
                    ((st.c[4 * j][t] + st.c[4 * j + 1][t]) + st.c[4 * j + 2][t]) +
                    st.c[4 * j + 3][t];
    }
}

// Levels ltop .. 0 (deepest first) in one block; the block barrier between levels orders each
// level's writes before its parents' reads.
template <int P>
__global__ __launch_bounds__(UP_TOP_WARPS * 32) void k_upward_top(
    int ltop, LevelOffsets lo, int nnodes, const int4 *__restrict__ cell, const TNode *tnode,
    const double *mass, const double *wgt, double *exps, unsigned *err) {
    __shared__ MergeShared<P> shared[UP_TOP_WARPS];
    __shared__ BinomRows<P> bt;
    __shared__ int s_off[LMAX + 3];   // (as in k_upward_level: read before pdl_begin)
    if (threadIdx.x < LMAX + 3) s_off[threadIdx.x] = lo.off[threadIdx.x];
    fill_binom_rows<P>(bt);
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    MergeShared<P> &sh = shared[warp];
    for (int l = ltop; l >= 0; --l) {
        const int first = s_off[l], mid = s_off[l + 1], ninner = (s_off[l + 2] - mid) / 4;
        int r = warp;
        MergeGeom g = {};
        if (r < ninner) merge_geom<P>(g, r, first, mid, nnodes, cell, tnode, mass, wgt, err);
        // the coefficients below: of the kernel before this one, then of the block's own level
        if (l == ltop) pdl_begin();
        else __syncthreads();
        while (r < ninner) {
            if (g.ok) merge_node<P>(g, exps, bt, sh);
            r += UP_TOP_WARPS;
            if (r < ninner) merge_geom<P>(g, r, first, mid, nnodes, cell, tnode, mass, wgt, err);
        }
    }
}

static int sm_count_up() { return device_sm_count(); }

// Largest level ltop such that levels 0 .. ltop all have at most `limit` inner nodes (-1: none).
static int small_top(const Context &c, int limit) {
    int ltop = -1;
    while (ltop + 1 < LMAX && (c.level_off[ltop + 3] - c.level_off[ltop + 2]) / 4 <= limit) ++ltop;
    return ltop;
}

static LevelOffsets level_offsets(const Context &c) {
    LevelOffsets offs;
    for (int l = 0; l < LMAX + 3; ++l) offs.off[l] = c.level_off[l];
    return offs;
}


int upward_moments(Context &c) {
    const bool ovl = c.launch_overlap;   // launch_pdl chains (tc_set_launch_overlap)
    const int nn = c.nnodes;
    const int2 *range = slot_ptr<int2>(c, S_RANGE);
    const int4 *cell = slot_ptr<int4>(c, S_CELL);
    TNode *tnode = slot_ptr<TNode>(c, S_TNODE);
    const Frame *frame = slot_ptr<Frame>(c, S_FRAME);
    unsigned *err = c.ctrl.err;
    double *mass = slot_ptr<double>(c, S_MASS), *w = slot_ptr<double>(c, S_W),
           *wx = slot_ptr<double>(c, S_WX), *wy = slot_ptr<double>(c, S_WY);
    const bool quads = nn >= LS_QUAD_NODES;
    TC_CUDA_TRY(launch_pdl(ovl, quads ? k_leaf_setup : k_leaf_setup_warp,
                           quads ? (int)(((long long)nn * 4 + 255) / 256)
                                 : (nn + LS_WARPS - 1) / LS_WARPS,
                           quads ? 256 : LS_WARPS * 32, 0,
                           c.stream, nn, c.nsrc, c.leafcap,
                           (const double *)slot_ptr<double>(c, S_XS),
                           (const double *)slot_ptr<double>(c, S_YS),
                           (const double *)slot_ptr<double>(c, S_VS), range, cell, tnode, mass, w,
                           wx, wy, frame, err));
    TC_KERNEL_CHECK();
    // The parent moments run on the auxiliary stream, beside the leaves' P2E on the main one
    // (P2E reads only the leaves' own moments; the E2E waits for ev_moments, and anything
    // queued later on the auxiliary stream, such as the interaction lists, follows them).
    TC_CUDA_TRY(stream_after(c, c.aux, c.stream, c.ev_leafset));
    AuxScope on_aux(c);
    // inner nodes exist on levels 0 .. LMAX-1, deepest first
    const LevelOffsets offs = level_offsets(c);
    const int ltop = small_top(c, MOM_TOP_MAX);
    // the first launch follows the event wait (on one stream: the leaves' kernel); each later one
    // follows a kernel (launch_pdl)
    bool after_kernel = c.single;
    for (int l = LMAX - 1; l > ltop; --l) {
        const int ninner = (c.level_off[l + 2] - c.level_off[l + 1]) / 4;
        if (ninner <= 0) continue;
        if (after_kernel)
            TC_CUDA_TRY(launch_pdl(ovl, k_moments_level, (ninner + 255) / 256, 256, 0, c.stream, l,
                                   offs, nn, cell, tnode, mass, w, wx, wy, frame, err));
        else
            k_moments_level<<<(ninner + 255) / 256, 256, 0, c.stream>>>(l, offs, nn, cell, tnode,
                                                                        mass, w, wx, wy, frame,
                                                                        err);
        TC_KERNEL_CHECK();
        after_kernel = true;
    }
    if (ltop >= 0) {
        if (after_kernel)
            TC_CUDA_TRY(launch_pdl(ovl, k_moments_top, 1, MOM_TOP_MAX, 0, c.stream, ltop, offs, nn,
                                   cell, tnode, mass, w, wx, wy, frame, err));
        else
            k_moments_top<<<1, MOM_TOP_MAX, 0, c.stream>>>(ltop, offs, nn, cell, tnode, mass, w,
                                                           wx, wy, frame, err);
        TC_KERNEL_CHECK();
    }
    TC_CUDA_TRY(mark_event(c, c.ev_moments));
    return TC_OK;
}

template <int P>
static int run_expansions(Context &c) {
    const bool ovl = c.launch_overlap;   // launch_pdl chains (tc_set_launch_overlap)
    const int nn = c.nnodes;
    const double *xs = slot_ptr<double>(c, S_XS), *ys = slot_ptr<double>(c, S_YS),
                 *vs = slot_ptr<double>(c, S_VS);
    const int2 *range = slot_ptr<int2>(c, S_RANGE);
    const int4 *cell = slot_ptr<int4>(c, S_CELL);
    const TNode *tnode = slot_ptr<TNode>(c, S_TNODE);
    const Frame *frame = slot_ptr<Frame>(c, S_FRAME);
    unsigned *err = c.ctrl.err;
    const double *mass = slot_ptr<double>(c, S_MASS), *w = slot_ptr<double>(c, S_W);
    double *exps = slot_ptr<double>(c, S_EXPS);
    const int sms = sm_count_up();

    const bool mixed = c.precision == 1;
    const size_t smem = mixed ? leaf_bytes<P, true>() : leaf_bytes<P, false>();
    const int occ = mixed ? blocks_per_sm<k_leaf_p2e<P, true>>(UP_WARPS * 32, smem)
                          : blocks_per_sm<k_leaf_p2e<P, false>>(UP_WARPS * 32, smem);
    const int grid = (int)std::min<long long>((nn + UP_WARPS - 1) / UP_WARPS, (long long)sms * occ);
    auto p2e = mixed ? k_leaf_p2e<P, true> : k_leaf_p2e<P, false>;
    TC_CUDA_TRY(launch_pdl(ovl, p2e, grid, UP_WARPS * 32, smem, c.stream, nn, c.nsrc, c.leafcap,
                           xs, ys, vs, range, cell, tnode, exps, frame));
    TC_KERNEL_CHECK();
    // the parents' moments (expansion centres) come from the auxiliary stream
    TC_CUDA_TRY(await_event(c, c.ev_moments));
    // E2E deepest level first: wide levels thread per node, narrow ones warp per node, the
    // small top levels in one single-block launch
    const LevelOffsets offs = level_offsets(c);
    const int ltop = small_top(c, UP_TOP_MAX_NODES);
    // the first launch follows the event wait; each later one follows a kernel (launch_pdl)
    bool after_kernel = c.single;
    for (int l = LMAX - 1; l > ltop; --l) {
        const int ninner = (c.level_off[l + 2] - c.level_off[l + 1]) / 4;
        if (ninner <= 0) continue;
        if (ninner >= UP_WIDE_MIN_NODES) {
            const int g = (int)std::min<long long>((ninner + 7) / 8,
                                                   (long long)sms * UP_WIDE_MIN_BLOCKS);
            if (after_kernel)
                TC_CUDA_TRY(launch_pdl(ovl, k_upward_wide<P>, g, 32, 0, c.stream, l, offs, nn, cell,
                                       (const TNode *)tnode, mass, w, exps, err));
            else
                k_upward_wide<P><<<g, 32, 0, c.stream>>>(l, offs, nn, cell, tnode, mass, w, exps,
                                                         err);
        } else {
            const int g = (int)std::min<long long>((ninner + UP_WARPS - 1) / UP_WARPS, (long long)sms * 8);
            if (after_kernel)
                TC_CUDA_TRY(launch_pdl(ovl, k_upward_level<P>, g, UP_WARPS * 32, 0, c.stream, l,
                                       offs, nn, cell, (const TNode *)tnode, mass, w, exps, err));
            else
                k_upward_level<P><<<g, UP_WARPS * 32, 0, c.stream>>>(l, offs, nn, cell, tnode, mass,
                                                                     w, exps, err);
        }
        TC_KERNEL_CHECK();
        after_kernel = true;
    }
    if (ltop >= 0) {
        if (after_kernel)
            TC_CUDA_TRY(launch_pdl(ovl, k_upward_top<P>, 1, UP_TOP_WARPS * 32, 0, c.stream, ltop,
                                   offs, nn, cell, (const TNode *)tnode, mass, w, exps, err));
        else
            k_upward_top<P><<<1, UP_TOP_WARPS * 32, 0, c.stream>>>(ltop, offs, nn, cell, tnode,
                                                                   mass, w, exps, err);
        TC_KERNEL_CHECK();
    }
    return TC_OK;
}

int upward_prepare(Context &c, int order) {
    // an order without kernel instances is refused here, before any work
    int rc = dispatch_order(order, [](auto) -> int { return TC_OK; });
    if (rc) return rc;
    const int nn = c.nnodes;
    double *mass, *w, *wx, *wy, *exps;
    if ((rc = ensure(c, S_MASS, nn, &mass)) || (rc = ensure(c, S_W, nn, &w)) ||
        (rc = ensure(c, S_WX, nn, &wx)) || (rc = ensure(c, S_WY, nn, &wy)) ||
        (rc = ensure(c, S_EXPS, (size_t)nn * 2 * order, &exps)))
        return rc;
    c.order = order;
    return TC_OK;
}

int upward_expansions(Context &c) {
    return dispatch_order(c.order,
                          [&](auto p) -> int { return run_expansions<decltype(p)::value>(c); });
}

int upward_pass(Context &c, int order) {
    int rc;
    if ((rc = upward_prepare(c, order)) || (rc = upward_moments(c)) || (rc = upward_expansions(c)))
        return rc;
    return TC_OK;
}

int prepare_upward() {
    int rc;
#define TC_LEAF_SHARED(P)                                                                         \
    if ((rc = allow_shared((const void *)k_leaf_p2e<P, true>, leaf_bytes<P, true>())) ||          \
        (rc = allow_shared((const void *)k_leaf_p2e<P, false>, leaf_bytes<P, false>())))          \
        return rc;
    TC_FOR_EACH_ORDER(TC_LEAF_SHARED)
#undef TC_LEAF_SHARED
    return TC_OK;
}

void kernels_upward(KernelList &v) {
    v.insert(v.end(), {(const void *)k_leaf_setup, (const void *)k_leaf_setup_warp, (const void *)k_moments_level,
                       (const void *)k_moments_top});
#define TC_UPWARD_KERNELS(P)                                                                     \
    v.insert(v.end(), {(const void *)k_leaf_p2e<P, true>, (const void *)k_leaf_p2e<P, false>,    \
                       (const void *)k_upward_level<P>, (const void *)k_upward_wide<P>,           \
                       (const void *)k_upward_top<P>});
    TC_FOR_EACH_ORDER(TC_UPWARD_KERNELS)
#undef TC_UPWARD_KERNELS
}

}  // namespace tc
