// potential.cu -- treecode_potential on the GPU.
//
// Restates drivers/treecode-potential.cpp:25-87 (per-target traversal) and
// kernels/potential-kernels.m4 (P2P, E2P).  The opening test is per target
// (r^2 < theta^2 |t - com|^2, treecode-potential.cpp:48-50), so the warp-cooperative traversal
// keeps, for every stack entry, the mask of lanes (targets) that still need the node:
//   far  = lanes in the mask that accept the node            -> E2P entry (node, far)
//   rest = mask & ~far; leaf -> P2P entry (node, rest); inner -> push children with `rest`.
// Each target therefore sees exactly the nodes the reference's own DFS would give it.
// Targets are first sorted by Morton key (in the sources' frame) so that the 32 targets of a
// warp are neighbours and the masks are mostly full.
//
// Lists are (node, lane mask) pairs in CSR form per group of 32 targets: one walk writes them into
// per-warp scratch runs, a scan and a copy put them in order (a second walk fills them where a
// run outgrew its region).
#include <cfloat>
#include <cmath>

#include "tc_internal.h"
#include "tc_math.cuh"

namespace tc {

constexpr int PT_WARPS = 4;
// A group's near field is cut into segments of PT_SEG sources, so that groups inside dense
// clusters do not serialise the kernel.  The segments also fix the grid of source tiles (a
// segment's tiles start at its own start, at a leaf's start, or 32 sources after another), and
// with it how the mixed form's FP32 sums are grouped.
constexpr int PT_SEG = 4096;
// With few groups a segment is cut further, at tile starts, into tasks of `seg` sources (a
// divisor of PT_SEG), and the far field becomes a task of its own.
constexpr int PT_MIN_SEG = 64;
constexpr int PT_FULL_GROUPS = 16384;

// Near-field sources per evaluation task.  The kernel holds about 2400 resident warps; with whole
// segments, fewer than ~16K groups leave most of them idle or waiting for the longest task.
// FP64, sources = targets, theta 0.5, the evaluation kernel with whole segments and with this
// rule: 4096 (128 groups, seg 64) 152 -> 23 us, 65,536 (2048 groups, seg 512) 307 -> 208 us;
// at 131,072 groups the tasks balance without cutting.  The mixed form keeps whole segments: its
// compensated FP32 sum runs over a segment, and cutting it moves results by 1e-9.
static int task_segment(int ngroups, bool mixed) {
    int seg = PT_SEG;
    while (!mixed && seg > PT_MIN_SEG &&
           (long long)ngroups * PT_SEG < (long long)PT_FULL_GROUPS * seg)
        seg >>= 1;
    return seg;
}

// Lists of one group of 32 targets.  The warp pops up to 32 stack entries (node, target mask)
// at a time, one per lane, so the latency of the node reads is shared by a whole batch.  A lane
// decides its node for the entry's targets with the group's bounding box first: when every
// point of the box is clearly far (or clearly near) -- with a relative margin of 1e-12, far
// above the rounding of the per-target test -- the whole mask follows; otherwise the exact
// per-target test (r^2 < theta^2 |t - com|^2, treecode-potential.cpp:48-50) runs for each
// target of the mask, one target per lane, node after node.  The walk is bound by its issue slots:
// with a lane looping over its own node's targets the 4M mixture's lists took 0.95 ms, so 0.55.
// Far targets give an E2P entry (node, far); the rest give a P2P entry for
// a leaf or push the node's four children with the rest.  Every target thus gets exactly the
// nodes its own depth-first traversal in the reference would give it.  Entries are written in
// the (deterministic) processing order; the count pass and the fill pass take the same steps.
// Stack entries per warp.  A batch of nb entries pushes at most 4 nb, so batches are taken only
// while top <= PL_STACK - 160; above that the walk pops one entry at a time (depth first), which
// grows the stack by at most 3 per level, 45 in all, before it shrinks again.  The stack thus
// never holds more than PL_STACK - 160 + 96 + 45 entries.
constexpr int PL_STACK = 512;

// Many FP64 targets: PS_GROUPS consecutive groups (128 targets) first walk the tree together.  A
// node that every target of their box accepts, far enough from the box (below), becomes an entry
// of their common far list, evaluated for all of them at once through a local expansion about the
// box's centre (k_potential_locals); a node that every target rejects is opened; all others, the
// ones near the border and the leaves nearby, are handed on to the groups' own walks as their
// starting nodes.  Every target still gets exactly the nodes of its own traversal.
// An entry's local expansion replaces 4 x ~220 issue slots of E2P by ~110 of translation; about
// 65% of the entries of 4M clustered targets (theta 0.5) become common.  Evaluation of 4M sources
// and targets 14.2 -> 12.0 ms, lists 0.55 -> 0.42 ms; 500K targets, theta 0.3, 3.02 -> 2.74 ms; at
// 131,071 targets (4096 groups) the sets' chains of cells take what they save (631 and 644 us).
// Lists have room for PS_LIST entries each; a common node that does not fit is handed on, and a
// set whose handed-on list overflows falls back to the root.
constexpr int PS_GROUPS = 4;
constexpr int PS_LIST = 192;
constexpr int PS_TERMS = 32;   // terms of a local expansion, one per lane
constexpr int PS_MIN_GROUPS = 8192;
struct SuperSets {
    const int *common, *ncommon;   // PS_LIST per set
    const int *start, *nstart;     // null: no sets, every group starts at the root
    const double4 *geo;            // centre x, y, half diagonal (the expansions' scale)
};

// The far field's truncated multipole is expanded in powers of (target offset / distance); rho
// bounds that ratio so that what PS_TERMS terms leave out stays below 1e-17 of a cell's weight,
// under the rounding of the sum: with |a_{k-1} z^-k| <= theta^k / k,
//   rho^q / q + sum_k theta^k / k C(q + k - 1, k - 1) rho^q / (1 - rho (q + k) / (q + 1)).
// (theta 0.5, order 12: rho 0.19.)  0: no common entries.  Some hundred pow calls.
static double super_rho(double theta, int order) {
    if (!(theta > 0 && theta <= 1)) return 0.0;
    constexpr int q = PS_TERMS;
    for (double rho = 0.3; rho > 0.04; rho -= 0.01) {
        const double rq = std::pow(rho, q);
        double bound = rq / q, binom = 1.0;   // C(q + k - 1, k - 1)
        for (int k = 1; k <= order; ++k) {
            const double left = 1.0 - rho * (q + k) / (q + 1);
            bound += left > 0.1 ? std::pow(theta, k) / k * binom * rq / left : 1.0;
            binom *= (double)(q + k) / k;
        }
        if (bound <= 1e-17) return rho;
    }
    return 0.0;
}

__global__ __launch_bounds__(PT_WARPS * 32) void k_potential_supers(
    int nsets, int m, const double *__restrict__ xt, const double *__restrict__ yt,
    const int *__restrict__ tperm, double theta, double rho, const TNode *__restrict__ tnode,
    int nnodes, int *__restrict__ common, int *__restrict__ ncommon, int *__restrict__ start,
    int *__restrict__ nstart, double4 *__restrict__ geo, unsigned *err,
    unsigned long long *stats) {
    pdl_begin();
    __shared__ int stack_all[PT_WARPS][PL_STACK];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    int *stack = stack_all[warp];
    const unsigned lt = lanemask_lt();
    const double theta2 = theta * theta, rho2 = rho * rho;
    unsigned long long cells = 0;
    for (int g = blockIdx.x * PT_WARPS + warp; g < nsets; g += gridDim.x * PT_WARPS) {
        double bxlo = 1e300, bxhi = -1e300, bylo = 1e300, byhi = -1e300;
        const int t0 = g * PS_GROUPS * 32, cnt = min(PS_GROUPS * 32, m - t0);
        bool finite = true;
        for (int q = lane; q < cnt; q += 32) {
            const int j = tperm[t0 + q];
            const double x = xt[j], y = yt[j];
            finite = finite && fabs(x) < 1e300 && fabs(y) < 1e300;
            bxlo = fmin(bxlo, x);
            bxhi = fmax(bxhi, x);
            bylo = fmin(bylo, y);
            byhi = fmax(byhi, y);
        }
        for (int o = 16; o; o >>= 1) {
            bxlo = fmin(bxlo, __shfl_xor_sync(FULL_MASK, bxlo, o));
            bxhi = fmax(bxhi, __shfl_xor_sync(FULL_MASK, bxhi, o));
            bylo = fmin(bylo, __shfl_xor_sync(FULL_MASK, bylo, o));
            byhi = fmax(byhi, __shfl_xor_sync(FULL_MASK, byhi, o));
        }
        finite = __all_sync(FULL_MASK, finite);
        const double cx = 0.5 * (bxlo + bxhi), cy = 0.5 * (bylo + byhi);
        const double hx = 0.5 * (bxhi - bxlo), hy = 0.5 * (byhi - bylo);
        const double half2 = hx * hx + hy * hy, half = sqrt(half2) * (1.0 + 1e-12);
        // a set of one point, or spread so that the scale's powers leave the number range, has no
        // expansion
        const bool expand = finite && half > 1e-10 && half < 1e10;
        int *com = common + (size_t)g * PS_LIST, *st = start + (size_t)g * PS_LIST;
        int nc = 0, ns = 0, top = 1;
        bool plain = !finite;
        __syncwarp();
        if (lane == 0) stack[0] = 0;
        __syncwarp();
        while (top > 0 && !plain) {
            const int nb = top > PL_STACK - 160 ? 1 : min(32, top), base = top - nb;
            int node = -1;
            if (lane < nb) node = stack[base + lane];
            __syncwarp();
            top = base;
            bool ok = lane < nb;
            if (ok && (unsigned)node >= (unsigned)nnodes) {
                atomicOr(err, DEVERR_BOUNDS);
                ok = false;
            }
            TNode nd = {};
            bool far = false, near = false, open = false;
            if (ok) {
                nd = tnode[node];
                const double rr = __dmul_rn(nd.r, nd.r);
                const double ex = fmax(fmax(bxlo - nd.xcom, nd.xcom - bxhi), 0.0);
                const double ey = fmax(fmax(bylo - nd.ycom, nd.ycom - byhi), 0.0);
                const double fx = fmax(nd.xcom - bxlo, bxhi - nd.xcom);
                const double fy = fmax(nd.ycom - bylo, byhi - nd.ycom);
                const double dmin2 = ex * ex + ey * ey, dmax2 = fx * fx + fy * fy;
                const double dx = nd.xcom - cx, dy = nd.ycom - cy;
                far = rr < theta2 * dmin2 * (1.0 - 1e-12) && expand &&
                      half2 <= rho2 * (dx * dx + dy * dy) * (1.0 - 1e-12);
                near = !far && rr >= theta2 * dmax2 * (1.0 + 1e-12);
                open = near && nd.child > node && nd.child + 4 <= nnodes;
            }
            const unsigned bc = __ballot_sync(FULL_MASK, far);
            const bool fits = far && nc + __popc(bc & lt) < PS_LIST;
            if (fits) com[nc + __popc(bc & lt)] = node;
            nc = min(nc + __popc(bc), PS_LIST);
            const bool hand = ok && !fits && !open;
            const unsigned bh = __ballot_sync(FULL_MASK, hand);
            const unsigned bo = __ballot_sync(FULL_MASK, open);
            if (ns + __popc(bh) > PS_LIST || top + 4 * __popc(bo) > PL_STACK) {
                plain = true;
                break;
            }
            if (hand) st[ns + __popc(bh & lt)] = node;
            ns += __popc(bh);
            if (open) {
                const int at = top + 4 * __popc(bo & lt);
#pragma unroll
                for (int c = 0; c < 4; ++c) stack[at + c] = nd.child + c;
            }
            top += 4 * __popc(bo);
            __syncwarp();
        }
        if (plain) {
            nc = 0;
            ns = 1;
            if (lane == 0) st[0] = 0;
        }
        if (lane == 0) {
            ncommon[g] = nc;
            nstart[g] = ns;
            // (without an expansion its coefficients are 0; a frame in which every finite target
            // has a finite offset)
            geo[g] = expand ? make_double4(cx, cy, half, 0.0) : make_double4(0.0, 0.0, 1.0, 0.0);
        }
        cells += nc;
        __syncwarp();
    }
    if (lane == 0 && cells) atomicAdd(&stats[STAT_SET_CELLS], cells);
}

// The local expansion of every set from its common far list, about the set's centre c with scale
// R, lane l forming coefficient L_l R^l:
//   m log|t - com| + Re sum_k a_{k-1} (t - com)^-k = Re sum_l L_l (t - c)^l,  z0 = com - c,
//   L_0 = m log|z0| + sum_k C_k,  L_l = z0^-l (-m / l + sum_k C(l+k-1, k-1) C_k),
//   C_k = (-1)^k a_{k-1} z0^-k.
// Cells in batches, two lanes forming the odd and the even powers (R / z0)^l of each.
constexpr int PS_BATCH = 16;
template <int P>
struct LocalShared {
    cplx pow[PS_BATCH][PS_TERMS + 1];   // (R / z0)^l, l = 1.. at l - 1 (odd row length: banks)
    cplx coef[P];                       // C_k
    double mass[PS_BATCH], log[PS_BATCH];
};
constexpr int PLOC_WARPS = 4;
__device__ const BinomTable g_binom_p = make_binom_table();   // per-lane indices

template <int P>
__global__ __launch_bounds__(PLOC_WARPS * 32) void k_potential_locals(
    int nsets, SuperSets sets, const TNode *__restrict__ tnode, const double *__restrict__ mass,
    const double *__restrict__ exps, cplx *__restrict__ local) {
    __shared__ LocalShared<P> shared[PLOC_WARPS];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    LocalShared<P> &sh = shared[warp];
    double bin[P];   // C(l + k - 1, k - 1), k = 1..P, l = lane
#pragma unroll
    for (int k = 1; k <= P; ++k) bin[k - 1] = g_binom_p.c[lane + k - 1][k - 1];
    const double minv = lane ? -1.0 / lane : 0.0;
    const int c = lane & (PS_BATCH - 1), half = lane / PS_BATCH;
    for (int g = blockIdx.x * PLOC_WARPS + warp; g < nsets; g += gridDim.x * PLOC_WARPS) {
        const int n = sets.ncommon[g];
        const int *com = sets.common + (size_t)g * PS_LIST;
        const double4 geo = sets.geo[g];
        const double R = geo.z;
        // a_{k-1} z0^-k from the scaled powers: lane k - 1 keeps (-1)^k R^-k
        const cplx ir = cpow_int({-1.0 / R, 0.0}, lane < P ? lane + 1 : 1);
        const double unscale = ir.re;
        cplx L = {0.0, 0.0};
        for (int b0 = 0; b0 < n; b0 += PS_BATCH) {
            const int nb = min(PS_BATCH, n - b0);
            const int mine = com[b0 + min(c, nb - 1)];
            const TNode nd = tnode[mine];
            const double zx = nd.xcom - geo.x, zy = nd.ycom - geo.y;
            const double r2 = zx * zx + zy * zy;
            // (where the square nears or passes the top of the number range, R / z0 < 1e-140 counts
            // for nothing, and the logarithm of an overflow is that of the top)
            const double iz = r2 < 1e300 ? R * rcp_nr(r2) : 0.0;
            const cplx u = {zx * iz, -zy * iz};
            const cplx u2 = cmul(u, u);
            cplx p = half ? u2 : u;
            __syncwarp();
            if (half) {
                sh.mass[c] = mass[mine];
                sh.log[c] = 0.5 * log(fmin(r2, DBL_MAX));
            }
#pragma unroll
            for (int q = 0; q < PS_TERMS / 2; ++q) {
                sh.pow[c][2 * q + half] = p;
                p = cmul(p, u2);
            }
            __syncwarp();
            double ar = 0, ai = 0;
            auto fetch = [&](int node) {
                if (lane < P) {
                    const double *ex = exps + (size_t)node * 2 * P;
                    ar = ex[lane];
                    ai = ex[P + lane];
                }
            };
            fetch(__shfl_sync(FULL_MASK, mine, 0));
            for (int k0 = 0; k0 < nb; ++k0) {
                const cplx a = {ar * unscale, ai * unscale};
                if (k0 + 1 < nb) fetch(__shfl_sync(FULL_MASK, mine, k0 + 1));
                const double mm = sh.mass[k0];
                if (lane < P) sh.coef[lane] = cmul(a, sh.pow[k0][lane]);
                const cplx w = lane ? sh.pow[k0][lane - 1] : cplx{1.0, 0.0};
                __syncwarp();
                double tr = lane ? mm * minv : mm * sh.log[k0], ti = 0.0;
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    const cplx ck = sh.coef[k];
                    tr = fma(bin[k], ck.re, tr);
                    ti = fma(bin[k], ck.im, ti);
                }
                L = cfma({tr, ti}, w, L);
                __syncwarp();
            }
        }
        local[(size_t)g * PS_TERMS + lane] = L;
        __syncwarp();
    }
}

// MODE 1: write the lists at the scanned offsets (CSR); MODE 2: count them and write each
// warp's entries into its own scratch region (ScratchLayout), recording where each group's run
// starts, so that a copy into CSR order replaces a second walk.  A region that fills up sets
// meta[0] (the host then falls back to MODE 1); meta[1 + k] receives the longest run of kind
// k any warp wrote, and the work counters are added.  (meta[META_WIDE] is the target sort's.)
template <int MODE>
__global__ __launch_bounds__(PT_WARPS * 32) void k_potential_lists(
    int ngroups, int m, const double *__restrict__ xt, const double *__restrict__ yt,
    const int *__restrict__ tperm, double theta, const TNode *__restrict__ tnode, int nnodes,
    int *__restrict__ counts, const int *__restrict__ offs, int2 *__restrict__ lists,
    int2 *__restrict__ scratch, ScratchLayout sl, int *__restrict__ sstart, int *meta,
    unsigned *err, unsigned long long *stats, int seg, SuperSets sets) {
    pdl_begin();
    constexpr bool FILL = MODE == 1;
    const int wglob = blockIdx.x * PT_WARPS + (threadIdx.x >> 5);
    int cur[2] = {0, 0};   // MODE 2: entries this warp has written, per kind
    bool full = false;
    __shared__ int2 stack_all[PT_WARPS][PL_STACK];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    int2 *stack = stack_all[warp];
    const unsigned lt = (1u << lane) - 1u;
    const double theta2 = theta * theta;
    unsigned long long e2p_pairs = 0, p2p_pairs = 0;   // warp-uniform work counters

    for (int g = blockIdx.x * PT_WARPS + warp; g < ngroups; g += gridDim.x * PT_WARPS) {
        const int t = g * 32 + lane;
        const bool valid = t < m;
        double x = 0, y = 0;
        if (valid) {
            const int j = tperm[t];
            x = xt[j];
            y = yt[j];
        }
        const unsigned vmask = __ballot_sync(FULL_MASK, valid);
        // bounding box of the group's targets
        double bxlo = valid ? x : 1e300, bxhi = valid ? x : -1e300;
        double bylo = valid ? y : 1e300, byhi = valid ? y : -1e300;
        for (int o = 16; o; o >>= 1) {
            bxlo = fmin(bxlo, __shfl_xor_sync(FULL_MASK, bxlo, o));
            bxhi = fmax(bxhi, __shfl_xor_sync(FULL_MASK, bxhi, o));
            bylo = fmin(bylo, __shfl_xor_sync(FULL_MASK, bylo, o));
            byhi = fmax(byhi, __shfl_xor_sync(FULL_MASK, byhi, o));
        }
        int o0 = 0, o1 = 0, l0 = 0, l1 = 0;
        if (FILL) {
            o0 = offs[g];
            l0 = offs[g + 1];
            o1 = offs[ngroups + g];
            l1 = offs[ngroups + g + 1];
        }
        __syncwarp();
        // the walk starts at the root, or at the nodes its set handed on, a batch whenever the
        // stack is empty
        const int *start = nullptr;
        int left = 0;
        if (sets.nstart) {
            start = sets.start + (size_t)(g / PS_GROUPS) * PS_LIST;
            left = sets.nstart[g / PS_GROUPS];
        } else if (lane == 0) {
            stack[0] = make_int2(0, (int)vmask);
        }
        __syncwarp();
        int n0 = 0, n1 = 0, gsrc = 0, top = sets.nstart ? 0 : 1;
        bool overflow = false;
        while ((top > 0 || left > 0) && !overflow) {
            int2 ent = make_int2(0, 0);
            bool act;
            if (top > 0) {
                const int nb = top > PL_STACK - 160 ? 1 : min(32, top), base = top - nb;
                act = lane < nb;
                if (act) ent = stack[base + lane];
                __syncwarp();
                top = base;
            } else {
                const int nb = min(32, left);
                act = lane < nb;
                if (act) ent = make_int2(start[lane], (int)vmask);
                start += nb;
                left -= nb;
            }
            const unsigned mask = (unsigned)ent.y;
            bool ok = act && mask != 0;
            if (act && (unsigned)ent.x >= (unsigned)nnodes) {
                atomicOr(err, DEVERR_BOUNDS);
                ok = false;
            }
            TNode nd = {};
            if (ok) nd = tnode[ent.x];
            unsigned far = 0;
            bool unsure = false;
            const double rr = __dmul_rn(nd.r, nd.r);
            if (ok) {
                const double ex = fmax(fmax(bxlo - nd.xcom, nd.xcom - bxhi), 0.0);
                const double ey = fmax(fmax(bylo - nd.ycom, nd.ycom - byhi), 0.0);
                const double fx = fmax(nd.xcom - bxlo, bxhi - nd.xcom);
                const double fy = fmax(nd.ycom - bylo, byhi - nd.ycom);
                const double dmin2 = ex * ex + ey * ey, dmax2 = fx * fx + fy * fy;
                if (rr < theta2 * dmin2 * (1.0 - 1e-12)) {
                    far = mask;                         // every target of the box is far
                } else if (rr >= theta2 * dmax2 * (1.0 + 1e-12)) {
                    far = 0;                            // every target of the box is near
                } else {
                    unsure = true;
                }
            }
            // The nodes that the box leaves open, one after another, every lane testing its own
            // target (r2 without contraction, as the compiled reference): ~15 instructions a node,
            // where a lane looping over its node's targets held up the batch for ~250.
            for (unsigned open = __ballot_sync(FULL_MASK, unsure); open; open &= open - 1) {
                const int src = __ffs(open) - 1;
                const double cx = __shfl_sync(FULL_MASK, nd.xcom, src);
                const double cy = __shfl_sync(FULL_MASK, nd.ycom, src);
                const double nr = __shfl_sync(FULL_MASK, rr, src);
                const double dx = __dsub_rn(x, cx), dy = __dsub_rn(y, cy);
                const double r2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
                const unsigned acc = __ballot_sync(FULL_MASK, nr < __dmul_rn(theta2, r2));
                if (lane == src) far = acc & mask;
            }
            const unsigned rest = mask & ~far;
            const bool leaf = nd.child < 0;
            const bool f_far = ok && far != 0;
            const bool f_near = ok && rest != 0 && leaf && nd.count > 0;
            bool f_push = ok && rest != 0 && !leaf;
            if (f_push && (nd.child <= ent.x || nd.child + 4 > nnodes)) {
                atomicOr(err, DEVERR_BOUNDS);
                f_push = false;
            }
            const unsigned bf = __ballot_sync(FULL_MASK, f_far);
            const unsigned bn = __ballot_sync(FULL_MASK, f_near);
            const unsigned bp = __ballot_sync(FULL_MASK, f_push);
            if (FILL) {
                if (f_far) {
                    const int at = o0 + n0 + __popc(bf & lt);
                    if (at < l0) lists[at] = make_int2(ent.x, (int)far);
                    else atomicOr(err, DEVERR_BOUNDS);
                }
                if (f_near) {
                    const int at = o1 + n1 + __popc(bn & lt);
                    if (at < l1) lists[at] = make_int2(ent.x, (int)rest);
                    else atomicOr(err, DEVERR_BOUNDS);
                }
            }
            if (MODE == 2) {
                if (f_far) {
                    const int at = cur[0] + n0 + __popc(bf & lt);
                    if (at < sl.cap[0])
                        scratch[sl.koff[0] + (size_t)wglob * sl.cap[0] + at] =
                            make_int2(ent.x, (int)far);
                    else full = true;
                }
                if (f_near) {
                    const int at = cur[1] + n1 + __popc(bn & lt);
                    if (at < sl.cap[1])
                        scratch[sl.koff[1] + (size_t)wglob * sl.cap[1] + at] =
                            make_int2(ent.x, (int)rest);
                    else full = true;
                }
            }
            n0 += __popc(bf);
            n1 += __popc(bn);
            e2p_pairs += (unsigned)__reduce_add_sync(FULL_MASK, f_far ? __popc(far) : 0);
            const unsigned cnt = f_near ? (unsigned)nd.count : 0u;
            gsrc += (int)__reduce_add_sync(FULL_MASK, cnt);
            p2p_pairs += __reduce_add_sync(FULL_MASK, f_near ? (unsigned)__popc(rest) * cnt : 0u);
            const int npush = 4 * __popc(bp);
            if (top + npush > PL_STACK) {
                if (lane == 0) atomicOr(err, DEVERR_STACK);
                overflow = true;
            } else {
                if (f_push) {
                    const int at = top + 4 * __popc(bp & lt);
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        stack[at + c] = make_int2(nd.child + 3 - c, (int)rest);
                }
                top += npush;
            }
            __syncwarp();
        }
        if (!FILL && lane == 0) {
            counts[g] = n0;
            counts[ngroups + g] = n1;
            // evaluation tasks: the group's near-field sources in runs of `seg`; below PT_SEG
            // the far field is a task of its own
            counts[2 * ngroups + g] =
                max(1, (gsrc + seg - 1) / seg + (seg < PT_SEG && n0 > 0 ? 1 : 0));
            if (MODE == 2) {
                sstart[g] = sl.koff[0] + wglob * sl.cap[0] + cur[0];
                sstart[ngroups + g] = sl.koff[1] + wglob * sl.cap[1] + cur[1];
                sstart[2 * ngroups + g] = gsrc;   // (for put_task)
            }
        }
        if (MODE == 2) {
            cur[0] += n0;
            cur[1] += n1;
        }
        __syncwarp();
    }
    if (MODE == 2) {
        if (__any_sync(FULL_MASK, full) && lane == 0) atomicOr(&meta[0], 1);
        if (lane == 0) {
            atomicMax(&meta[1], cur[0]);
            atomicMax(&meta[2], cur[1]);
        }
    }
    if (MODE == 2 && stats && lane == 0) {
        if (e2p_pairs) atomicAdd(&stats[STAT_E2P_PAIRS], e2p_pairs);
        if (p2p_pairs) atomicAdd(&stats[STAT_P2P_PAIRS], p2p_pairs);
    }
}

// Few groups (up to PT_LPT_GROUPS): tasks in bins of falling work, the longest first (TaskBins), so
// that no long one is left for the end: mixed solves of 700,001 targets 1569 -> 1517 us, FP64 ones
// of 131,072 905 -> 881 us, 1,048,576 (theta 0.3) 3221 -> 3157 us.  The tail is a smaller share of
// more groups, while the table takes 64 bytes a task: 32,768 groups FP64 3295 -> 3200 us, mixed 1997 ->
// 1946; 65,536 groups 5681 -> 5630 (1%) and 3490 -> 3491.
constexpr int PT_LPT_GROUPS = 32768;

// Where the evaluation's tasks go: entry (task, group) t at t, or (stride > 0) in its bin.
struct TaskTable {
    int2 *entry;
    int stride;
    int *fill;
    const int *near_sources;   // per group
    int seg;
};

// Puts task t (the p-th of group g's) in the table.
__device__ __forceinline__ void put_task(const TaskTable &tt, int t, int p, int g, int nfar) {
    if (tt.stride == 0) {
        tt.entry[t] = make_int2(t, g);
        return;
    }
    // work: near-field sources, and three for a far-field cell
    const int np = tt.seg < PT_SEG && nfar > 0 ? p - 1 : p;
    int work = p == 0 ? 3 * nfar : 0;
    if (np >= 0) work += max(0, min(tt.seg, tt.near_sources[g] - np * tt.seg));
    const int bin = TASK_BINS - 1 - min(TASK_BINS - 1, (int)((long long)work * TASK_BINS / tt.seg));
    const int at = atomicAdd(&tt.fill[bin], 1);
    if (at < tt.stride) tt.entry[(size_t)bin * tt.stride + at] = make_int2(t, g);
}

// The lists in CSR order from the scratch runs of k_potential_lists<2>, and the task -> group
// map: warp per group.
__global__ __launch_bounds__(256) void k_potential_lists_copy(int ngroups,
                                                              const int *__restrict__ counts,
                                                              const int *__restrict__ offs,
                                                              const int *__restrict__ sstart,
                                                              const int2 *__restrict__ scratch,
                                                              int2 *__restrict__ lists,
                                                              TaskTable tt) {
    pdl_begin();
    const int lane = lane_id();
    const int *toff = offs + 2 * ngroups;
    const int tbase = toff[0];
    for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups;
         g += (gridDim.x * blockDim.x) >> 5) {
        for (int k = 0; k < 2; ++k) {
            const int n = counts[k * ngroups + g];
            const int2 *src = scratch + sstart[k * ngroups + g];
            int2 *dst = lists + offs[k * ngroups + g];
            for (int i = lane; i < n; i += 32) dst[i] = src[i];
        }
        for (int t = toff[g] + lane; t < toff[g + 1]; t += 32)
            put_task(tt, t - tbase, t - toff[g], g, counts[g]);
    }
}

constexpr int PE_WARPS = 4;
constexpr int PE_CHUNK = 32;

__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void two_sum_add(float &hi, float &lo, float x) {
    const float s = hi + x;
    const float bb = s - hi;
    lo += (hi - (s - bb)) + (x - bb);
    hi = s;
}

// The same with x = t l, in the roundings that the mixed evaluation is pinned to: MUL_ADD takes the
// product into the first sum and into the remainder unrounded (the sparse tiles), otherwise it
// is rounded first (the dense ones).  Left to the compiler, the choice changed with unrelated
// code around it and moved results by 1e-9.
template <bool MUL_ADD>
__device__ __forceinline__ void two_sum_mul(float &hi, float &lo, float t, float l) {
    const float x = __fmul_rn(t, l);
    const float s = MUL_ADD ? __fmaf_rn(t, l, hi) : __fadd_rn(hi, x);
    const float bb = __fsub_rn(s, hi);
    const float e = MUL_ADD ? __fmaf_rn(t, l, -bb) : __fsub_rn(x, bb);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), e));
    hi = s;
}

__device__ __forceinline__ void split2(double v, float &hi, float &lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

// Tasks: group g owns tasks [toff[g], toff[g+1]); task 0 evaluates the far field and the first
// PT_SEG near-field sources of the group, task p > 0 the p-th segment.
// The mixed form: the series of E2P and the P2P logs in FP32 (offsets from the group's first
// target split hi + lo, lg2.approx, compensated sums); the monopole term m log|z| of E2P stays
// FP64.
template <int P>
__global__ __launch_bounds__(PE_WARPS * 32) void k_potential_eval_mixed(
    int ngroups, int m, const double *__restrict__ xt, const double *__restrict__ yt,
    const int *__restrict__ tperm, const TNode *__restrict__ tnode,
    const double *__restrict__ mass, const int2 *__restrict__ range, const double *__restrict__ xs,
    const double *__restrict__ ys, const double *__restrict__ vs,
    const int *__restrict__ offs, const int2 *__restrict__ lists, double *__restrict__ out,
    double *__restrict__ partial, int *task_ctr, TaskTable tt,
    const float2 *__restrict__ sexp, const float *__restrict__ sscale) {
    pdl_begin();
    // E2P coefficients in pairs (D_2j.re, D_2j+1.re, D_2j.im, D_2j+1.im): the even and
    // the odd series run side by side in f32x2 lanes
    __shared__ float4 s_coef32[PE_WARPS][P / 2];
    // the tile as negated float offsets (hi + lo) from the group's reference point,
    // two sources per entry for paired-FP32 (f32x2) arithmetic: (-x hi, -x hi', -x lo, -x lo'),
    // the same for y, and (v, v')
    __shared__ float4 s_nx[PE_WARPS][PE_CHUNK / 2];
    __shared__ float4 s_ny[PE_WARPS][PE_CHUNK / 2];
    __shared__ float2 s_v2[PE_WARPS][PE_CHUNK / 2];
    __shared__ double s_part[PE_WARPS][32];        // P2P lane partials of a sparse mask
    __shared__ int s_lane_of[PE_WARPS][32];        // the lane of the mask's q-th target
    __shared__ double s_neg_log_c[LOG_NTAB];       // log_pos's table
    load_log_table(s_neg_log_c);
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const double eps = 10 * DBL_EPSILON;
    const int *toff = offs + 2 * ngroups;
    const int tbase = toff[0];
    const int ntasks = toff[ngroups] - tbase;
    const TaskBins bins(tt.stride ? tt.fill : nullptr);

    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(task_ctr, 1);
        task = __shfl_sync(FULL_MASK, task, 0);
        if (task >= ntasks) break;
        const int2 entry = tt.entry[tt.stride ? bins.place(task, tt.stride) : task];
        task = entry.x;
        const int g = entry.y;
        if ((unsigned)task >= (unsigned)ntasks || (unsigned)g >= (unsigned)ngroups) break;
        const int part = task - (toff[g] - tbase);
        const int nparts = toff[g + 1] - toff[g];
        const int t = g * 32 + lane;
        const bool valid = t < m;
        int j = 0;
        double x = 0, y = 0;
        if (valid) {
            j = tperm[t];
            x = xt[j];
            y = yt[j];
        }
        // reference point of the mixed form's offsets: the group's first target
        const double xref = __shfl_sync(FULL_MASK, x, 0), yref = __shfl_sync(FULL_MASK, y, 0);
        double far = 0, near = 0;

        // E2P (potential-kernels.m4:59-89): m log(r2)/2 + Re sum_{j=1..p} a_{j-1} z^-j.  The next
        // entry's cell record and coefficients are loaded while the current one is evaluated.
        if (part == 0) {
            const int b0 = offs[g], e0 = offs[g + 1];
            float sh = 0, sl = 0;
            int2 ent_n = make_int2(0, 0);
            TNode nd_n = {};
            double m_n = 0;
            float R_n = 1.f;
            float2 c32_n = make_float2(0.f, 0.f);
            auto fetch = [&](int at) {
                ent_n = lists[at];
                nd_n = tnode[ent_n.x];
                m_n = mass[ent_n.x];
                R_n = sscale[ent_n.x];
                if (lane < P) c32_n = sexp[(size_t)ent_n.x * P + lane];
            };
            if (b0 < e0) fetch(b0);
            for (int it = b0; it < e0; ++it) {
                const int2 ent = ent_n;
                const TNode nd = nd_n;
                const double mm = m_n;
                const float R = R_n;
                __syncwarp();
                if (lane < P) {
                    float *cp = reinterpret_cast<float *>(s_coef32[warp]);
                    cp[4 * (lane >> 1) + (lane & 1)] = c32_n.x;
                    cp[4 * (lane >> 1) + 2 + (lane & 1)] = c32_n.y;
                }
                __syncwarp();
                if (it + 1 < e0) fetch(it + 1);
                if ((ent.y >> lane) & 1) {
                    const double rz = x - nd.xcom, iz = y - nd.ycom;
                    const double r2 = rz * rz + iz * iz;
                    // series: Re(u' Q(u')), u' = R / z, Q(u') = sum_j D_j u'^j
                    const float zr = (float)rz, zi = (float)iz;
                    const float inv = rcp_approx(zr * zr + zi * zi);
                    const float ur = R * zr * inv, ui = -R * zi * inv;
                    // Q(u') = E(w) + u' O(w), w = u'^2, E and O the even and odd parts
                    // of the series, evaluated together by Horner in f32x2 lanes
                    const float wr = fmaf(ur, ur, -ui * ui), wi = 2.f * ur * ui;
                    const float2 wr2 = make_float2(wr, wr), wi2 = make_float2(wi, wi);
                    const float2 nwi2 = make_float2(-wi, -wi);
                    const float4 cl = s_coef32[warp][P / 2 - 1];
                    float2 qr2 = make_float2(cl.x, cl.y), qi2 = make_float2(cl.z, cl.w);
#pragma unroll
                    for (int j = P / 2 - 2; j >= 0; --j) {
                        const float4 d = s_coef32[warp][j];
                        const float2 tr = __ffma2_rn(qi2, nwi2, make_float2(d.x, d.y));
                        const float2 ti = __ffma2_rn(qi2, wr2, make_float2(d.z, d.w));
                        const float2 nqr = __ffma2_rn(qr2, wr2, tr);
                        qi2 = __ffma2_rn(qr2, wi2, ti);
                        qr2 = nqr;
                    }
                    const float2 q = make_float2(
                        qr2.x + fmaf(ur, qr2.y, -ui * qi2.y),
                        qi2.x + fmaf(ur, qi2.y, ui * qr2.y));
                    two_sum_add(sh, sl, ur * q.x - ui * q.y);
                    far += mm * log_pos(r2, s_neg_log_c) * 0.5;
                }
            }
            far += (double)sh + (double)sl;
        }

        // P2P (potential-kernels.m4:19-57): 0.5 sum v log(r2 + eps), sources
        // [part * PT_SEG, (part + 1) * PT_SEG) of the group's listed leaves.  Tiles of up to
        // PE_CHUNK consecutive sources of one leaf; the next tile is loaded into registers while
        // the current one is evaluated.
        {
            const int b1 = offs[ngroups + g], e1 = offs[ngroups + g + 1];
            int it = b1, skip = part * PT_SEG, budget = PT_SEG;
            int s_next = 0, e_next = 0;
            unsigned mask_next = 0;
            while (it < e1) {
                const int2 ent = lists[it++];
                const int2 rg = range[ent.x];
                const int cnt = rg.y - rg.x;
                if (skip < cnt) {
                    s_next = rg.x + skip;
                    e_next = rg.y;
                    mask_next = (unsigned)ent.y;
                    break;
                }
                skip -= cnt;
            }
            auto next_tile = [&](int &t0, int &tn, unsigned &msk) {
                while (s_next >= e_next && it < e1) {
                    const int2 ent = lists[it++];
                    const int2 rg = range[ent.x];
                    s_next = rg.x;
                    e_next = rg.y;
                    mask_next = (unsigned)ent.y;
                }
                t0 = s_next;
                tn = min(min(PE_CHUNK, e_next - s_next), budget);
                if (tn < 0) tn = 0;
                msk = mask_next;
                s_next += tn;
                budget -= tn;
            };
            int t0, tn;
            unsigned msk;
            next_tile(t0, tn, msk);
            double px = 0, py = 0, pv = 0;
            if (lane < tn) {
                px = xs[t0 + lane];
                py = ys[t0 + lane];
                pv = vs[t0 + lane];
            }
            float nh = 0, nl = 0, txh = 0, txl = 0, tyh = 0, tyl = 0;
            split2(x - xref, txh, txl);
            split2(y - yref, tyh, tyl);
            const float ln2 = 0.6931471805599453f, epsf = (float)eps;
            // a sparse leaf's spreading (below): its mask, 32 / k, lane / k and the lane's target
            unsigned spread = 0;
            int sr = 0, sq = 0;
            float qxh = 0, qxl = 0, qyh = 0, qyl = 0;
            while (tn > 0) {
                const int cnt = tn;
                const unsigned cmask = msk;   // this tile's targets (msk moves on to the next tile)
                const bool mine = (cmask >> lane) & 1;
                __syncwarp();
                {
                    // source `lane` to entry lane / 2, half lane % 2; lanes past the tile add a
                    // zero-valued source at the reference point (finite, contributes 0)
                    float a = 0.f, b2 = 0.f, c2 = 0.f, d2 = 0.f, vv = 0.f;
                    if (lane < cnt) {
                        split2(px - xref, a, b2);
                        split2(py - yref, c2, d2);
                        vv = (float)pv;
                    }
                    float *nx = reinterpret_cast<float *>(s_nx[warp]);
                    float *ny = reinterpret_cast<float *>(s_ny[warp]);
                    const int e = 4 * (lane >> 1) + (lane & 1);
                    nx[e] = -a;
                    nx[e + 2] = -b2;
                    ny[e] = -c2;
                    ny[e + 2] = -d2;
                    reinterpret_cast<float *>(s_v2[warp])[lane] = vv;
                }
                __syncwarp();
                next_tile(t0, tn, msk);
                if (lane < tn) {
                    px = xs[t0 + lane];
                    py = ys[t0 + lane];
                    pv = vs[t0 + lane];
                }
                // A tile needed by few targets of the group (k <= 8) is spread over the lanes:
                // lane l takes target q = l % k of the mask and sources l / k, l / k + r, ...
                // (r = 32 / k), and each target adds its r lane partials in lane order.  Denser
                // tiles keep one target per lane.
                const int k = __popc(cmask);
                if (k > 8) {
                    if (mine) {
                        // two sources per step in f32x2 lanes; even and odd sources are
                        // summed apart and added at the end of the tile
                        const float2 txh2 = make_float2(txh, txh), txl2 = make_float2(txl, txl);
                        const float2 tyh2 = make_float2(tyh, tyh), tyl2 = make_float2(tyl, tyl);
                        const float2 eps2 = make_float2(epsf, epsf);
                        float2 acc = make_float2(0.f, 0.f);
                        const int npairs = (cnt + 1) >> 1;
#pragma unroll 4
                        for (int q = 0; q < npairs; ++q) {
                            const float4 nx = s_nx[warp][q], ny = s_ny[warp][q];
                            const float2 dx = __fadd2_rn(__fadd2_rn(txh2, make_float2(nx.x, nx.y)),
                                                         __fadd2_rn(txl2, make_float2(nx.z, nx.w)));
                            const float2 dy = __fadd2_rn(__fadd2_rn(tyh2, make_float2(ny.x, ny.y)),
                                                         __fadd2_rn(tyl2, make_float2(ny.z, ny.w)));
                            const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, eps2));
                            acc = __ffma2_rn(make_float2(lg2_approx(r2.x), lg2_approx(r2.y)),
                                             s_v2[warp][q], acc);
                        }
                        two_sum_mul<false>(nh, nl, acc.x + acc.y, ln2);
                    }
                } else if (k > 0) {
                    if (cmask != spread) {   // once per leaf: its tiles share the mask
                        spread = cmask;
                        __syncwarp();
                        if (mine) s_lane_of[warp][__popc(cmask & ((1u << lane) - 1u))] = lane;
                        __syncwarp();
                        sr = 32 / k;
                        sq = lane / k;
                        const int tl = s_lane_of[warp][lane - sq * k];   // lane of this lane's target
                        qxh = __shfl_sync(FULL_MASK, txh, tl);
                        qxl = __shfl_sync(FULL_MASK, txl, tl);
                        qyh = __shfl_sync(FULL_MASK, tyh, tl);
                        qyl = __shfl_sync(FULL_MASK, tyl, tl);
                    }
                    const int r = sr;
                    double part = 0;
                    {
                        float acc = 0;
                        const float *nx = reinterpret_cast<const float *>(s_nx[warp]);
                        const float *ny = reinterpret_cast<const float *>(s_ny[warp]);
                        const float *sv = reinterpret_cast<const float *>(s_v2[warp]);
                        if (lane < r * k)
                            for (int q = sq; q < cnt; q += r) {
                                const int e = 4 * (q >> 1) + (q & 1);
                                const float dx = (qxh + nx[e]) + (qxl + nx[e + 2]);
                                const float dy = (qyh + ny[e]) + (qyl + ny[e + 2]);
                                acc = fmaf(lg2_approx(fmaf(dx, dx, fmaf(dy, dy, epsf))), sv[q], acc);
                            }
                        part = (double)acc;
                    }
                    s_part[warp][lane] = part;
                    __syncwarp();
                    if (mine) {
                        const int q = __popc(cmask & ((1u << lane) - 1u));
                        double sum = 0;
                        for (int i = 0; i < r; ++i) sum += s_part[warp][q + i * k];
                        two_sum_mul<true>(nh, nl, (float)sum, ln2);
                    }
                    __syncwarp();
                }
            }
            near = (double)nh + (double)nl;
        }
        const double res = 0.5 * near + far;
        if (nparts == 1) {
            if (valid) out[j] = res;
        } else {
            partial[(size_t)task * 32 + lane] = res;
        }
        __syncwarp();
    }
}

// The FP64 form: 12 FP64 operations per P2P pair (16 lanes of the pipe per scheduler, so 24 cycles per
// 32 pairs) and about 20 others.  On 1M clustered sources and targets 65% of the cycles issue and the
// FP64 pipe is busy for 56%; an FP64 instruction keeps its scheduler for a second cycle (28%), which
// leaves 7% of them unused.  Blocks of 8 warps share one set of table copies (64 KB); three blocks, 24
// warps, fit on an SM.
// Tasks: group g owns tasks [toff[g], toff[g+1]).  seg == PT_SEG: task 0 evaluates the far field
// and the first segment of the group's near field, task p > 0 the p-th segment.  seg < PT_SEG:
// the far field is task 0 (where the group has one), and the p-th near-field task takes the tiles
// that start in sources [p seg, (p + 1) seg) of the group's near field.
constexpr int PD_WARPS = 8;
constexpr int PD_MIN_BLOCKS = 3;

// Per-warp staging: a cell's coefficients, or a tile's sources (never both at once); the lane
// partials of a sparse tile.
template <int P>
struct EvalShared {
    union {
        cplx coef[P > PS_TERMS ? P : PS_TERMS];
        struct {
            double2 xy[PE_CHUNK];
            double v[PE_CHUNK];
        } src;
    };
    double part[32];
    int lane_of[32];   // sparse tiles: the lane of the q-th target of the mask
};

template <int P>
constexpr size_t eval_smem() {
    return sizeof(double2) * NLOG_NTAB * NLOG_COPIES + sizeof(EvalShared<P>) * PD_WARPS;
}

// SETS: the groups' common far field is added from their set's local expansion (`local`, null where
// there are no sets).
// WIDE: for solves with a target NEAR_REACH or more away from a source, whose squares may pass
// log_near's range or overflow: log_pos, whose logarithm of infinity is 1024 ln 2, and a true
// division (the arithmetic of the kernel before log_near).  4096 sources and targets with one such
// target 159 us a solve instead of 140, 64K 383 and 359, 1M 3394 and 3017.
template <int P, bool SETS, bool WIDE>
__global__ __launch_bounds__(PD_WARPS * 32, PD_MIN_BLOCKS) void k_potential_eval(
    int ngroups, int m, const double *__restrict__ xt, const double *__restrict__ yt,
    const int *__restrict__ tperm, const TNode *__restrict__ tnode,
    const double *__restrict__ mass, const double *__restrict__ exps,
    const int2 *__restrict__ range, const double *__restrict__ xs,
    const double *__restrict__ ys, const double *__restrict__ vs,
    const int *__restrict__ offs, const int2 *__restrict__ lists, double *__restrict__ out,
    double *__restrict__ partial, int *task_ctr, TaskTable tt, int seg,
    const double4 *__restrict__ geo, const cplx *__restrict__ local) {
    extern __shared__ __align__(16) unsigned char eval_dyn[];
    double2 *s_tab = reinterpret_cast<double2 *>(eval_dyn);
    double *s_neg_log_c = reinterpret_cast<double *>(eval_dyn);
    static_assert(sizeof(double) * LOG_NTAB <= sizeof(double2) * NLOG_NTAB * NLOG_COPIES, "");
    // (constant tables: before the kernel before this one is done)
    if constexpr (WIDE) load_log_table(s_neg_log_c);
    else load_near_log_table(s_tab);
    pdl_begin();
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    const unsigned tab = shared_address(s_tab);
    const int copy = (lane & (NLOG_COPIES - 1)) * (int)sizeof(double2);
    EvalShared<P> &sh =
        reinterpret_cast<EvalShared<P> *>(s_tab + NLOG_NTAB * NLOG_COPIES)[warp];
    const double eps = 10 * DBL_EPSILON;
    auto log_of = [&](double r2) {
        if constexpr (WIDE) return log_pos(r2, s_neg_log_c);
        else return log_near(r2, tab, copy);
    };
    const int *toff = offs + 2 * ngroups;
    const int tbase = toff[0];
    const int ntasks = toff[ngroups] - tbase;
    const TaskBins bins(tt.stride ? tt.fill : nullptr);

    for (;;) {
        int task = 0;
        if (lane == 0) task = atomicAdd(task_ctr, 1);
        task = __shfl_sync(FULL_MASK, task, 0);
        if (task >= ntasks) break;
        const int2 entry = tt.entry[tt.stride ? bins.place(task, tt.stride) : task];
        task = entry.x;
        const int g = entry.y;
        if ((unsigned)task >= (unsigned)ntasks || (unsigned)g >= (unsigned)ngroups) break;
        const int part = task - (toff[g] - tbase);
        const int nparts = toff[g + 1] - toff[g];
        // the near-field task of this part; -1: the far field alone
        const int npart = seg < PT_SEG && offs[g + 1] > offs[g] ? part - 1 : part;
        const int t = g * 32 + lane;
        const bool valid = t < m;
        int j = 0;
        double x = 0, y = 0;
        if (valid) {
            j = tperm[t];
            x = xt[j];
            y = yt[j];
        }
        double far = 0, near = 0;

        // E2P (potential-kernels.m4:59-89): m log(r2)/2 + Re sum_{j=1..p} a_{j-1} z^-j.  The next
        // entry's cell record and coefficients are loaded while the current one is evaluated.
        if (part == 0) {
            const int b0 = offs[g], e0 = offs[g + 1];
            if (SETS && (!WIDE || local)) {   // the set's common far field: Re sum_l L_l R^l ((t - c) / R)^l
                const double4 q4 = geo[g / PS_GROUPS];
                __syncwarp();
                sh.coef[lane] = local[(size_t)(g / PS_GROUPS) * PS_TERMS + lane];
                __syncwarp();
                const double ir = 1.0 / q4.z;
                const cplx d = {valid ? (x - q4.x) * ir : 0.0, valid ? (y - q4.y) * ir : 0.0};
                cplx q = sh.coef[PS_TERMS - 1];
#pragma unroll
                for (int k = PS_TERMS - 2; k >= 0; --k) q = cfma(q, d, sh.coef[k]);
                far = q.re;
            }
            int2 ent_n = make_int2(0, 0);
            TNode nd_n = {};
            double m_n = 0, cr_n = 0, ci_n = 0;
            auto fetch = [&](int at) {
                ent_n = lists[at];
                nd_n = tnode[ent_n.x];
                m_n = mass[ent_n.x];
                if (lane < P) {
                    const double *ex = exps + (size_t)ent_n.x * 2 * P;
                    cr_n = ex[lane];
                    ci_n = ex[P + lane];
                }
            };
            if (b0 < e0) fetch(b0);
            for (int it = b0; it < e0; ++it) {
                const int2 ent = ent_n;
                const TNode nd = nd_n;
                const double mm = m_n;
                __syncwarp();
                if (lane < P) sh.coef[lane] = {cr_n, ci_n};
                __syncwarp();
                if (it + 1 < e0) fetch(it + 1);
                if ((ent.y >> lane) & 1) {
                    const double rz = x - nd.xcom, iz = y - nd.ycom;
                    const double r2 = rz * rz + iz * iz;
                    const double inv = WIDE ? 1.0 / r2 : rcp_nr(r2);
                    const cplx u = {rz * inv, -iz * inv};
                    cplx q = sh.coef[P - 1];
#pragma unroll
                    for (int k = P - 2; k >= 0; --k) q = cfma(q, u, sh.coef[k]);
                    far += mm * log_of(r2) * 0.5 + (u.re * q.re - u.im * q.im);
                }
            }
        }

        // P2P (potential-kernels.m4:19-57): 0.5 sum v log(r2 + eps) over the tiles of the
        // group's listed leaves that start in sources [npart * seg, (npart + 1) * seg).  Tiles
        // of up to PE_CHUNK consecutive sources of one leaf and one segment; the next tile is
        // loaded into registers while the current one is evaluated.
        if (npart >= 0) {
            const int b1 = offs[ngroups + g], e1 = offs[ngroups + g + 1];
            // positions count the group's near-field sources; the segment ends at pos_seg
            const int lo = npart * seg;
            const int seg0 = lo - (lo & (PT_SEG - 1)), pos_seg = seg0 + PT_SEG;
            const int hi = lo + seg;
            int it = b1, pos = 0;
            int s_next = 0, e_next = 0;
            unsigned mask_next = 0;
            // the first tile that starts at or after lo
            while (it < e1) {
                const int2 ent = lists[it++];
                const int2 rg = range[ent.x];
                const int cnt = rg.y - rg.x;
                if (pos + cnt > lo) {
                    const int first = max(0, seg0 - pos);   // the leaf's first tile of the segment
                    const int skip = first + (max(0, lo - pos - first) + PE_CHUNK - 1) / PE_CHUNK *
                                                 PE_CHUNK;
                    if (skip < cnt) {
                        s_next = rg.x + skip;
                        e_next = rg.y;
                        mask_next = (unsigned)ent.y;
                        pos += skip;
                        break;
                    }
                }
                pos += cnt;
            }
            auto next_tile = [&](int &t0, int &tn, unsigned &msk) {
                while (s_next >= e_next && it < e1) {
                    const int2 ent = lists[it++];
                    const int2 rg = range[ent.x];
                    s_next = rg.x;
                    e_next = rg.y;
                    mask_next = (unsigned)ent.y;
                }
                t0 = s_next;
                tn = pos < hi ? min(min(PE_CHUNK, e_next - s_next), pos_seg - pos) : 0;
                if (tn < 0) tn = 0;
                msk = mask_next;
                s_next += tn;
                pos += tn;
            };
            int t0, tn;
            unsigned msk;
            next_tile(t0, tn, msk);
            double px = 0, py = 0, pv = 0;
            if (lane < tn) {
                px = xs[t0 + lane];
                py = ys[t0 + lane];
                pv = vs[t0 + lane];
            }
            // a sparse leaf's spreading (below): its mask, 32 / k, lane / k and the lane's target
            unsigned spread = 0;
            int sr = 0, sq = 0;
            double qx = 0, qy = 0;
            while (tn > 0) {
                const int cnt = tn;
                const unsigned cmask = msk;   // this tile's targets (msk moves on to the next tile)
                const bool mine = (cmask >> lane) & 1;
                __syncwarp();
                // (lanes past the tile: a zero value at the origin, for the two-source steps)
                const bool live = lane < cnt;
                sh.src.xy[lane] = make_double2(live ? px : 0.0, live ? py : 0.0);
                sh.src.v[lane] = live ? pv : 0.0;
                __syncwarp();
                next_tile(t0, tn, msk);
                if (lane < tn) {
                    px = xs[t0 + lane];
                    py = ys[t0 + lane];
                    pv = vs[t0 + lane];
                }
                // A tile needed by few targets of the group (k <= 16) is spread over the lanes:
                // lane l takes target q = l % k of the mask and sources l / k, l / k + r, ...
                // (r = 32 / k), and each target adds its r lane partials in lane order.  Denser
                // tiles keep one target per lane, two sources per step.
                const int k = __popc(cmask);
                if (k > 16) {
                    if (mine) {
                        const double2 *v2 = reinterpret_cast<const double2 *>(sh.src.v);
                        double n0 = 0, n1 = 0;
#pragma unroll 2
                        for (int q = 0; q < cnt; q += 2) {
                            const double2 sp = sh.src.xy[q], sq = sh.src.xy[q + 1];
                            const double2 v = v2[q >> 1];
                            const double xr = x - sp.x, yr = y - sp.y;
                            const double xq = x - sq.x, yq = y - sq.y;
                            n0 = fma(log_of(fma(xr, xr, fma(yr, yr, eps))), v.x, n0);
                            n1 = fma(log_of(fma(xq, xq, fma(yq, yq, eps))), v.y, n1);
                        }
                        near += n0 + n1;
                    }
                } else if (k > 0) {
                    if (cmask != spread) {   // once per leaf: its tiles share the mask
                        spread = cmask;
                        __syncwarp();
                        if (mine) sh.lane_of[__popc(cmask & ((1u << lane) - 1u))] = lane;
                        __syncwarp();
                        sr = 32 / k;
                        sq = lane / k;
                        const int tl = sh.lane_of[lane - sq * k];   // lane of this lane's target
                        qx = __shfl_sync(FULL_MASK, x, tl);
                        qy = __shfl_sync(FULL_MASK, y, tl);
                    }
                    const int r = sr;
                    double sum = 0;
                    if (lane < r * k)
                        for (int q = sq; q < cnt; q += r) {
                            const double2 sp = sh.src.xy[q];
                            const double xr = qx - sp.x, yr = qy - sp.y;
                            sum = fma(log_of(fma(xr, xr, fma(yr, yr, eps))), sh.src.v[q], sum);
                        }
                    sh.part[lane] = sum;
                    __syncwarp();
                    if (mine) {
                        const int q = __popc(cmask & ((1u << lane) - 1u));
                        double tot = 0;
                        for (int i = 0; i < r; ++i) tot += sh.part[q + i * k];
                        near += tot;
                    }
                    __syncwarp();
                }
            }
        }
        const double res = 0.5 * near + far;
        if (nparts == 1) {
            if (valid) out[j] = res;
        } else {
            partial[(size_t)task * 32 + lane] = res;
        }
        __syncwarp();
    }
}

__global__ void k_task_map_groups(int ngroups, const int *__restrict__ counts,
                                  const int *__restrict__ offs, TaskTable tt) {
    const int *toff = offs + 2 * ngroups;
    const int tbase = toff[0];
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x)
        for (int t = toff[g]; t < toff[g + 1]; ++t)
            put_task(tt, t - tbase, t - toff[g], g, counts[g]);
}

// Sum of the parts of every multi-task group, in task order (deterministic).  Bound by latency:
// what is older than the evaluation (offsets, order) is read before the wait for it, and the parts
// GP_BATCH at a time (24 parts a group at 4096 sources: 142.0 -> 139.9 us a solve).
constexpr int GP_BATCH = 8;

__global__ __launch_bounds__(256) void k_potential_gather_parts(int ngroups, int m,
                                                                const int *__restrict__ tperm,
                                                                const int *__restrict__ offs,
                                                                const double *__restrict__ partial,
                                                                double *__restrict__ out) {
    const int lane = lane_id();
    const int *toff = offs + 2 * ngroups;
    const int stride = (gridDim.x * blockDim.x) >> 5;
    bool waited = false;
    for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += stride) {
        const int t0 = toff[g] - toff[0], np = toff[g + 1] - toff[g];
        if (np <= 1) continue;
        const int t = g * 32 + lane;
        const int to = t < m ? tperm[t] : 0;
        if (!waited) pdl_begin();   // the offsets and the order are older than the evaluation
        waited = true;
        const double *p = partial + (size_t)t0 * 32 + lane;
        double s = 0;
        int k = 0;
        for (; k + GP_BATCH <= np; k += GP_BATCH) {
            double v[GP_BATCH];
#pragma unroll
            for (int u = 0; u < GP_BATCH; ++u) v[u] = p[(size_t)(k + u) * 32];
#pragma unroll
            for (int u = 0; u < GP_BATCH; ++u) s += v[u];
        }
        for (; k < np; ++k) s += p[(size_t)k * 32];
        if (t < m) out[to] = s;
    }
    if (!waited) pdl_begin();
}

// Mixed form: a_k / R^(k+1) in FP32, R = the cell's power-of-two radius (see force.cu).
template <int P>
__global__ void k_scale_coeffs_pot(int nnodes, const TNode *__restrict__ tnode,
                                   const double *__restrict__ exps, float2 *__restrict__ sexp,
                                   float *__restrict__ sscale) {
    pdl_begin();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)nnodes * P;
         i += (long long)gridDim.x * blockDim.x) {
        const int node = (int)(i / P), k = (int)(i % P);
        const double r = tnode[node].r;
        int e = 0;
        if (r > 0 && r < 1e300) frexp(r, &e);
        const double *ex = exps + (size_t)node * 2 * P;
        sexp[i] = make_float2((float)ldexp(ex[k], -e * (k + 1)), (float)ldexp(ex[P + k], -e * (k + 1)));
        if (k == 0) sscale[node] = (float)ldexp(1.0, e);
    }
}

static int sm_count_p() { return device_sm_count(); }

// The lists are built on the auxiliary stream, where the target sort went before (sort_sources);
// `between` (the expansion work) runs on the main stream meanwhile, and the evaluation waits for
// both.
int potential(Context &c, double theta, const double *xt, const double *yt, int m, double *out,
              OverlapFn between) {
    if (m == 0) return between ? between(c) : TC_OK;
    int rc;
    const int ngroups = (m + 31) / 32;
    // counts / offsets: E2P | P2P list lengths and evaluation tasks, ngroups each
    int *counts, *offs;
    if ((rc = ensure(c, S_PCOUNT, (size_t)3 * ngroups, &counts)) ||
        (rc = ensure(c, S_POFF, (size_t)3 * ngroups + 1, &offs)))
        return rc;
    const TNode *tnode = slot_ptr<TNode>(c, S_TNODE);
    unsigned *err = c.ctrl.err;
    const int grid = (int)std::min<long long>((ngroups + PT_WARPS - 1) / PT_WARPS,
                                              (long long)sm_count_p() * 16);
    int *vo;
    // One walk counts the lists and writes them into per-warp scratch runs; after the scan a
    // copy puts them in CSR order.  If a run outgrew its region a second walk writes them
    // instead, and the regions are sized up for the next solve.  The runs live in the sort's
    // record buffer when they fit in it, else in a block held only for the build.
    const int nwarps = grid * PT_WARPS;
    const int seg = task_segment(ngroups, c.precision == 1);
    // sets of groups with a common far field (FP64, many groups: below PS_MIN_GROUPS a set's chain
    // of cells takes longer than it saves)
    SuperSets sets = {};
    const int nsets = (ngroups + PS_GROUPS - 1) / PS_GROUPS;
    const double rho = c.precision == 0 && ngroups >= PS_MIN_GROUPS ? super_rho(theta, c.order) : 0.0;
    const bool with_sets = rho > 0;
    cplx *set_local = nullptr;
    ScratchLayout sl;
    ListScratch ls;   // released (when transient) after the copy, in stream order
    int *sstart, *meta = c.ctrl.meta;
    unsigned long long *stats = c.ctrl.stats;
    const bool chain = c.launch_overlap && c.single;   // on one stream: launch_pdl
    TC_CUDA_TRY(stream_after(c, c.aux, c.stream, c.ev_fork));
    {
        AuxScope on_aux(c);
        if (!c.targets_sorted && (rc = sort_targets(c, xt, yt, m, &c.tperm))) return rc;
        vo = c.tperm;
        c.targets_sorted = false;
        if ((rc = list_scratch(c, 2, nwarps, ngroups, sizeof(int2), sl, ls)) ||
            (rc = ensure(c, S_LSTART, (size_t)3 * ngroups, &sstart)))
            return rc;
        if (with_sets) {
            int *lists2, *num;
            double4 *geo;
            if ((rc = ensure(c, S_SETLIST, (size_t)2 * nsets * PS_LIST, &lists2)) ||
                (rc = ensure(c, S_SETNUM, (size_t)2 * nsets, &num)) ||
                (rc = ensure(c, S_SETGEO, (size_t)nsets, &geo)) ||
                (rc = ensure(c, S_SETLOCAL, (size_t)nsets * PS_TERMS, &set_local)))
                return rc;
            int *start = lists2 + (size_t)nsets * PS_LIST;
            TC_CUDA_TRY(launch_pdl(
                c.launch_overlap, k_potential_supers,
                (int)std::min<long long>((nsets + PT_WARPS - 1) / PT_WARPS,
                                         (long long)sm_count_p() * 16),
                PT_WARPS * 32, 0, c.stream, nsets, m, xt, yt, (const int *)vo, theta, rho, tnode,
                c.nnodes, lists2, num, start, num + nsets, geo, err, stats));
            TC_KERNEL_CHECK();
            sets = {lists2, num, start, num + nsets, geo};
        }
        TC_CUDA_TRY(launch_pdl(c.launch_overlap, k_potential_lists<2>, grid, PT_WARPS * 32, 0,
                               c.stream, ngroups, m, xt, yt, (const int *)vo, theta, tnode, c.nnodes,
                               counts, (const int *)nullptr, (int2 *)nullptr,
                               static_cast<int2 *>(ls.p), sl, sstart, meta, err, stats, seg, sets));
        TC_KERNEL_CHECK();
        // the lists' totals and meta, written to h_pinned by the scan
        if ((rc = exclusive_scan(c, counts, offs, 3 * ngroups, ngroups, c.h_pinned + 32, meta)))
            return rc;
        TC_CUDA_TRY(cudaEventRecord(c.ev_totals, c.stream));
    }
    if (between && (rc = between(c))) {
        cudaStreamSynchronize(c.aux);   // leave nothing of this solve in flight
        return rc;
    }
    TC_CUDA_TRY(wait_event(c, c.ev_totals));
    const int n_e2p = (int)c.h_pinned[32], total = (int)c.h_pinned[33];
    const int ntasks = (int)c.h_pinned[34] - total;
    const bool overflow = c.h_pinned[35] != 0;
    const bool wide = c.h_pinned[35 + META_WIDE] != 0;
    c.list_walks = overflow ? 2 : 1;
    scratch_learn(c, 2, nwarps, ngroups, c.h_pinned + 36);   // for the next solve
    c.counts.n_e2p = n_e2p;
    c.counts.n_p2p = total - n_e2p;
    c.counts.l2p_targets = with_sets ? m : 0;   // (n_e2l and the pairs: read back with the result)
    int2 *lists;
    TaskTable tt = {nullptr, ngroups <= PT_LPT_GROUPS ? ntasks : 0, c.ctrl.task_fill,
                    sstart + 2 * (size_t)ngroups, seg};
    {
        AuxScope on_aux(c);
        if ((rc = ensure(c, S_PE2P, (size_t)total + 1, &lists)) ||
            (rc = ensure(c, S_TASKMAP, (size_t)(tt.stride ? TASK_BINS : 1) * ntasks, &tt.entry)))
            return rc;
        if (!overflow) {
            TC_CUDA_TRY(launch_pdl(
                chain, k_potential_lists_copy,
                (int)std::min<long long>((ngroups + 7) / 8, (long long)sm_count_p() * 16), 256, 0,
                c.stream, ngroups, (const int *)counts, (const int *)offs, (const int *)sstart,
                static_cast<const int2 *>(ls.p), lists, tt));
        } else {
            // (the second walk does not add to the work counters)
            k_potential_lists<1><<<grid, PT_WARPS * 32, 0, c.stream>>>(
                ngroups, m, xt, yt, vo, theta, tnode, c.nnodes, nullptr, offs, lists, nullptr,
                sl, nullptr, nullptr, err, stats, seg, sets);
            TC_KERNEL_CHECK();
            k_task_map_groups<<<(int)std::min<long long>((ngroups + 255) / 256,
                                                         (long long)sm_count_p() * 8),
                                256, 0, c.stream>>>(ngroups, counts, offs, tt);
        }
        TC_KERNEL_CHECK();
        TC_CUDA_TRY(mark_event(c, c.ev_join));
    }
    TC_CUDA_TRY(await_event(c, c.ev_join));
    phase_mark(c, 4);
    int *task_ctr = c.ctrl.near_ctr;   // (cleared at the solve's start)
    double *partial;
    if ((rc = ensure(c, S_FPART, (size_t)ntasks * 32, &partial))) return rc;
    // the evaluation for the tree's expansion order
    rc = dispatch_order(c.order, [&](auto order) -> int {
        constexpr int P = decltype(order)::value;
        int rc2;
        const bool mixed = c.precision == 1;
        float2 *sexp = nullptr;
        float *sscale = nullptr;
        if (mixed) {
            if ((rc2 = ensure(c, S_SEXP, (size_t)c.nnodes * P, &sexp)) ||
                (rc2 = ensure(c, S_SSCALE, (size_t)c.nnodes, &sscale)))
                return rc2;
            const long long items = (long long)c.nnodes * P;
            TC_CUDA_TRY(launch_pdl(
                chain, k_scale_coeffs_pot<P>,
                (int)std::min<long long>((items + 255) / 256, (long long)sm_count_p() * 8), 256, 0,
                c.stream, c.nnodes, tnode, (const double *)slot_ptr<double>(c, S_EXPS), sexp,
                sscale));
            TC_KERNEL_CHECK();
        }
        if (mixed) {
            const int occ = blocks_per_sm<k_potential_eval_mixed<P>>(PE_WARPS * 32, 0);
            const int egrid = (int)std::min<long long>((ntasks + PE_WARPS - 1) / PE_WARPS,
                                                       (long long)sm_count_p() * occ);
            phase_mark(c, 6);
            TC_CUDA_TRY(launch_pdl(
                chain, k_potential_eval_mixed<P>, egrid, PE_WARPS * 32, 0, c.stream, ngroups, m, xt,
                yt, (const int *)vo, tnode, (const double *)slot_ptr<double>(c, S_MASS),
                (const int2 *)slot_ptr<int2>(c, S_RANGE), (const double *)slot_ptr<double>(c, S_XS),
                (const double *)slot_ptr<double>(c, S_YS),
                (const double *)slot_ptr<double>(c, S_VS), (const int *)offs, (const int2 *)lists,
                out, partial, task_ctr, tt, (const float2 *)sexp,
                (const float *)sscale));
        } else {
            auto eval = wide        ? k_potential_eval<P, true, true>
                        : with_sets ? k_potential_eval<P, true, false>
                                    : k_potential_eval<P, false, false>;
            const int occ =
                blocks_per_sm<k_potential_eval<P, false, false>>(PD_WARPS * 32, eval_smem<P>());
            const int egrid = (int)std::min<long long>((ntasks + PD_WARPS - 1) / PD_WARPS,
                                                       (long long)sm_count_p() * occ);
            phase_mark(c, 6);
            if (with_sets) {
                const int occ_l = blocks_per_sm<k_potential_locals<P>>(PLOC_WARPS * 32, 0);
                k_potential_locals<P><<<(int)std::min<long long>((nsets + PLOC_WARPS - 1) / PLOC_WARPS,
                                                                 (long long)sm_count_p() * occ_l),
                                        PLOC_WARPS * 32, 0, c.stream>>>(
                    nsets, sets, tnode, slot_ptr<double>(c, S_MASS), slot_ptr<double>(c, S_EXPS),
                    set_local);
                TC_KERNEL_CHECK();
            }
            TC_CUDA_TRY(launch_pdl(
                chain, eval, egrid, PD_WARPS * 32, eval_smem<P>(), c.stream, ngroups,
                m, xt, yt, (const int *)vo, tnode, (const double *)slot_ptr<double>(c, S_MASS),
                (const double *)slot_ptr<double>(c, S_EXPS),
                (const int2 *)slot_ptr<int2>(c, S_RANGE), (const double *)slot_ptr<double>(c, S_XS),
                (const double *)slot_ptr<double>(c, S_YS),
                (const double *)slot_ptr<double>(c, S_VS), (const int *)offs, (const int2 *)lists,
                out, partial, task_ctr, tt, seg, sets.geo,
                (const cplx *)set_local));
        }
        TC_KERNEL_CHECK();
        return TC_OK;
    });
    if (rc) return rc;
    phase_mark(c, 7);
    if (ntasks > ngroups) {
        TC_CUDA_TRY(launch_pdl(
            c.launch_overlap, k_potential_gather_parts,
            (int)std::min<long long>((ngroups + 7) / 8, (long long)sm_count_p() * 16), 256, 0,
            c.stream, ngroups, m, (const int *)vo, (const int *)offs, (const double *)partial, out));
        TC_KERNEL_CHECK();
    }
    return TC_OK;
}

int prepare_potential() {
    int rc;
#define TC_EVAL_SHARED(P)                                                                         \
    if ((rc = allow_shared((const void *)k_potential_eval<P, false, false>, eval_smem<P>())) ||   \
        (rc = allow_shared((const void *)k_potential_eval<P, true, false>, eval_smem<P>())) ||    \
        (rc = allow_shared((const void *)k_potential_eval<P, true, true>, eval_smem<P>())))       \
        return rc;
    TC_FOR_EACH_ORDER(TC_EVAL_SHARED)
#undef TC_EVAL_SHARED
    return TC_OK;
}

void kernels_potential(KernelList &v) {
    v.insert(v.end(), {(const void *)k_potential_lists<1>, (const void *)k_potential_lists<2>,
                       (const void *)k_potential_lists_copy, (const void *)k_task_map_groups,
                       (const void *)k_potential_gather_parts, (const void *)k_potential_supers});
#define TC_POTENTIAL_KERNELS(P)                                                                  \
    v.insert(v.end(), {(const void *)k_potential_eval_mixed<P>,                              \
                       (const void *)k_potential_eval<P, false, false>,                          \
                       (const void *)k_potential_eval<P, true, false>,                           \
                       (const void *)k_potential_eval<P, true, true>,                            \
                       (const void *)k_potential_locals<P>,                                      \
                       (const void *)k_scale_coeffs_pot<P>});
    TC_FOR_EACH_ORDER(TC_POTENTIAL_KERNELS)
#undef TC_POTENTIAL_KERNELS
}

}  // namespace tc
