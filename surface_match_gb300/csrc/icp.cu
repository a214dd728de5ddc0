// icp.cu - pose refinement and scoring of matchScene (ppf.cpp:422-495): ICP::regist
// (icp.cpp:214-278) with findCorresponds (icp.cpp:123-167), the symmetric point-to-plane
// step (icp.cpp:39-121) and inliner (util.cpp:628-641).
//
// All candidates are refined at once; the searches spread each candidate's source points
// over many CTAs, so the whole GPU works even for a handful of candidates. One ICP iteration
// is four launches: correspondences (one warp per source point on the grid cell walker; per
// scene point the closest source point wins a 64-bit atomicMin of (distance bits, source
// index), which is the reference's "first minimum in model order" without its O(n*m)
// grouping scan); pair selection, pair count, centroids, normal-equation terms and the FP64
// solve in one thread-block cluster per candidate; residual distances; and their reduction +
// the convergence logic in one cluster per candidate. Every reduction has the same fixed
// layout: kIcpSlots slots (slot = source index mod kIcpSlots, a thread each), each a Kahan sum
// over its source points in ascending order, merged by a fixed tree (warp, the CTA's warps,
// then the cluster's CTAs through distributed shared memory) - the layout the CPU oracle
// emulates, so poses are bit-identical. The selection walk over the candidates
// (numMatches) runs on the host afterwards and only reads the per-candidate results.
#include <cfloat>

#include <cooperative_groups.h>

#include "sm_icp.h"
#include "sm_kdgrid.cuh"
#include "sm_stages.h"

namespace sm {
using namespace smd;
namespace cg = cooperative_groups;

namespace {

constexpr int kT  = 256;              // search CTAs: a warp (or a thread) per point
constexpr int kW  = kT / 32;
constexpr int kR  = smi::kIcpThreads; // reduction CTAs: a slot per thread
constexpr int kRW = kR / 32;
constexpr int kRC = smi::kIcpBlocks;  // reduction CTAs per candidate: one thread-block cluster
constexpr int kFitU = 4;              // pairs whose loads a reduction thread has in flight
constexpr int kStepLists = 3;         // candidate lists that a stage's steps take in turn
constexpr int kTraceIters  = 32;
constexpr int kTraceFloats = 2 * kTraceIters * 4 + 2;

// Per-candidate state, resident in global memory across the launches of one refinement.
struct Cand {
    smi::Pose34 M, keep, step;
    float       Pm[3], Qm[3];
    float       resMse, mse, score;
    int         cnt, iterations, converged, status, active, inl;
};

struct Stage {
    const float4 *src, *srcN; // model points / normals
    int           n;          // points
    HGridView     G;          // scene subset grid (pts.w = subset rank)
    const float4 *dPos, *dNrm; // the subset's positions / normals by rank
    int           nDst;
    int           iters;
    float         mseMin, mseMax, rej2;
    int           traceOff; // 0 sparse, 1 dense
    // reference search order: nearest points as the k-d tree reduced to the stage's subset
    // finds them (rankOf maps a point id to its subset rank, tposOf a rank to its tree
    // position); tree.nd == nullptr: the nearest points of the grid G
    smk::KdView   tree;
    int           treeM; // tree positions
    const int    *rankOf, *tposOf;
    const float  *exc; // largest excursion of the subset's points from their leaves' boxes
};

struct Work {
    Cand               *cand;
    int                *nnId;   // ncand x maxSrc: subset rank of the pair's scene point (-1 none)
    int                *nnR;    // ncand x maxSrc: the same, kept through pair selection
    int                *nnPrev; // ncand x maxSrc: nearest subset point of the last iteration
    float4             *x4;     // ncand x maxSrc: moved source point, w = squared distance
    float4             *n4;     // ncand x maxSrc: rotated source normal
    float              *resid;  // ncand x maxSrc: residual distance of each pair
    unsigned long long *win;    // ncand x maxDst
    int                 maxSrc, maxDst;
    float              *trace;  // ncand x kTraceFloats (nullable)
    unsigned long long *live;   // (candidate, source point) searches of K1 (nullable: not counted)
    // a stage's candidate lists (any order), list l at list[l * ncand ..], cnt[l] of them: step `it`
    // refines list it % kStepLists and lists those that go on in the next one, while the third is
    // cleared; list kStepLists holds those the stage leaves active
    int                *cnt, *list;
    int                 ncand;
    unsigned long long *heard; // page-locked: {tag, candidates} of the last step begun
};

// The candidates of list l: their number and the k-th.
__device__ __forceinline__ int step_list(int it) { return it % kStepLists; }
__device__ __forceinline__ int step_count(const Work &w, int l) { return w.cnt[l]; }
__device__ __forceinline__ int step_cand(const Work &w, int l, int k) { return w.list[l * w.ncand + k]; }
// Candidate and source point of item k of the list's candidates times n source points.
__device__ __forceinline__ void step_item(const Work &w, int l, long long k, int n, int &ci, int &i) {
    const int c = k < (1ll << 31) ? (int)((unsigned)k / (unsigned)n) : (int)(k / n);
    ci          = step_cand(w, l, c);
    i           = (int)(k - (long long)c * n);
}
__device__ __forceinline__ void step_add(const Work &w, int l, int ci) {
    w.list[l * w.ncand + atomicAdd(&w.cnt[l], 1)] = ci;
}

__device__ __forceinline__ unsigned long long win_key(float d, int i) {
    return ((unsigned long long)__float_as_uint(d) << 32) | (unsigned)i;
}

// The nearest point of the stage's subset to each lane's (x, y, z) (`need`: it has one), exact
// where its squared distance is at most lim: subset rank (-1: none found) and squared distance
// d. With TREE the point that the reference's search finds (sm_kdgrid.cuh).
template <bool TREE>
__device__ __forceinline__ int stage_nearest(const Stage &s, float x, float y, float z, float lim,
                                             bool need, float &d) {
    if (TREE)
        return smk::lanes_kd_nearest(s.tree, s.treeM, s.G, s.tposOf, s.rankOf, *s.exc, x, y, z, lim,
                                     need, &d);
    return lanes_nn_walk(s.G, x, y, z, lim, need, &d);
}

// K1: correspondences of the (candidate, source point) items of the step's candidates. A warp
// takes up to 32 items, spread over the launch so that the far-off points, whose searches are
// the long ones, fall on many warps: it loads, moves and stores them a lane each and searches for
// them one after the other. (What surrounds a search was a quarter of its instructions when the
// whole warp did it for each item: ten launches of the large scene 219 -> 201 us; in reference
// order, where the root paths are a lane's too, 705 -> 563 us.) The CTAs are one resident wave,
// so that the launches after the last candidate stopped cost little: 9 us for a CTA per 8 points
// of every candidate, 3 us now. In reference order (TREE) a pair is what findClosestPoint
// (util.cpp:603-626) returns: a one-nearest search of the reduced k-d tree with the tree's
// pruning; one beyond the rejection distance is dropped, so the search is needed up to that
// distance only.
template <bool TREE>
__global__ void __launch_bounds__(kT, TREE ? 3 : 4)
    k_corr(Work w, Stage s, int it, unsigned tag) {
    chain_enter(); // launched chained
    const int       lane  = threadIdx.x & 31;
    const int       l     = step_list(it);
    const long long items = (long long)step_count(w, l) * s.n;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        w.cnt[step_list(it + 2)] = 0; // (the last step's: k_update adds to the next one's)
        *(volatile unsigned long long *)w.heard =
            ((unsigned long long)tag << 32) | (unsigned)step_count(w, l);
        if (w.live)
            atomicAdd(w.live, (unsigned long long)items);
    }
    const long long warps = (long long)gridDim.x * kW;
    for (long long base = blockIdx.x * kW + (threadIdx.x >> 5); base < items; base += 32 * warps) {
        const long long k    = base + lane * warps;
        const bool      have = k < items;
        int             ci = 0, i = 0;
        if (have)
            step_item(w, l, k, s.n, ci, i);
        const size_t o   = (size_t)ci * w.maxSrc + i;
        const Cand  &C   = w.cand[ci];
        float4       x   = make_float4(0.f, 0.f, 0.f, 0.f);
        float        lim = s.rej2;
        if (have) {
            // written by this candidate's previous iteration of this stage (not in the first), a
            // rank of this stage's subset or -1
            const int    jp = it > 0 ? w.nnPrev[o] : -1;
            const float4 sp = s.src[i];
            float4       qp = make_float4(0.f, 0.f, 0.f, 0.f);
            if (jp >= 0 && jp < s.nDst)
                qp = s.dPos[jp];
            smi::pose_apply(C.M, sp.x, sp.y, sp.z, x.x, x.y, x.z);
            // the last iteration's nearest point of this stage bounds the search exactly
            if (jp >= 0 && jp < s.nDst)
                lim = fminf(lim, smm::dist2(x.x, x.y, x.z, qp.x, qp.y, qp.z));
        }
        float     d;
        const int j = stage_nearest<TREE>(s, x.x, x.y, x.z, lim, have, d); // subset rank
        if (have) {
            const bool   ok = j >= 0 && d <= s.rej2;
            const float4 sn = s.srcN[i];
            float4       y;
            smi::pose_rotate(C.M, sn.x, sn.y, sn.z, y.x, y.y, y.z);
            w.nnPrev[o] = j;
            x.w         = d;
            y.w         = 0.0f;
            w.x4[o]     = x;
            w.n4[o]     = y;
            w.nnId[o]   = ok ? j : -1;
            w.nnR[o]    = ok ? j : -1;
            if (ok)
                atomicMin(&w.win[(size_t)ci * w.maxDst + j], win_key(d, i));
        }
    }
}

// The reductions of one refinement iteration run in one thread-block cluster of kRC CTAs
// (kR threads each) per candidate, with the fixed layout of sm_icp.h: slot t (CTA t / kR,
// thread t % kR) sums, with Kahan, the terms of the pairs i = t, t + kIcpSlots, ... in
// ascending order; each CTA merges its slots by the tree (warp shfl_down offsets 16..1, then
// warp 0 over the warp partials, offsets kRW/2..1) and publishes its totals in its shared
// memory; rank 0 reads the kRC partials through distributed shared memory and merges them
// by the block tree (offsets kRC/2..1). No global fence or counter between CTAs, and the
// centroids, the normal equations and the solve share one launch.
//
// The warp tree of many sums: at each offset a lane takes only half of the sums it still holds
// (the lower half in the lower lanes), so 32 sums take 31 merges a lane instead of 160; the
// merges and their operands are those of the plain tree. The tree over the warps and the one
// over the CTAs run a lane per sum, serially in registers. (27 sums by the plain trees, every
// lane merging all of them, made a third of the launch.)
__device__ __forceinline__ smi::KahanF shfl_xor(const smi::KahanF &v, int off) {
    smi::KahanF o;
    o.s = __shfl_xor_sync(0xffffffffu, v.s, off);
    o.c = __shfl_xor_sync(0xffffffffu, v.c, off);
    return o;
}

// W <= 32 sums padded to P = 2^k: the tree's root of sum l * P / 32 ends on lane l (for P < 32
// on the first of 32 / P lanes).
template <int P, int OFF> __device__ __forceinline__ void warp_tree(smi::KahanF (&v)[P]) {
    const bool high = (threadIdx.x & OFF) != 0;
    if constexpr (P > 1) {
        smi::KahanF h[P / 2];
#pragma unroll
        for (int k = 0; k < P / 2; k++) {
            const smi::KahanF keep = high ? v[P / 2 + k] : v[k];
            const smi::KahanF got  = shfl_xor(high ? v[k] : v[P / 2 + k], OFF);
            h[k]                   = high ? got : keep;  // the lower lane's partial
            h[k].merge(high ? keep : got);
        }
        if constexpr (OFF > 1)
            warp_tree<P / 2, OFF / 2>(h);
        v[0] = h[0];
    } else {
        const smi::KahanF got = shfl_xor(v[0], OFF);
        smi::KahanF       r   = high ? got : v[0];
        r.merge(high ? v[0] : got);
        v[0] = r;
        if constexpr (OFF > 1)
            warp_tree<1, OFF / 2>(v);
    }
}

// The block's totals of W sums (v: padded to P): lane k < W of warp 0 returns the k-th.
template <int W, int P>
__device__ __forceinline__ smi::KahanF block_tree(smi::KahanF (&v)[P], float (*red)[W][2]) {
    constexpr int G = 32 / P; // lanes per sum after the warp tree
    const int     lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    warp_tree<P, 16>(v);
    if (lane % G == 0 && lane / G < W) {
        red[wp][lane / G][0] = v[0].s;
        red[wp][lane / G][1] = v[0].c;
    }
    __syncthreads();
    smi::KahanF t;
    t.init();
    if (wp == 0 && lane < W) {
        smi::KahanF p[kRW];
#pragma unroll
        for (int r = 0; r < kRW; r++) {
            p[r].s = red[r][lane][0];
            p[r].c = red[r][lane][1];
        }
#pragma unroll
        for (int off = kRW / 2; off >= 1; off >>= 1)
#pragma unroll
            for (int r = 0; r < off; r++)
                p[r].merge(p[r + off]);
        t = p[0];
    }
    __syncthreads(); // red may be reused
    return t;
}

__device__ __forceinline__ int block_sum_int(int x, int *red) {
    x = __reduce_add_sync(0xffffffffu, x);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = x;
    __syncthreads();
    int t = 0;
    for (int k = 0; k < kRW; k++)
        t += red[k];
    __syncthreads();
    return t;
}

// Rank 0's warp 0: lane k < W merges the cluster's kRC published partials of sum k (read through
// distributed shared memory) by the block tree.
template <int W>
__device__ __forceinline__ smi::KahanF cluster_merge(cg::cluster_group &cl, float (*part)[2]) {
    const int   lane = threadIdx.x & 31;
    smi::KahanF p[kRC];
#pragma unroll
    for (int r = 0; r < kRC; r++) {
        p[r].init();
        if (lane < W) {
            const float *rp = cl.map_shared_rank(&part[lane][0], (unsigned)r);
            p[r].s          = rp[0];
            p[r].c          = rp[1];
        }
    }
#pragma unroll
    for (int off = kRC / 2; off >= 1; off >>= 1)
#pragma unroll
        for (int r = 0; r < off; r++)
            p[r].merge(p[r + off]);
    return p[0];
}

// K2: pair selection (the closest source point per scene point: the atomicMin winner), pair
// count and centroids, then the normal-equation terms of the pairs and the FP64 solve.
__global__ void __cluster_dims__(kRC, 1, 1) __launch_bounds__(kR) k_fit(Work w, Stage s, int it) {
    chain_enter(); // launched chained
    __shared__ float red[kRW][smi::kNumSystem][2];
    __shared__ float part[smi::kNumSystem][2]; // this CTA's totals, read by rank 0
    __shared__ int   ired[kRW];
    __shared__ int   pcnt;
    __shared__ float sPQ[6]; // rank 0: the centroids, read by every CTA
    __shared__ int   sTotal;
    cg::cluster_group cl = cg::this_cluster();
    const int         rk = (int)cl.block_rank();
    const int         l  = step_list(it);
    if ((int)(blockIdx.x / kRC) >= step_count(w, l))
        return; // (the whole cluster: one candidate)
    const int     ci   = step_cand(w, l, blockIdx.x / kRC);
    Cand         &C    = w.cand[ci];
    int          *nnId = w.nnId + (size_t)ci * w.maxSrc;
    const int    *nnR  = w.nnR + (size_t)ci * w.maxSrc;
    const float4 *x4   = w.x4 + (size_t)ci * w.maxSrc;
    const float4 *n4   = w.n4 + (size_t)ci * w.maxSrc;
    const int     slot = rk * kR + threadIdx.x;
    smi::KahanF   m[8]; // 6 sums
    for (int k = 0; k < 8; k++)
        m[k].init();
    // a thread's pairs i = slot, slot + kIcpSlots, ... in ascending order, kFitU of them
    // loaded at once (their loads are independent; the sums still take them in order)
    int cnt = 0;
    for (int base = slot; base < s.n; base += kFitU * smi::kIcpSlots) {
        int                r[kFitU];
        float4             x[kFitU], q[kFitU];
        unsigned long long wk[kFitU];
#pragma unroll
        for (int u = 0; u < kFitU; u++) {
            const int i = base + u * smi::kIcpSlots;
            r[u]        = i < s.n ? nnR[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < kFitU; u++) {
            wk[u] = 0ull;
            if (r[u] >= 0) {
                x[u]  = x4[base + u * smi::kIcpSlots];
                wk[u] = w.win[(size_t)ci * w.maxDst + r[u]];
                q[u]  = s.dPos[r[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kFitU; u++) {
            const int i = base + u * smi::kIcpSlots;
            if (r[u] < 0)
                continue;
            if (wk[u] != win_key(x[u].w, i)) {
                nnId[i] = -1; // this thread reads it again below
                continue;
            }
            cnt++;
            m[0].add(x[u].x);
            m[1].add(x[u].y);
            m[2].add(x[u].z);
            m[3].add(q[u].x);
            m[4].add(q[u].y);
            m[5].add(q[u].z);
        }
    }
    const int cntB = block_sum_int(cnt, ired);
    const smi::KahanF mt = block_tree<6>(m, reinterpret_cast<float (*)[6][2]>(&red[0][0][0]));
    if (threadIdx.x < 6) {
        part[threadIdx.x][0] = mt.s;
        part[threadIdx.x][1] = mt.c;
    }
    if (threadIdx.x == 0)
        pcnt = cntB;
    cl.sync(); // the partials are published
    if (rk == 0 && threadIdx.x < 32) {
        const smi::KahanF mm    = cluster_merge<6>(cl, part);
        int               total = 0;
        for (int r = 0; r < kRC; r++)
            total += *cl.map_shared_rank(&pcnt, (unsigned)r);
        if (threadIdx.x < 6) {
            const float c      = smm::fdiv(mm.value(), (float)total);
            sPQ[threadIdx.x]   = c;
            if (threadIdx.x < 3)
                C.Pm[threadIdx.x] = c;
            else
                C.Qm[threadIdx.x - 3] = c;
        }
        if (threadIdx.x == 0) {
            C.cnt  = total;
            sTotal = total;
        }
    }
    cl.sync(); // rank 0 has read the partials and published the centroids
    const float *pq    = cl.map_shared_rank(sPQ, 0u);
    const float  Pm0   = pq[0], Pm1 = pq[1], Pm2 = pq[2];
    const float  Qm0   = pq[3], Qm1 = pq[4], Qm2 = pq[5];
    const int    total = *cl.map_shared_rank(&sTotal, 0u);
    cl.sync(); // every CTA has read rank 0's centroids (rank 0 may leave after this)
    if (total < 6)
        return;
    smi::KahanF v[32]; // kNumSystem sums
    for (int k = 0; k < 32; k++)
        v[k].init();
    for (int base = slot; base < s.n; base += 2 * smi::kIcpSlots) {
        int    id[2];
        float4 x[2], xn[2], q[2], qn[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = base + u * smi::kIcpSlots;
            id[u]       = i < s.n ? nnId[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (id[u] >= 0) {
                const int i = base + u * smi::kIcpSlots;
                x[u]        = x4[i];
                xn[u]       = n4[i];
                q[u]        = s.dPos[id[u]];
                qn[u]       = s.dNrm[id[u]];
            }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (id[u] < 0)
                continue;
            float t[smi::kNumSystem];
            smi::system_terms(x[u].x - Pm0, x[u].y - Pm1, x[u].z - Pm2, q[u].x - Qm0,
                              q[u].y - Qm1, q[u].z - Qm2, xn[u].x + qn[u].x, xn[u].y + qn[u].y,
                              xn[u].z + qn[u].z, t);
            for (int k = 0; k < smi::kNumSystem; k++)
                v[k].add(t[k]);
        }
    }
    const smi::KahanF vt = block_tree<smi::kNumSystem>(v, red);
    if (threadIdx.x < smi::kNumSystem) {
        part[threadIdx.x][0] = vt.s;
        part[threadIdx.x][1] = vt.c;
    }
    cl.sync(); // the partials are published
    if (rk == 0 && threadIdx.x < 32) {
        const float tot = cluster_merge<smi::kNumSystem>(cl, part).value();
        cl.sync(); // (rank 0 has read every partial: the others may leave)
        float sys[smi::kNumSystem];
#pragma unroll
        for (int k = 0; k < smi::kNumSystem; k++)
            sys[k] = __shfl_sync(0xffffffffu, tot, k);
        const float pm[3] = {Pm0, Pm1, Pm2}, qm[3] = {Qm0, Qm1, Qm2};
        smi::solve_step_warp(sys, pm, qm, C.step.m);
    } else {
        cl.sync();
    }
}

// K4: residual distance of each pair after the step, items as in K1 (ten launches of the large
// scene in reference order 528 -> 452 us)
template <bool TREE>
__global__ void __launch_bounds__(kT, TREE ? 3 : 5) k_resid(Work w, Stage s, int it) {
    chain_enter(); // launched chained
    const int       l     = step_list(it);
    const long long items = (long long)step_count(w, l) * s.n;
    const long long warps = (long long)gridDim.x * kW;
    for (long long base = blockIdx.x * kW + (threadIdx.x >> 5); base < items; base += 32 * warps) {
        const long long k    = base + (threadIdx.x & 31) * warps;
        bool            have = k < items;
        int             ci = 0, i = 0;
        if (have)
            step_item(w, l, k, s.n, ci, i);
        const size_t o = (size_t)ci * w.maxSrc + i;
        float        y0 = 0.f, y1 = 0.f, y2 = 0.f, lim = 0.f, d;
        if (have) {
            const Cand  &C = w.cand[ci];
            const int    j = w.nnId[o];
            const float4 x = w.x4[o];
            have           = C.cnt >= 6 && j >= 0;
            if (have) {
                const float4 q = s.dPos[j];
                smi::pose_apply(C.step, x.x, x.y, x.z, y0, y1, y2);
                // the pair's scene point bounds the search exactly
                lim = smm::dist2(y0, y1, y2, q.x, q.y, q.z);
            }
        }
        stage_nearest<TREE>(s, y0, y1, y2, lim, have, d);
        if (have)
            w.resid[o] = smm::fsqrt(d);
    }
}

// K5: mean residual, the regist loop logic (icp.cpp:233-272), winner reset; one cluster per
// candidate (the same layout as K2), rank 0's warp 0 runs the logic and lists the candidate for
// the next iteration if it goes on
__global__ void __cluster_dims__(kRC, 1, 1) __launch_bounds__(kR) k_update(Work w, Stage s, int it) {
    chain_enter(); // launched chained
    __shared__ float red[kRW][1][2];
    __shared__ float part[1][2];
    cg::cluster_group cl = cg::this_cluster();
    const int         rk = (int)cl.block_rank();
    const int         l  = step_list(it);
    if ((int)(blockIdx.x / kRC) >= step_count(w, l))
        return;
    const int  ci   = step_cand(w, l, blockIdx.x / kRC);
    Cand      &C    = w.cand[ci];
    const int  slot = rk * kR + threadIdx.x;
    const int  lane = threadIdx.x & 31;
    const int *nnR  = w.nnR + (size_t)ci * w.maxSrc;
    // the step's product with the pose, an entry per lane (used below if the step is taken)
    float moved = 0.0f;
    if (rk == 0 && threadIdx.x < 12)
        moved = smi::pose_mul_entry(C.step.m, C.M.m, lane);
    for (int i = slot; i < s.n; i += smi::kIcpSlots)
        if (nnR[i] >= 0)
            w.win[(size_t)ci * w.maxDst + nnR[i]] = ~0ull;
    const int cnt = C.cnt;
    float     mse = FLT_MAX;
    if (cnt >= 6) {
        const float *D    = w.resid + (size_t)ci * w.maxSrc;
        const int   *nnId = w.nnId + (size_t)ci * w.maxSrc;
        smi::KahanF  v[1];
        v[0].init();
        for (int base = slot; base < s.n; base += kFitU * smi::kIcpSlots) {
            int   id[kFitU];
            float d[kFitU];
#pragma unroll
            for (int u = 0; u < kFitU; u++) {
                const int i = base + u * smi::kIcpSlots;
                id[u]       = i < s.n ? nnId[i] : -1;
                d[u]        = i < s.n ? D[i] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kFitU; u++)
                if (id[u] >= 0)
                    v[0].add(d[u]);
        }
        const smi::KahanF vt = block_tree<1>(v, red);
        if (threadIdx.x == 0) {
            part[0][0] = vt.s;
            part[0][1] = vt.c;
        }
        cl.sync(); // the partials are published
        if (rk == 0 && threadIdx.x < 32)
            mse = __shfl_sync(0xffffffffu, smm::fdiv(cluster_merge<1>(cl, part).value(), (float)cnt), 0);
        cl.sync(); // rank 0 has read every partial: the others may leave
    }
    if (rk != 0 || threadIdx.x >= 32)
        return;
    const int   done   = C.iterations;
    const float resMse = C.resMse;
    __syncwarp();
    if (lane == 0 && w.trace && done < kTraceIters) {
        float *t = w.trace + (size_t)ci * kTraceFloats + (s.traceOff * kTraceIters + done) * 4;
        t[0]     = (float)cnt;
        t[1]     = mse;
        t[2]     = cnt >= 6 ? C.Pm[0] : -1.0f;
        t[3]     = cnt >= 6 ? C.step.m[3] : 0.0f;
    }
    int  stop = 0;
    bool take = false;
    if (cnt < 6) {
        stop = 1;
    } else {
        if (mse < s.mseMin)
            stop = 1;
        const float rate = smm::fdiv(resMse - mse, resMse);
        if (rate < 0.05f)
            stop = 1;
        if (done >= s.iters)
            stop = 1;
        take = rate > 0.0f;
    }
    if (take && lane < 12)
        C.M.m[lane] = moved;
    if (lane == 0) {
        if (cnt > 6 && mse < s.mseMax)
            C.converged = 1;
        if (take)
            C.resMse = mse;
        if (cnt >= 6)
            C.iterations = done + 1;
        if (!stop && done + 1 < s.iters)
            step_add(w, step_list(it + 1), ci);
    }
}

__global__ void k_init(Work w, const float *__restrict__ cands, float voteThreshold, int sparse) {
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci < 2 * (kStepLists + 1))
        w.cnt[ci] = 0; // the candidate counts of both stages
    if (ci >= w.ncand)
        return;
    Cand        &C = w.cand[ci];
    const float *P = cands + (size_t)ci * smi::kPoseFloats;
    for (int e = 0; e < 12; e++)
        C.M.m[e] = P[e];
    C.keep   = C.M;
    C.score  = P[17];
    C.status = P[17] < voteThreshold ? 1 : 0;
    C.active = (C.status == 0 && sparse) ? 1 : 0;
    if (w.trace)
        for (int e = 0; e < kTraceFloats; e++)
            w.trace[(size_t)ci * kTraceFloats + e] = -1.0f;
}

__global__ void k_stage_begin(Work w, int iters) {
    chain_enter(); // launched chained
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= w.ncand)
        return;
    Cand &C      = w.cand[ci];
    C.resMse     = FLT_MAX;
    C.iterations = 0;
    C.converged  = 0;
    C.inl        = 0;
    if (C.active && iters > 0)
        step_add(w, 0, ci);
}

// After a refinement: failed candidates get their status; converged ones keep the pose and are
// listed for the scoring.
__global__ void k_stage_end(Work w, int failStatus) {
    chain_enter(); // launched chained
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= w.ncand)
        return;
    Cand &C = w.cand[ci];
    if (!C.active)
        return;
    if (!C.converged) {
        C.status = failStatus;
        C.active = 0;
    } else {
        C.keep = C.M;
        step_add(w, kStepLists, ci);
    }
}

// Inliers of each candidate left (list kStepLists): source points with a scene point closer than the
// scoring distance (warp_any_within); with TREE the scene point that the reference's search of the
// whole tree returns (inliner, util.cpp:628-641). A warp takes consecutive points, 32 at a time a
// lane each, and adds to a candidate's count once per 32 (two launches of the large scene in
// reference order 250 -> 158 us).
template <bool TREE>
__global__ void __launch_bounds__(kT, TREE ? 3 : 5)
    k_inliers(Work w, const float4 *__restrict__ src, int n, HGridView F, float r2,
              smk::KdView t, int treeM, const int *__restrict__ treePos,
              const float *__restrict__ exc) {
    chain_enter(); // launched chained
    const long long items = (long long)step_count(w, kStepLists) * n;
    const long long warps = (long long)gridDim.x * kW, per = (items + warps - 1) / warps;
    long long       k   = (blockIdx.x * (long long)kW + (threadIdx.x >> 5)) * per;
    const long long end = k + per < items ? k + per : items;
    const int       lane = threadIdx.x & 31;
    for (; k < end; k += 32) {
        const bool have = k + lane < end;
        int        ci = -1, i = 0;
        float      x = 0.f, y = 0.f, z = 0.f;
        if (have) {
            step_item(w, kStepLists, k + lane, n, ci, i);
            const float4 p = src[i];
            smi::pose_apply(w.cand[ci].M, p.x, p.y, p.z, x, y, z);
        }
        bool in = false;
        if (TREE) {
            float     d;
            const int j = smk::lanes_kd_nearest(t, treeM, F, treePos, nullptr, *exc, x, y, z, r2, have, &d);
            in          = j >= 0 && d < r2;
        } else {
            for (unsigned m = __ballot_sync(0xffffffffu, have); m; m &= m - 1u) {
                const int  l = __ffs(m) - 1;
                const bool h = warp_any_within(F, __shfl_sync(0xffffffffu, x, l), __shfl_sync(0xffffffffu, y, l),
                                               __shfl_sync(0xffffffffu, z, l), r2);
                if (lane == l)
                    in = h;
            }
        }
        // a count per candidate of the 32 points
        const unsigned same = __match_any_sync(0xffffffffu, ci);
        const unsigned hits = __ballot_sync(0xffffffffu, in) & same;
        if (hits && lane == __ffs(same) - 1)
            atomicAdd(&w.cand[ci].inl, __popc(hits));
    }
}

__global__ void k_score(Work w, int ncand, int n, float minScore, int failStatus, int slot) {
    chain_enter(); // launched chained
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= ncand)
        return;
    Cand &C = w.cand[ci];
    if (!C.active)
        return;
    if (w.trace)
        w.trace[(size_t)ci * kTraceFloats + 2 * kTraceIters * 4 + slot] = (float)C.inl;
    C.score = fminf(1.0f, smm::fdiv((float)C.inl, (float)n));
    if (C.score < minScore) {
        C.status = failStatus;
        C.active = 0;
    }
}

__global__ void k_finish(Work w, int ncand, int refine, float minScore, int *status, float *score,
                         float *pose) {
    chain_enter(); // launched chained
    const int ci = blockIdx.x * blockDim.x + threadIdx.x;
    if (ci >= ncand)
        return;
    Cand &C = w.cand[ci];
    if (!C.status && refine && C.score < minScore)
        C.status = 5;
    status[ci] = C.status;
    score[ci]  = C.status ? -1.0f : C.score;
    for (int e = 0; e < 12; e++)
        pose[(size_t)ci * 12 + e] = C.keep.m[e];
}


// CTAs of a launch over `items` warps' worth of work: at most one resident wave (perSm CTAs of kT
// threads, the kernels' launch bounds).
int wave(const Ctx &c, long long items, int perSm) {
    int nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    return (int)std::max<long long>(1, std::min<long long>((items + kW - 1) / kW, (long long)nsm * perSm));
}

// The candidates of the refinement step of this tag, once it has begun: a poll of page-locked
// memory, which ends with the stream's work (-1: not told, the caller goes on).
int step_heard(Ctx &c, unsigned tag) {
    const volatile unsigned long long *word =
        reinterpret_cast<const volatile unsigned long long *>(c.hostCounts + kHostStep);
    for (int spin = 1;; spin++) {
        const unsigned long long v = *word;
        if ((unsigned)(v >> 32) == tag)
            return (int)(unsigned)v;
        if (spin % 1024 == 0) {
            const cudaError_t e = cudaStreamQuery(c.stream);
            if (e == cudaErrorNotReady)
                continue;
            SM_CUDA(e);
            const unsigned long long last = *word;
            return (unsigned)(last >> 32) == tag ? (int)(unsigned)last : -1;
        }
    }
}

// Most stages end after two or three steps: their candidates converge, whatever the limit. A
// step is launched while the one before it runs, and none after one that found no candidates left
// (four empty launches otherwise for every step up to the limit: a refinement limited to 15
// dense steps took 0.49 ms, 0.43 now).
void run_stage(Ctx &c, const Work &w, const Stage &s) {
    const int       gc   = w.ncand * kRC; // reductions: a cluster per candidate
    const bool      tree = s.tree.nd != nullptr;
    const long long all  = (long long)w.ncand * s.n;
    const int gCorr = wave(c, all, tree ? 3 : 4), gResid = wave(c, all, tree ? 3 : 5);
    launch_chained(c, k_stage_begin, nblocks(w.ncand, 128), 128, 0, w, s.iters);
    for (int it = 0; it < s.iters; it++) {
        if (it >= 2 && step_heard(c, c.stepTag) == 0)
            break;
        const unsigned tag = c.stepTag = std::max(c.stepTag + 1u, 1u);
        cudaEvent_t    t0  = c.clock.begin(c.stream);
        if (tree)
            launch_chained(c, k_corr<true>, gCorr, kT, 0, w, s, it, tag);
        else
            launch_chained(c, k_corr<false>, gCorr, kT, 0, w, s, it, tag);
        c.clock.end(c.stream, t0, KernelClock::kCorr, 0.0); // bytes from the live count
        t0 = c.clock.begin(c.stream);
        launch_chained(c, k_fit, gc, kR, 0, w, s, it);
        c.clock.end(c.stream, t0, KernelClock::kFit, 0.0);
        t0 = c.clock.begin(c.stream);
        if (tree)
            launch_chained(c, k_resid<true>, gResid, kT, 0, w, s, it);
        else
            launch_chained(c, k_resid<false>, gResid, kT, 0, w, s, it);
        c.clock.end(c.stream, t0, KernelClock::kResid, 0.0);
        t0 = c.clock.begin(c.stream);
        launch_chained(c, k_update, gc, kR, 0, w, s, it);
        c.clock.end(c.stream, t0, KernelClock::kUpdate, 0.0);
    }
}

} // namespace

void icp_all(Ctx &c, const Model &m, const IcpScene &sc, const IcpParams &p, const float *cands,
             int ncand, int *status, float *score, float *pose, float *trace) {
    if (ncand <= 0)
        return;
    Work w;
    w.maxSrc = std::max(std::max(m.ns, m.nr), 1);
    w.maxDst = std::max(std::max(sc.sampled.m, sc.resampled.m), 1);
    w.cand   = c.arena.get<Cand>("icp.cand", ncand);
    w.nnId   = c.arena.get<int>("icp.nnId", (size_t)ncand * w.maxSrc);
    w.nnR    = c.arena.get<int>("icp.nnR", (size_t)ncand * w.maxSrc);
    w.nnPrev = c.arena.get<int>("icp.nnPrev", (size_t)ncand * w.maxSrc);
    w.x4     = c.arena.get<float4>("icp.x4", (size_t)ncand * w.maxSrc);
    w.n4     = c.arena.get<float4>("icp.n4", (size_t)ncand * w.maxSrc);
    w.resid  = c.arena.get<float>("icp.resid", (size_t)ncand * w.maxSrc);
    w.win    = c.arena.get<unsigned long long>("icp.win", (size_t)ncand * w.maxDst);
    w.trace  = trace;
    w.live   = nullptr;
    w.heard  = reinterpret_cast<unsigned long long *>(c.hostCounts + kHostStep);
    *(volatile unsigned long long *)w.heard = 0; // (tags start at 1)
    if (c.clock.on) {
        w.live = c.arena.get<unsigned long long>("icp.live", 1);
        SM_CUDA(cudaMemsetAsync(w.live, 0, sizeof(unsigned long long), c.stream));
    }
    constexpr int sparseIters = 5;
    constexpr int lists       = kStepLists + 1; // of the sparse stage, then of the dense one
    w.ncand = ncand;
    w.cnt   = c.arena.get<int>("icp.cnt", 2 * lists);
    w.list  = c.arena.get<int>("icp.list", (size_t)2 * lists * ncand);
    SM_CUDA(cudaMemsetAsync(w.win, 0xff, (size_t)ncand * w.maxDst * 8, c.stream));
    k_init<<<nblocks(ncand, 128), 128, 0, c.stream>>>(w, cands, p.voteThreshold, p.sparse);
    SM_LAUNCH_CHECK();
    const float rej2 = p.rejectDist * p.rejectDist;
    const float sc2  = p.scoreDist * p.scoreDist;
    const bool tree = sc.tree != nullptr;
    auto inliers = [&](const float4 *src, int n) {
        const int g = wave(c, (long long)ncand * n, tree ? 3 : 5);
        if (tree)
            launch_chained(c, k_inliers<true>, g, kT, 0, w, src, n, sc.full.view(), sc2,
                           sc.tree->view(nullptr, sc.pos, nullptr, sc.tpF), sc.tree->m,
                           (const int *)sc.tree->treePos, sc.exc + 2);
        else
            launch_chained(c, k_inliers<false>, g, kT, 0, w, src, n, sc.full.view(), sc2,
                           smk::KdView{}, 0, (const int *)nullptr, (const float *)nullptr);
    };
    if (p.sparse) {
        Stage s{m.sp, m.sn, m.ns, sc.sampled.view(), sc.posS, sc.nrmS, sc.sampled.m, sparseIters,
                p.sampleStep * 0.5f, p.sampleStep, rej2, 0};
        if (tree) {
            s.tree   = sc.tree->view(sc.ioiS, sc.pos, sc.neS, sc.tpS);
            s.treeM  = sc.tree->m;
            s.rankOf = sc.rankS;
            s.tposOf = sc.tposS;
            s.exc    = sc.exc;
        }
        run_stage(c, w, s);
        launch_chained(c, k_stage_end, nblocks(ncand, 128), 128, 0, w, 2);
        inliers(m.sp, m.ns);
        launch_chained(c, k_score, nblocks(ncand, 128), 128, 0, w, ncand, m.ns, p.minScore, 3,
                       0);
        if (p.dense) {
            Stage d{m.rp, m.rn, m.nr, sc.resampled.view(), sc.posR, sc.nrmR, sc.resampled.m,
                    p.denseSteps, p.reSampleStep * 0.5f, p.sampleStep, rej2, 1};
            if (tree) {
                d.tree   = sc.tree->view(sc.ioiR, sc.pos, sc.neR, sc.tpR);
                d.treeM  = sc.tree->m;
                d.rankOf = sc.rankR;
                d.tposOf = sc.tposR;
                d.exc    = sc.exc + 1;
            }
            w.cnt += lists;
            w.list += (size_t)lists * ncand;
            run_stage(c, w, d);
            launch_chained(c, k_stage_end, nblocks(ncand, 128), 128, 0, w, 4);
            inliers(m.rp, m.nr);
            launch_chained(c, k_score, nblocks(ncand, 128), 128, 0, w, ncand, m.nr, p.minScore,
                           5, 1);
        }
    }
    launch_chained(c, k_finish, nblocks(ncand, 128), 128, 0, w, ncand,
                   (p.sparse || p.dense) ? 1 : 0, p.minScore, status, score, pose);
}

} // namespace sm
