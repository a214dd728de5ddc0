// kdtree.cu - the reference-order k-d tree on the GPU: build, searches, and the greedy
// sampler in tree order.
//
// Reference counterparts: KDTreeVectorOfVectorsAdaptor (kdtree/kdtree.h:52-161) over the
// vendored nanoflann (kdtree/nanoflann.hpp: divideTree 1120-1176, middleSplit_ 1290-1339,
// planeSplit 1352-1393, searchLevel 1846-1930) and samplePointCloud (util.cpp:107-139).
//
// Build. nanoflann splits a node's index range [left, right) recursively: the cut axis is
// the one of largest point spread among the axes whose box side is within (1 - 1e-5) of
// the widest, the cut value the box middle clamped to the points' range, and the range is
// reordered by two in-place Hoare passes (values < cut to the front, then values <= cut).
// Each pass has a closed form: with T the number of elements that go to the front, the
// j-th element of the front part that does not belong there is swapped with the j-th
// element from the back of the rear part that does - so a pass is a prefix sum and a
// batch of disjoint swaps. The GPU builds all nodes of one depth at once (segments of the
// position array, one kernel per step, prefix sums over the whole array) until every open
// range holds at most kSmall points; those finish in one CTA each, in shared memory, with
// the same steps. Node bounds are then tightened bottom-up (divlow/divhigh are the
// children's tight bounds, the root box becomes the tight box of all points, as nanoflann
// does through its by-reference bbox).
//
// Greedy sampling in tree order. The reference keeps a point unless an already kept point's
// radius search found it, visiting points in tree position order (util.cpp:107-139). Each
// point's fate depends only on the earlier points within the step: it is dropped once a
// kept one reaches it, and kept once all of them are decided and none of the kept ones
// reaches it. The GPU decides them through a device queue of grid cells, each waiting for the
// open point that blocks its first one (below, k_sp_run), so decisions
// travel along the dependency chains of the greedy order. "Reaches" is the reference's
// radius search membership: squared distance below step^2 and not pruned by the search
// above the point's leaf - decided by walking the point's root-to-leaf path
// (smk::kd_reaches) unless the distance bound proves the pruning cannot happen (points
// moved by normal estimation can leave their leaf's box).
#include <climits>
#include <cmath>

#include "sm_kdgrid.cuh"
#include "sm_kdtree.cuh"
#include "sm_scan.cuh"
#include "sm_stages.h"

namespace sm {
using namespace smd;
using smk::KdView;

namespace {

struct GridParamsK {
    float org[3], g;
    int   dim[3];
};

constexpr int kSmall    = 1024; // ranges of at most this many points finish in one CTA
constexpr int kSmallSeg = 96;   // open sub-ranges per level inside that CTA (> 10 points each: <= 93)

// An open range of the build (one future node) and its split.
struct Seg {
    int   left, right, node, cutfeat;
    float lo[3], hi[3]; // the box nanoflann passes down (parent box cut at the split)
    int   mn[3], mx[3]; // ordered-int min / max of the points (computeMinMax)
    float cutval;
    int   index;    // split offset from left
    int   child[2]; // next-level segment of each child (-1: leaf or small range)
    int   depth;    // depth of the node (root 0)
};

// Lanes add their point's ordered coordinates to the bounds of their range (s < 0: none);
// a warp whose lanes share one range reduces first and adds once.
template <class S>
__device__ __forceinline__ void add_bounds(S *seg, int s, const float4 &p) {
    const int  o[3] = {f2ord(p.x), f2ord(p.y), f2ord(p.z)};
    const int  s0   = __shfl_sync(0xffffffffu, s, 0);
    const bool same = __all_sync(0xffffffffu, s == s0);
    if (same) {
        if (s0 < 0)
            return;
        int lo[3], hi[3];
        for (int a = 0; a < 3; a++) {
            lo[a] = __reduce_min_sync(0xffffffffu, o[a]);
            hi[a] = __reduce_max_sync(0xffffffffu, o[a]);
        }
        if ((threadIdx.x & 31) == 0)
            for (int a = 0; a < 3; a++) {
                atomicMin(&seg[s0].mn[a], lo[a]);
                atomicMax(&seg[s0].mx[a], hi[a]);
            }
        return;
    }
    if (s >= 0)
        for (int a = 0; a < 3; a++) {
            atomicMin(&seg[s].mn[a], o[a]);
            atomicMax(&seg[s].mx[a], o[a]);
        }
}

// The same by a whole CTA: where every thread with a point names one range, the CTA adds once
// (at the first levels every warp of the launch would add to the same few words: 95 us a level).
template <class S>
__device__ __forceinline__ void add_bounds_block(S *seg, int s, const float4 &p) {
    __shared__ int sOne, lo[3], hi[3];
    if (threadIdx.x == 0)
        sOne = -1;
    if (threadIdx.x < 3) {
        lo[threadIdx.x] = INT_MAX;
        hi[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
    if (s >= 0)
        sOne = s; // (any one of them)
    __syncthreads();
    const int one = sOne;
    if (!__syncthreads_and(s < 0 || s == one)) {
        add_bounds(seg, s, p);
        return;
    }
    if (one < 0)
        return;
    const int o[3] = {f2ord(p.x), f2ord(p.y), f2ord(p.z)};
    for (int a = 0; a < 3; a++) {
        const int l = __reduce_min_sync(0xffffffffu, s >= 0 ? o[a] : INT_MAX);
        const int h = __reduce_max_sync(0xffffffffu, s >= 0 ? o[a] : INT_MIN);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&lo[a], l);
            atomicMax(&hi[a], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        atomicMin(&seg[one].mn[threadIdx.x], lo[threadIdx.x]);
        atomicMax(&seg[one].mx[threadIdx.x], hi[threadIdx.x]);
    }
}

__device__ __forceinline__ float coord_of(const float4 &p, int a) {
    return a == 0 ? p.x : (a == 1 ? p.y : p.z);
}

// middleSplit_'s choice of axis and cut value (nanoflann.hpp:1290-1329).
__device__ void choose_cut(const float lo[3], const float hi[3], const int mn[3], const int mx[3],
                           int &cutfeat, float &cutval) {
    const float EPS     = 0.00001f;
    float       maxSpan = hi[0] - lo[0];
    for (int i = 1; i < 3; ++i) {
        const float span = hi[i] - lo[i];
        if (span > maxSpan)
            maxSpan = span;
    }
    float maxSpread = -1.0f, minElem = 0.0f, maxElem = 0.0f;
    cutfeat = 0;
    for (int i = 0; i < 3; ++i) {
        const float span = hi[i] - lo[i];
        if (span > (1.0f - EPS) * maxSpan) {
            const float a = ord2f(mn[i]), b = ord2f(mx[i]);
            const float spread = b - a;
            if (spread > maxSpread) {
                cutfeat   = i;
                maxSpread = spread;
                minElem   = a;
                maxElem   = b;
            }
        }
    }
    const float splitVal = (lo[cutfeat] + hi[cutfeat]) / 2.0f;
    if (splitVal < minElem)
        cutval = minElem;
    else if (splitVal > maxElem)
        cutval = maxElem;
    else
        cutval = splitVal;
}

// middleSplit_'s split offset from the two partition limits (nanoflann.hpp:1333-1338).
__device__ __forceinline__ int split_index(int count, int lim1, int lim2) {
    if (lim1 > count / 2)
        return lim1;
    if (lim2 < count / 2)
        return lim2;
    return count / 2;
}

__device__ __forceinline__ int4 leaf_node(int l, int r) { return make_int4(l, r, -1, 0); }

// ---- top levels: one kernel per step over the whole position array -------------------
// Control words: nodes, small ranges, error, then per level its open ranges and whether a
// point lies on a cut (else the second pass has nothing to do). The levels' launches are chained
// and sized by bounds; the host looks at the counts every kKdLevels levels only. (One round trip,
// two counter copies, a flag kernel per pass and ordinary launches a level a call on 0.92 M
// points took 9.35 ms, with these 8.82; the build is some 2.2 ms of launches.)
enum { kKdNodes = 0, kKdSmallN = 1, kKdErr = 2, kKdOpen = 8, kKdOnCut = 8 + 2 * smk::kMaxDepth };
constexpr int kKdCtl    = kKdOnCut + 2 * smk::kMaxDepth;
constexpr int kKdLevels = 4;
static_assert((63 - kKdOpen) % kKdLevels != 0, "the counts' word 63 is sync_checked's");

__global__ void k_kd_root(Seg *seg, Seg *small, int m, Box box, int4 *nd, int *parent, int *ctl) {
    Seg s{};
    s.left  = 0;
    s.right = m;
    s.node  = 0;
    s.depth = 0;
    for (int a = 0; a < 3; a++) {
        s.lo[a] = box.mn[a];
        s.hi[a] = box.mx[a];
        s.mn[a] = INT_MAX;
        s.mx[a] = INT_MIN;
    }
    s.child[0] = s.child[1] = -1;
    seg[0]        = s;
    parent[0]     = -1;
    ctl[kKdNodes] = 1;
    ctl[kKdOpen]  = m > kSmall ? 1 : 0; // open ranges of the first level
    if (m <= smk::kLeafMax) {
        nd[0] = leaf_node(0, m);
    } else if (m <= kSmall) {
        small[0]       = s; // the whole cloud is one small range
        ctl[kKdSmallN] = 1;
    }
}

__global__ void k_kd_init(const float4 *__restrict__ pos, const int *__restrict__ ids, int m,
                          float4 *__restrict__ rec, int *__restrict__ segOf, Seg *__restrict__ seg) {
    const int i  = blockIdx.x * blockDim.x + threadIdx.x;
    float4    p  = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < m) {
        const int id = ids[i];
        p            = pos[id];
        rec[i]       = make_float4(p.x, p.y, p.z, __int_as_float(id));
        segOf[i]     = 0;
    }
    add_bounds_block(seg, i < m ? 0 : -1, p);
}

__global__ void k_kd_cut(Seg *__restrict__ seg, const int *__restrict__ nseg) {
    chain_enter(); // launched chained
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= *nseg)
        return;
    Seg &S = seg[s];
    choose_cut(S.lo, S.hi, S.mn, S.mx, S.cutfeat, S.cutval);
}

// pass 1: value < cut over [left, right); pass 2: value <= cut over [left + lim1, right)
__device__ __forceinline__ int pass_start(const Seg &S, int pass, const int *g1) {
    return pass == 1 ? S.left : S.left + (g1[S.right] - g1[S.left]);
}

// A pass's flags as the values of a scan (the flag of position i is then g[i + 1] - g[i]),
// evaluated in position order and handed over as bits. Pass 1 notes points on a cut; without any
// pass 2 is skipped.
struct KdFlags {
    const float4 *rec;
    const int    *segOf;
    const Seg    *seg;
    const int    *nseg, *g1;
    int          *onCut;
    int           pass, m;
    __device__ __forceinline__ bool skip() const { return *nseg == 0 || (pass == 2 && *onCut == 0); }
    __device__ __forceinline__ void load(long long tile, long long, int (&v)[kScanIpt]) const {
        __shared__ uint32_t bits[kScanTile / 32];
        bool                on = false;
#pragma unroll
        for (int k = 0; k < kScanIpt; k++) {
            const int j = k * kScanBs + threadIdx.x, i = (int)tile + j;
            bool      f = false;
            const int s = i < m ? segOf[i] : -1;
            if (s >= 0) {
                const Seg &S = seg[s];
                if (pass == 1 || i >= pass_start(S, 2, g1)) {
                    const float x = coord_of(rec[i], S.cutfeat);
                    f             = pass == 1 ? x < S.cutval : x <= S.cutval;
                    on            = on || x == S.cutval;
                }
            }
            const uint32_t b = __ballot_sync(0xffffffffu, f);
            if ((threadIdx.x & 31) == 0)
                bits[j >> 5] = b;
        }
        if (pass == 1 && on)
            *onCut = 1;
        __syncthreads();
        const uint32_t b = bits[threadIdx.x / 4] >> ((threadIdx.x & 3) * 8);
#pragma unroll
        for (int k = 0; k < kScanIpt; k++)
            v[k] = (b >> k) & 1u;
    }
};

// The open range of position i in a pass: its start there, false when i takes no part.
__device__ __forceinline__ bool kd_part(const KdFlags &F, int i, int &a, int &right) {
    if (i >= F.m)
        return false;
    const int s = F.segOf[i];
    if (s < 0)
        return false;
    const Seg &S = F.seg[s];
    a            = pass_start(S, F.pass, F.g1);
    right        = S.right;
    return i >= a;
}

// The back part's misplaced elements record their positions by rank from the back.
__global__ void k_kd_rank(KdFlags F, const int *__restrict__ g, int *__restrict__ badR) {
    chain_enter(); // launched chained
    if (F.skip())
        return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int       a, right;
    if (!kd_part(F, i, a, right))
        return;
    const int ga = g[a], gi = g[i], T = g[right] - ga;
    if (i - a >= T && g[i + 1] != gi)
        badR[a + (T - (gi - ga) - 1)] = i;
}

// The front part's misplaced elements swap with their partners (disjoint pairs).
__global__ void k_kd_swap(KdFlags F, float4 *__restrict__ rec, const int *__restrict__ g,
                          const int *__restrict__ badR) {
    chain_enter(); // launched chained
    if (F.skip())
        return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int       a, right;
    if (!kd_part(F, i, a, right))
        return;
    const int ga = g[a], gi = g[i], T = g[right] - ga;
    if (i - a < T && g[i + 1] == gi) {
        const int    p = badR[a + (i - a - (gi - ga))];
        const float4 x = rec[i];
        rec[i]         = rec[p];
        rec[p]         = x;
    }
}

// Children of every open range: nodes, leaves, small ranges and next-level ranges.
__global__ void k_kd_children(Seg *__restrict__ seg, const int *__restrict__ nseg,
                              const int *__restrict__ onCut, const int *__restrict__ g1,
                              const int *__restrict__ g2, int4 *__restrict__ nd,
                              int *__restrict__ parent, int *__restrict__ ctl,
                              Seg *__restrict__ next, int *__restrict__ nnext,
                              Seg *__restrict__ small) {
    chain_enter(); // launched chained
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= *nseg)
        return;
    Seg      &S     = seg[s];
    const int count = S.right - S.left;
    const int lim1  = g1[S.right] - g1[S.left];
    const int lim2  = *onCut ? lim1 + (g2[S.right] - g2[S.left + lim1]) : lim1;
    const int index = split_index(count, lim1, lim2);
    S.index         = index;
    const int c1    = atomicAdd(&ctl[kKdNodes], 2);
    nd[S.node]      = make_int4(0, 0, c1 | (S.cutfeat << 30), S.left + index);
    if (S.depth + 1 >= smk::kMaxDepth)
        atomicExch(&ctl[kKdErr], 1);
    for (int k = 0; k < 2; k++) {
        const int l = k == 0 ? S.left : S.left + index;
        const int r = k == 0 ? S.left + index : S.right;
        Seg       C{};
        C.left  = l;
        C.right = r;
        C.node  = c1 + k;
        for (int a = 0; a < 3; a++) {
            C.lo[a] = S.lo[a];
            C.hi[a] = S.hi[a];
            C.mn[a] = INT_MAX;
            C.mx[a] = INT_MIN;
        }
        if (k == 0)
            C.hi[S.cutfeat] = S.cutval;
        else
            C.lo[S.cutfeat] = S.cutval;
        C.child[0] = C.child[1] = -1;
        C.depth    = S.depth + 1;
        parent[c1 + k]          = S.node;
        S.child[k]              = -1;
        if (r - l <= smk::kLeafMax) {
            nd[c1 + k] = leaf_node(l, r);
        } else if (r - l <= kSmall) {
            small[atomicAdd(&ctl[kKdSmallN], 1)] = C;
        } else {
            const int id = atomicAdd(nnext, 1);
            next[id]     = C;
            S.child[k]   = id;
        }
    }
}

// Next-level segment of every position, and the next level's point bounds.
__global__ void k_kd_advance(const float4 *__restrict__ rec, int *__restrict__ segOf, int m,
                             const Seg *__restrict__ seg, const int *__restrict__ nseg,
                             Seg *__restrict__ next) {
    chain_enter(); // launched chained
    if (*nseg == 0)
        return;
    const int i  = blockIdx.x * blockDim.x + threadIdx.x;
    int       ns = -1;
    float4    p  = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < m) {
        const int s = segOf[i];
        if (s >= 0) {
            const Seg &S = seg[s];
            ns           = S.child[i < S.left + S.index ? 0 : 1];
            segOf[i]     = ns;
            p            = rec[i];
        }
    }
    add_bounds_block(next, ns, p);
}

// ---- small ranges: one CTA of 1024 threads, one position per thread -------------------
struct SubSeg {
    int   left, right, node, cutfeat;
    float lo[3], hi[3];
    int   mn[3], mx[3];
    float cutval;
    int   index, child[2], depth;
};

__global__ void __launch_bounds__(kSmall)
    k_kd_small(const Seg *__restrict__ small, float4 *__restrict__ rec, int4 *__restrict__ nd,
               int *__restrict__ parent, int *__restrict__ nodeCount, int *__restrict__ err) {
    __shared__ float4 r[kSmall];
    __shared__ short  sid[kSmall];
    __shared__ int    sc1[kSmall + 1], sc2[kSmall + 1], bad[kSmall];
    __shared__ SubSeg ss[2][kSmallSeg];
    __shared__ int    nsub[2];
    __shared__ int    wsum[33];
    const Seg S0  = small[blockIdx.x];
    const int n   = S0.right - S0.left;
    const int t   = threadIdx.x;
    if (t < n)
        r[t] = rec[S0.left + t];
    sid[t] = (short)(t < n ? 0 : -1);
    if (t == 0) {
        SubSeg z{};
        z.left  = 0;
        z.right = n;
        z.node  = S0.node;
        z.depth = S0.depth;
        for (int a = 0; a < 3; a++) {
            z.lo[a] = S0.lo[a];
            z.hi[a] = S0.hi[a];
            z.mn[a] = INT_MAX;
            z.mx[a] = INT_MIN;
        }
        ss[0][0] = z;
        nsub[0]  = 1;
        nsub[1]  = 0;
    }
    __syncthreads();
    int cur = 0;
    while (nsub[cur] > 0) {
        SubSeg *L = ss[cur];
        SubSeg *N = ss[cur ^ 1];
        // point bounds per open range
        add_bounds(L, sid[t], r[t]);
        __syncthreads();
        if (t < nsub[cur])
            choose_cut(L[t].lo, L[t].hi, L[t].mn, L[t].mx, L[t].cutfeat, L[t].cutval);
        __syncthreads();
        // (without a point on its range's cut the second pass moves nothing, and the flags' scan is
        // a ballot: the large scene's 1,578 ranges took 448 us, now 383)
        bool onCut = false;
        for (int pass = 1; pass <= (onCut ? 2 : 1); pass++) {
            int *sc = pass == 1 ? sc1 : sc2;
            int  f  = 0;
            int  a  = 0;
            bool on = false;
            if (sid[t] >= 0) {
                const SubSeg &Q = L[sid[t]];
                a = pass == 1 ? Q.left : Q.left + (sc1[Q.right] - sc1[Q.left]);
                if (t >= a) {
                    const float x = coord_of(r[t], Q.cutfeat);
                    f             = pass == 1 ? (x < Q.cutval) : (x <= Q.cutval);
                    on            = x == Q.cutval;
                }
            }
            const unsigned fb = __ballot_sync(0xffffffffu, f);
            if ((t & 31) == 0)
                wsum[t >> 5] = __popc(fb);
            const bool any = __syncthreads_or(on);
            onCut          = pass == 1 ? any : onCut;
            const int wi   = warp_incl_scan(wsum[t & 31]);
            const int wb   = __shfl_sync(0xffffffffu, wi, (t >> 5) - 1);
            sc[t]          = ((t >> 5) ? wb : 0) + __popc(fb & ((1u << (t & 31)) - 1u));
            if (t == kSmall - 1)
                sc[kSmall] = wi;
            __syncthreads();
            int T = 0, lt = 0;
            if (sid[t] >= 0 && t >= a) {
                const SubSeg &Q = L[sid[t]];
                T               = sc[Q.right] - sc[a];
                lt              = sc[t] - sc[a];
                if (f && t - a >= T)
                    bad[a + (T - lt - 1)] = t;
            }
            __syncthreads();
            float4 mine = r[t], other = mine;
            int    p    = -1;
            if (sid[t] >= 0 && t >= a && !f && t - a < T) {
                p     = bad[a + (t - a - lt)];
                other = r[p];
            }
            __syncthreads();
            if (p >= 0) {
                r[t] = other;
                r[p] = mine;
            }
            __syncthreads();
        }
        if (t == 0)
            nsub[cur ^ 1] = 0;
        __syncthreads();
        if (t < nsub[cur]) {
            SubSeg   &Q     = L[t];
            const int count = Q.right - Q.left;
            const int lim1  = sc1[Q.right] - sc1[Q.left];
            const int lim2  = onCut ? lim1 + (sc2[Q.right] - sc2[Q.left + lim1]) : lim1;
            const int index = split_index(count, lim1, lim2);
            Q.index         = index;
            const int c1    = atomicAdd(nodeCount, 2);
            nd[Q.node]      = make_int4(0, 0, c1 | (Q.cutfeat << 30), S0.left + Q.left + index);
            if (Q.depth + 1 >= smk::kMaxDepth)
                atomicExch(err, 1);
            for (int k = 0; k < 2; k++) {
                const int l = k == 0 ? Q.left : Q.left + index;
                const int rr = k == 0 ? Q.left + index : Q.right;
                parent[c1 + k] = Q.node;
                Q.child[k]     = -1;
                if (rr - l <= smk::kLeafMax) {
                    nd[c1 + k] = leaf_node(S0.left + l, S0.left + rr);
                } else {
                    const int id = atomicAdd(&nsub[cur ^ 1], 1);
                    if (id >= kSmallSeg) {
                        atomicExch(err, 2);
                        continue;
                    }
                    SubSeg C{};
                    C.left  = l;
                    C.right = rr;
                    C.node  = c1 + k;
                    C.depth = Q.depth + 1;
                    for (int a = 0; a < 3; a++) {
                        C.lo[a] = Q.lo[a];
                        C.hi[a] = Q.hi[a];
                        C.mn[a] = INT_MAX;
                        C.mx[a] = INT_MIN;
                    }
                    if (k == 0)
                        C.hi[Q.cutfeat] = Q.cutval;
                    else
                        C.lo[Q.cutfeat] = Q.cutval;
                    N[id]      = C;
                    Q.child[k] = id;
                }
            }
        }
        __syncthreads();
        if (t == 0 && nsub[cur ^ 1] > kSmallSeg)
            nsub[cur ^ 1] = 0; // overflow reported through err; stop
        if (sid[t] >= 0) {
            const SubSeg &Q = L[sid[t]];
            sid[t]          = (short)Q.child[t < Q.left + Q.index ? 0 : 1];
        }
        __syncthreads();
        cur ^= 1;
    }
    if (t < n)
        rec[S0.left + t] = r[t];
}

// ---- finish: tight boxes bottom-up, split bounds, per-position indexes ----------------
__global__ void k_kd_finish(int4 *__restrict__ nd, const int *__restrict__ parent,
                            const int *__restrict__ nodeCount, const float4 *__restrict__ rec,
                            float *__restrict__ box, int *__restrict__ arrive,
                            int *__restrict__ vacc, int *__restrict__ leafOf,
                            int *__restrict__ treePos) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= *nodeCount)
        return;
    const int4 n = nd[v];
    if (!smk::is_leaf(n))
        return;
    float lo[3], hi[3];
    {
        const float4 p = rec[n.x];
        lo[0] = hi[0] = p.x;
        lo[1] = hi[1] = p.y;
        lo[2] = hi[2] = p.z;
    }
    for (int i = n.x; i < n.y; i++) {
        const float4 p  = rec[i];
        const float  c3[3] = {p.x, p.y, p.z};
        for (int a = 0; a < 3; a++) {
            if (lo[a] > c3[a])
                lo[a] = c3[a];
            if (hi[a] < c3[a])
                hi[a] = c3[a];
        }
        const int id = __float_as_int(p.w);
        vacc[i]      = id;
        leafOf[i]    = v;
        treePos[id]  = i;
    }
    for (int a = 0; a < 3; a++) {
        box[6 * v + a]     = lo[a];
        box[6 * v + 3 + a] = hi[a];
    }
    // the second child to finish tightens the parent
    int u = v;
    for (;;) {
        const int p = parent[u];
        if (p < 0)
            return;
        __threadfence();
        if (atomicAdd(&arrive[p], 1) == 0)
            return;
        __threadfence();
        const int4 pn = nd[p];
        const int  c1 = smk::child1_of(pn), cf = smk::divfeat_of(pn);
        const volatile float *b1 = box + 6 * c1;
        const volatile float *b2 = box + 6 * (c1 + 1);
        for (int a = 0; a < 3; a++) {
            box[6 * p + a]     = fminf(b1[a], b2[a]);
            box[6 * p + 3 + a] = fmaxf(b1[3 + a], b2[3 + a]);
        }
        nd[p].x = __float_as_int(b1[3 + cf]); // divlow: child1's upper bound on the cut axis
        nd[p].y = __float_as_int(b2[cf]);     // divhigh: child2's lower bound
        u       = p;
    }
}

// ---- greedy sampling in tree order ---------------------------------------------------
// A point is kept once every earlier point (tree order) within the step is decided and none of
// the kept ones dropped it; a kept point drops the later points its search reaches. So only
// kept points search their neighbourhood, and what is left is the dependency chain. Points sit
// in cells of about the step, in tree order within a cell; only a cell's first open point can
// be the next decided. A cell is a work item: the warp that holds it looks for a blocker of
// its first open point - an open earlier point within the step - and either files the cell
// under the blocker (the blocker's decision queues it again) or keeps the point, drops what it
// reaches, queues the cells filed under any of these, and goes on with the next point. A cell
// is in one place at a time: queued, held, or filed. The earliest open point of all has no
// blocker, so there is always a cell to go on with, and a warp waits for queue slots only.
// (Handling every point through the queue, with a neighbourhood pass per point to count its
// earlier neighbours and one when it was decided, took 7.8 + 7.3 ms for the large scene's
// 0.92 M points at steps 4.3 and 1.4 mm, where 7,000 and 56,000 are kept; now 1.26 + 1.35 ms.
// The rest is the chain: about 150 decisions of 8 us in a row at the larger step.)
constexpr int       kSpBs     = 256;
constexpr long long kSpIdle   = 1ll << 22; // polls of an unwritten queue slot before giving up
constexpr int       kSpUnroll = 4;         // neighbourhood entries in flight per lane
// CTAs per SM (2 measured best of 1, 2 and 4 beside the voting stage: the warps that hold cells
// at once), nanoseconds between two looks at a queue slot, and words between two control words
// (on one line, with every waiting warp reading it at each look, a decision took 40 us instead
// of 10: the large scene's two long samplings 3.3 + 4.4 ms instead of 1.2 + 1.6 ms)
constexpr int       kSpCtas     = 2;
constexpr int       kSpSleep    = 100;
constexpr int       kSpCtl      = 32;
constexpr int       kSpUnlinked = -2;      // a filed cell's link until it is stored
constexpr long long kSpCells    = 1ll << 25; // most cells of the dense table (128 MB)
constexpr float     kSpCoarse   = 1.5f;      // above so many steps a side its cells are hashed ones

// Hashed cells, where a dense table of cells just above the step would not fit: a cell's number is
// its slot in an open-addressed table of its key, 21 bits of each coordinate. Coordinates count
// cells from 0 and wrap, so a cell can hold points 2^21 cells apart, which are no more than further
// candidates; beyond 2^50 cells, where points within the step share the coordinate itself, they are
// drawn from its bits. So cells stay just above the step whatever the extent. (Coarser cells of the
// dense table instead, as the extent grows: every decision goes through all points of 27 cells, and
// two points 100 m away made the sampling of 10,000 others at 1.4 mm take 842 ms, against 0.2 ms.)
constexpr int                kSpWrap = 21;
constexpr unsigned long long kSpMask = (1ull << kSpWrap) - 1;
__device__ __forceinline__ unsigned long long sp_wrapped(float x, double perCell) {
    const double q = floor((double)x * perCell);
    return (fabs(q) < 1125899906842624.0 ? (unsigned long long)(long long)q
                                         : smm::mix64((unsigned long long)__float_as_uint(x))) &
           kSpMask;
}

struct SampleArgs {
    KdView          t;
    int             dim[3];
    const unsigned long long *keys; // hashed cells: slot -> key (all ones: empty)
    uint32_t        slotMask;
    const float4   *ent;      // cell runs: {x, y, z, tree position bits}, tree order in a run
    const float    *sure;     // the entries' sure_reach
    const int      *cellRank; // cell -> occupied rank (-1: empty)
    const int      *cellList; // occupied rank -> cell
    const int      *cellEnd;  // occupied rank -> end of its run of the entries
    // occupied rank -> an entry of its run that no open one comes before, and its tree position
    unsigned long long *cur;
    int            *dec;      // per entry: 0 open, 1 kept, 2 dropped
    int            *filed;    // per entry: first cell filed under it (-1: none)
    int            *nextCell; // per occupied rank: the next cell filed under the same entry
    int            *ring;     // queue of cells (-1: slot not written)
    unsigned        ringMask;
    int            *head, *tail;
    int            *open;     // cells with points not yet decided
    float           r2;
    int            *keptFlag; // per tree position
    int            *err;      // a bounded wait expired
};
__device__ __forceinline__ unsigned long long sp_cur(int k, int pos) {
    return (unsigned long long)(unsigned)pos << 32 | (unsigned)k;
}

__device__ __forceinline__ int ld_vol(const int *p) { return *(const volatile int *)p; }

// Distance of a (moved) point from its leaf's build-time box.
__device__ __forceinline__ double excursion(const float *box, const float4 &p) {
    const float c[3] = {p.x, p.y, p.z};
    double      s    = 0.0;
    for (int a = 0; a < 3; a++) {
        const double lo = box[a], hi = box[3 + a], x = c[a];
        const double o  = x < lo ? lo - x : (x > hi ? x - hi : 0.0);
        s += o * o;
    }
    return sqrt(s);
}

// Squared distance below which a radius search of radius^2 r2 surely reaches a point that lies
// `e` outside its leaf's build-time box: the search's lower bound at any node above the leaf is at
// most (distance + e)^2 (the margins cover the float rounding of the search's running bound and
// of the result). Computed once per point in FP64, so that a test is a float comparison: a test
// with the square root in FP64 waited a microsecond for that pipe.
__device__ __forceinline__ float sure_reach(float r2, double e) {
    const double s = sqrt((double)r2 * (1.0 - 1e-4)) - e;
    return s > 0.0 ? (float)(s * s * (1.0 - 1e-6)) : 0.0f;
}

// Whether the radius search from kept point q reaches the point p at tree position ip
// (radiusSearch membership, nanoflann.hpp:1736-1749): distance first; the walk down the path only
// near the radius or for points that left their leaf's box.
__device__ __forceinline__ bool reaches(const SampleArgs &a, const float4 &q, const float4 &p,
                                        int ip, float sure) {
    const float qq[3] = {q.x, q.y, q.z};
    const float d     = smk::eval_metric(qq, p);
    if (!(d < a.r2))
        return false;
    if (d < sure)
        return true;
    uint64_t key;
    return smk::kd_sure(a.t, qq, ip, a.r2) || smk::kd_reaches(a.t, qq, ip, a.r2, &key);
}

// The cell of each tree position (noCell where reduce() excluded it).
__global__ void k_sp_keys(const int *__restrict__ vaccA, const float4 *__restrict__ pos, int m,
                          GridParamsK gp, uint32_t noCell, uint32_t *__restrict__ key,
                          uint32_t *__restrict__ val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const int id = vaccA[i];
    uint32_t  k  = noCell;
    if (id >= 0) {
        const float4 p  = pos[id];
        const int    cx = smg::coord(p.x, gp.org[0], gp.g, gp.dim[0]);
        const int    cy = smg::coord(p.y, gp.org[1], gp.g, gp.dim[1]);
        const int    cz = smg::coord(p.z, gp.org[2], gp.g, gp.dim[2]);
        k               = (uint32_t)((cz * gp.dim[1] + cy) * gp.dim[0] + cx);
    }
    key[i] = k;
    val[i] = (uint32_t)i;
}

// The same with hashed cells, which enter the table (of at least twice as many slots as points).
__global__ void k_sp_keys_hashed(const int *__restrict__ vaccA, const float4 *__restrict__ pos, int m,
                                 double perCell, unsigned long long *__restrict__ keys,
                                 uint32_t slotMask, uint32_t noCell, uint32_t *__restrict__ key,
                                 uint32_t *__restrict__ val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const int id = vaccA[i];
    uint32_t  k  = noCell;
    if (id >= 0) {
        const float4             p = pos[id];
        const unsigned long long w = sp_wrapped(p.x, perCell) | sp_wrapped(p.y, perCell) << kSpWrap |
                                     sp_wrapped(p.z, perCell) << (2 * kSpWrap);
        uint32_t h = (uint32_t)smm::mix64(w) & slotMask;
        for (uint32_t q = 0; q <= slotMask; q++) {
            const unsigned long long prev = atomicCAS(&keys[h], ~0ull, w);
            if (prev == ~0ull || prev == w)
                break;
            h = (h + 1) & slotMask;
        }
        k = h;
    }
    key[i] = k;
    val[i] = (uint32_t)i;
}

__global__ void k_sp_heads(const uint32_t *__restrict__ key, int m, uint32_t noCell,
                           int *__restrict__ head) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > m)
        return;
    head[k] = (k < m && key[k] != noCell && (k == 0 || key[k - 1] != key[k])) ? 1 : 0;
}

// The cells' runs, and the runs' points in run order: {x, y, z, tree position bits}, with the
// distance a search surely reaches it at.
__global__ void k_sp_cells(const uint32_t *__restrict__ key, const uint32_t *__restrict__ sortPos,
                           int m, uint32_t noCell, const int *__restrict__ head,
                           const int *__restrict__ rank, const float *__restrict__ nodeBox,
                           const int *__restrict__ leafOf, int *__restrict__ cellRank,
                           int *__restrict__ cellList, int *__restrict__ cellEnd,
                           float4 *__restrict__ ent, float *__restrict__ sure, SampleArgs a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m || key[k] == noCell)
        return;
    const int r = rank[k] + head[k] - 1; // the run's occupied rank
    if (head[k]) {
        cellRank[key[k]] = r;
        cellList[r]      = (int)key[k];
        a.cur[r]         = sp_cur(k, (int)sortPos[k]);
    }
    if (k == m - 1 || key[k + 1] != key[k])
        cellEnd[r] = k + 1;
    if (k == m - 1 || key[k + 1] == noCell) // (the active entries sort first)
        *a.open = r + 1;
    const int    ip = (int)sortPos[k];
    const float4 p  = a.t.pos[a.t.vacc[ip]];
    ent[k]          = make_float4(p.x, p.y, p.z, __int_as_float(ip));
    sure[k]         = sure_reach(a.r2, excursion(nodeBox + 6 * (size_t)leafOf[ip], p));
    a.dec[k]        = 0;
    a.filed[k]      = -1;
}

// Entry of flattened neighbourhood index t: binary search over the lanes' prefixes.
__device__ __forceinline__ int nb_entry(int t, int excl, int nb) {
    int lo = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int mid = lo + step;
        const int ev  = __shfl_sync(0xffffffffu, excl, mid & 31);
        if (mid < 27 && ev <= t)
            lo = mid;
    }
    return __shfl_sync(0xffffffffu, nb, lo) + (t - __shfl_sync(0xffffffffu, excl, lo));
}

// Memory order. A cell moves between warps through the ring: pushed after a fence, taken by an
// acquire. Filing stores the link and then looks at the entry's decision, deciding stores the
// decision and then looks at the entry's list, each with a sequentially consistent fence
// between: whichever comes second sees the other. A kept point's mark is a release by one lane
// after a warp barrier, so that it covers the drops of all lanes; a warp that finds no blocker
// fences and meets at a barrier before one lane looks at the point's own state, so that any lane's
// look at such a mark counts.
__device__ __forceinline__ void fence_sc() { asm volatile("fence.sc.gpu;" ::: "memory"); }
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ int  exch_acquire(int *p, int v) {
    int o;
    asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(o) : "l"(p), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ int exch_release(int *p, int v) {
    int o;
    asm volatile("atom.release.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(o) : "l"(p), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Queues the cells filed under entry j. A slot is written once its last reader has emptied it:
// at most every cell is queued, and the ring holds twice as many.
__device__ __forceinline__ void sp_wake(const SampleArgs &a, int j) {
    int c = exch_acquire(&a.filed[j], -1);
    if (c < 0)
        return;
    fence_acq_rel();
    while (c >= 0) {
        // (a cell enters the list before its link is stored)
        int nx = ld_vol(&a.nextCell[c]);
        for (long long it = 0; nx == kSpUnlinked; it++) {
            if (it > kSpIdle) {
                atomicExch(a.err, 1);
                return;
            }
            nx = ld_vol(&a.nextCell[c]);
        }
        const int cid = a.cellList[c];
        int      *s   = &a.ring[(unsigned)atomicAdd(a.tail, 1) & a.ringMask];
        for (long long it = 0; atomicCAS(s, -1, cid) != -1; it++)
            if (it > kSpIdle) {
                atomicExch(a.err, 1);
                return;
            }
        c = nx;
    }
}

// The next queued cell, by lane 0: -1 when every point is decided (or a wait expired).
__device__ __forceinline__ int sp_take(const SampleArgs &a) {
    int *s = &a.ring[(unsigned)atomicAdd(a.head, 1) & a.ringMask];
    for (long long it = 0;; it++) {
        if (ld_vol(s) >= 0) {
            const int c = exch_acquire(s, -1);
            if (c >= 0)
                return c;
        }
        // (thousands of warps may wait here: the shared words are read now and then only)
        if ((it & 15) == 15) {
            if (ld_vol(a.open) <= 0 || ld_vol(a.err))
                return -1;
            if (it > kSpIdle) {
                atomicExch(a.err, 1);
                return -1;
            }
        }
        __nanosleep(kSpSleep);
    }
}

// The runs around a cell, a neighbour per lane (-1: none, lane kSpOwn: the cell itself). A take
// is a chain of dependent loads, so what a later step needs is read with the one before it.
constexpr int kSpOwn = 13;
struct SpRuns {
    int nr, nend;      // occupied rank, end of its run
    int from, pos;     // its first open entry (or one before it) and that one's tree position
    int nb, excl, tot; // this pass's begin, exclusive prefix of the lengths and their sum
    template <bool HASHED> __device__ __forceinline__ void find(const SampleArgs &a, int cid) {
        const int lane = threadIdx.x & 31;
        const int dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
        nr   = -1;
        nend = from = pos = 0;
        if (HASHED) {
            const unsigned long long c = a.keys[cid];
            const unsigned long long w =
                ((c + (long long)dx) & kSpMask) |
                (((c >> kSpWrap) + (long long)dy) & kSpMask) << kSpWrap |
                (((c >> (2 * kSpWrap)) + (long long)dz) & kSpMask) << (2 * kSpWrap);
            uint32_t           h = (uint32_t)smm::mix64(w) & a.slotMask;
            unsigned long long k = lane < 27 ? a.keys[h] : ~0ull;
            while (k != w && k != ~0ull) { // (a free slot ends every probe)
                h = (h + 1) & a.slotMask;
                k = a.keys[h];
            }
            if (k != ~0ull)
                nr = a.cellRank[h];
        } else {
            const int cx = cid % a.dim[0], cy = (cid / a.dim[0]) % a.dim[1],
                      cz = cid / (a.dim[0] * a.dim[1]);
            const int x = cx + dx, y = cy + dy, z = cz + dz;
            if (lane < 27 && x >= 0 && y >= 0 && z >= 0 && x < a.dim[0] && y < a.dim[1] &&
                z < a.dim[2])
                nr = a.cellRank[(z * a.dim[1] + y) * a.dim[0] + x];
        }
        if (nr >= 0)
            nend = a.cellEnd[nr];
        look(a);
    }
    __device__ __forceinline__ void look(const SampleArgs &a) {
        if (nr < 0)
            return;
        const unsigned long long w = *(const volatile unsigned long long *)&a.cur[nr];
        from = (int)(unsigned)w;
        pos  = (int)(w >> 32);
    }
    // each run from its first open entry, the cell's own from entry `own`; with before >= 0 runs
    // whose first open point's tree position is above it count as empty
    __device__ __forceinline__ void begin(int own, int before) {
        const bool self = (threadIdx.x & 31) == kSpOwn;
        nb              = self ? own : from;
        const int len   = nr < 0 || (before >= 0 && !self && pos > before) ? 0 : nend - nb;
        const int incl  = warp_incl_scan(len);
        tot             = __shfl_sync(0xffffffffu, incl, 31);
        excl            = incl - len;
    }
    __device__ __forceinline__ int entry(int t) const { return nb_entry(min(t, tot - 1), excl, nb); }
};

// An open entry with tree position below ip within the step of p: -1 when there is none.
__device__ __forceinline__ int sp_blocker(const SampleArgs &a, SpRuns &R, int k, const float4 &p,
                                          int ip) {
    const int   lane = threadIdx.x & 31;
    const float q[3] = {p.x, p.y, p.z};
    R.begin(k, ip - 1);
    for (int base = 0; base < R.tot; base += 32 * kSpUnroll) {
        int    kb[kSpUnroll], dec[kSpUnroll];
        float4 b[kSpUnroll];
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++)
            kb[u] = R.entry(base + u * 32 + lane);
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++) {
            b[u]   = a.ent[kb[u]];
            dec[u] = ld_vol(&a.dec[kb[u]]);
        }
        int last = -1, at = -1; // the lane's latest blocker waits longest: the one to wait for
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++) {
            const int ib = __float_as_int(b[u].w);
            if (base + u * 32 + lane < R.tot && dec[u] == 0 && ib < ip && ib > last &&
                smk::eval_metric(q, b[u]) < a.r2) {
                last = ib;
                at   = kb[u];
            }
        }
        const int w = __reduce_max_sync(0xffffffffu, last);
        if (w >= 0)
            return __shfl_sync(0xffffffffu, at, __ffs(__ballot_sync(0xffffffffu, last == w)) - 1);
    }
    return -1;
}

// Drops the open later points of kept point p's runs from the 1024th on that its search reaches and
// queues the cells filed under them.
__device__ __forceinline__ void sp_drop_far(const SampleArgs &a, const SpRuns &R, const float4 &p,
                                            int ip) {
    const int lane = threadIdx.x & 31;
    for (int base = 1024; base < R.tot; base += 32) {
        const int    kb = R.entry(base + lane);
        const float4 b  = a.ent[kb];
        const bool   go = base + lane < R.tot && __float_as_int(b.w) > ip && ld_vol(&a.dec[kb]) == 0 &&
                        reaches(a, p, b, __float_as_int(b.w), a.sure[kb]);
        if (go)
            *(volatile int *)&a.dec[kb] = 2;
        if (!__any_sync(0xffffffffu, go))
            continue;
        fence_sc();
        if (go && ld_vol(&a.filed[kb]) >= 0)
            sp_wake(a, kb);
    }
}

// Drops the open later points that the search of kept point p (entry k) reaches: a bit of the
// lane for each (bit j: entry 32 j + lane) of the first 1024, for the caller to wake after its
// fence. Those from the 1024th on are woken here.
__device__ __forceinline__ unsigned sp_drop(const SampleArgs &a, SpRuns &R, int k, const float4 &p,
                                            int ip) {
    const int   lane = threadIdx.x & 31;
    const float q[3] = {p.x, p.y, p.z};
    unsigned    drop = 0u;
    R.begin(k + 1, -1);
    for (int base = 0; base < min(R.tot, 1024); base += 32 * kSpUnroll) {
        int    kb[kSpUnroll], dec[kSpUnroll];
        float  sure[kSpUnroll];
        float4 b[kSpUnroll];
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++)
            kb[u] = R.entry(base + u * 32 + lane);
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++) {
            b[u]    = a.ent[kb[u]];
            sure[u] = a.sure[kb[u]];
            dec[u]  = ld_vol(&a.dec[kb[u]]);
        }
#pragma unroll
        for (int u = 0; u < kSpUnroll; u++) {
            const int ib = __float_as_int(b[u].w);
            if (base + u * 32 + lane < R.tot && dec[u] == 0 && ib > ip &&
                smk::eval_metric(q, b[u]) < a.r2 && reaches(a, p, b[u], ib, sure[u])) {
                *(volatile int *)&a.dec[kb[u]] = 2;
                drop |= 1u << (base / 32 + u);
            }
        }
    }
    if (R.tot > 1024)
        sp_drop_far(a, R, p, ip);
    return drop;
}

// Before the queue runs nothing is decided: a warp per cell files it under the first blocker of
// its first point, or queues it. (Through the queue these are a third of its takes, each with the
// queue's fences: the large scene's last sampling took 1.79 ms in k_sp_run alone, now 0.08 ms here
// and 1.27 ms there.)
template <bool HASHED> __global__ void __launch_bounds__(kSpBs) k_sp_first(SampleArgs a) {
    const int lane = threadIdx.x & 31;
    const int n = *a.open, nw = gridDim.x * (kSpBs / 32);
    for (int r = blockIdx.x * (kSpBs / 32) + (threadIdx.x >> 5); r < n; r += nw) {
        SpRuns R{};
        const int cid = a.cellList[r];
        R.find<HASHED>(a, cid);
        const int    k = __shfl_sync(0xffffffffu, R.from, kSpOwn);
        const float4 p = a.ent[k];
        const int    j = sp_blocker(a, R, k, p, __float_as_int(p.w));
        if (lane == 0) {
            if (j >= 0)
                a.nextCell[r] = atomicExch(&a.filed[j], r);
            else
                a.ring[(unsigned)atomicAdd(a.tail, 1) & a.ringMask] = cid;
        }
    }
}

template <bool HASHED> __global__ void __launch_bounds__(kSpBs) k_sp_run(SampleArgs a) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        const int cid = __shfl_sync(0xffffffffu, lane == 0 ? sp_take(a) : 0, 0);
        if (cid < 0)
            return;
        __syncwarp(); // (lane 0's acquire holds for the warp)
        SpRuns R{};
        R.find<HASHED>(a, cid);
        const int r = __shfl_sync(0xffffffffu, R.nr, kSpOwn);
        const int e = __shfl_sync(0xffffffffu, R.nend, kSpOwn);
        int       k = __shfl_sync(0xffffffffu, R.from, kSpOwn);
        for (bool again = false;; again = true) {
            if (again)
                R.look(a);
            // the cell's first open entry
            unsigned open = 0u;
            float4   p;
            for (; k < e; k += 32) {
                const int  kl = min(k + lane, e - 1);
                const bool un = ld_vol(&a.dec[kl]) == 0;
                p             = a.ent[kl];
                open          = __ballot_sync(0xffffffffu, un && k + lane < e);
                if (open)
                    break;
            }
            if (!open) {
                if (lane == 0) {
                    *(volatile unsigned long long *)&a.cur[r] = sp_cur(e, INT_MAX);
                    atomicSub(a.open, 1);
                }
                break;
            }
            const int at = __ffs(open) - 1;
            k += at;
            p.x = __shfl_sync(0xffffffffu, p.x, at);
            p.y = __shfl_sync(0xffffffffu, p.y, at);
            p.z = __shfl_sync(0xffffffffu, p.z, at);
            p.w = __shfl_sync(0xffffffffu, p.w, at);
            const int ip = __float_as_int(p.w);
            if (lane == 0)
                *(volatile unsigned long long *)&a.cur[r] = sp_cur(k, ip);
            const int j = sp_blocker(a, R, k, p, ip);
            if (j >= 0) {
                if (lane == 0) {
                    // file the cell under j; if j was decided meanwhile, whoever takes j's list
                    // (this lane or the one that decided j) queues the cell
                    *(volatile int *)&a.nextCell[r] = kSpUnlinked;
                    *(volatile int *)&a.nextCell[r] = exch_release(&a.filed[j], r);
                    fence_sc();
                    if (ld_vol(&a.dec[j]) != 0)
                        sp_wake(a, j);
                }
                __syncwarp();
                break;
            }
            // no open earlier point within the step. A kept point drops before it counts as
            // decided, so p's own state is final now
            fence_acq_rel();
            __syncwarp();
            if (__shfl_sync(0xffffffffu, lane == 0 ? ld_vol(&a.dec[k]) : 0, 0) != 0)
                continue; // dropped meanwhile: on to the cell's next open entry
            const unsigned drop = sp_drop(a, R, k, p, ip);
            const unsigned any  = __reduce_or_sync(0xffffffffu, drop);
            __syncwarp(); // (every lane's drops)
            if (lane == 0) {
                a.keptFlag[ip] = 1;
                st_release(&a.dec[k], 1);
            }
            fence_sc();
            for (unsigned m = any; m; m &= m - 1u) {
                const int jb = __ffs(m) - 1, kb = R.entry(jb * 32 + lane);
                if (((drop >> jb) & 1u) && ld_vol(&a.filed[kb]) >= 0)
                    sp_wake(a, kb);
            }
            if (lane == 0 && ld_vol(&a.filed[k]) >= 0)
                sp_wake(a, k);
            __syncwarp();
        }
    }
}

__global__ void k_sp_out(const int *__restrict__ flag, const int *__restrict__ pre, int m,
                         const int *__restrict__ vaccA, int *__restrict__ outIds,
                         int *__restrict__ ioi) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const bool kept = flag[i] != 0;
    if (kept)
        outIds[pre[i]] = vaccA[i];
    if (ioi)
        ioi[i] = kept ? vaccA[i] : -1;
}

// ---- k-nearest searches on the tree ------------------------------------------------------
// The k nearest ids of query t < *nq (a device count) in the reference's order (distance, then
// first found), and how many: by a thread over the tree.
__device__ __forceinline__ void kd_knn_query(const KdView &t, const float q[3], int k,
                                             int *__restrict__ nbr, float *__restrict__ dist,
                                             int *__restrict__ cnt) {
    smk::KnnSet<kMaxKnn> rs;
    rs.init(k);
    smk::kd_search(t, q, rs); // (no tree is deeper than its stack: the build refuses them)
    for (int j = 0; j < k; j++) {
        nbr[j] = j < rs.count ? rs.idx[j] : -1;
        if (dist)
            dist[j] = rs.dist[j];
    }
    if (cnt)
        *cnt = rs.count;
}

// One query per thread, at qpos[t].
__global__ void k_kd_knn(KdView t, const float4 *__restrict__ qpos, const int *__restrict__ nq,
                         int k, int *__restrict__ nbr, float *__restrict__ dist) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nq)
        return;
    const float4 p    = qpos[i];
    const float  q[3] = {p.x, p.y, p.z};
    kd_knn_query(t, q, k, nbr + (size_t)i * k, dist + (size_t)i * k, nullptr);
}

// One query per warp over part `part` of a normal estimation's list, answered on the grid of the
// tree's points (sm_kdgrid.cuh); as k_knn (prep.cu).
constexpr int kKnnBs = 256;
__global__ void __launch_bounds__(kKnnBs)
    k_kd_knn_grid(KdView t, int m, HGridView g, const int *__restrict__ treePos, NormalList L,
                  int part, int k, bool grow, const float4 *__restrict__ nrm) {
    const int lane = threadIdx.x & 31;
    const int i    = L.begin(part) +
                  (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (i >= L.end(part))
        return;
    const float4 p = t.pos[L.list[i]];
    int          id;
    int          n   = smk::warp_kd_knearest(t, m, g, treePos, p.x, p.y, p.z, k, &id);
    int         *out = L.nbr + (size_t)i * k;
    if (n < 0) {
        if (lane == 0) {
            const float q[3] = {p.x, p.y, p.z};
            kd_knn_query(t, q, k, out, nullptr, L.nbrCnt + i);
        }
        __syncwarp();
        n  = L.nbrCnt[i];
        id = lane < n ? out[lane] : -1;
    } else {
        if (lane < k)
            out[lane] = lane < n ? id : -1;
        if (lane == 0)
            L.nbrCnt[i] = n;
    }
    if (grow)
        L.add_neighbour(lane < n, id, nrm);
}

// The same by the tree's own search, a thread per query, where the grid's cells are coarse.
__global__ void k_kd_knn_list(KdView t, NormalList L, int part, int k, bool grow,
                              const float4 *__restrict__ nrm) {
    const int lane = threadIdx.x & 31;
    const int i0   = L.begin(part) + (blockIdx.x * blockDim.x + threadIdx.x - lane);
    const int end  = L.end(part);
    if (i0 >= end)
        return;
    if (i0 + lane < end) {
        const float4 p    = t.pos[L.list[i0 + lane]];
        const float  q[3] = {p.x, p.y, p.z};
        kd_knn_query(t, q, k, L.nbr + (size_t)(i0 + lane) * k, nullptr, L.nbrCnt + i0 + lane);
    }
    if (!grow)
        return;
    __syncwarp();
    for (int i = i0; i < min(i0 + 32, end); i++) {
        const bool in = lane < L.nbrCnt[i];
        L.add_neighbour(in, in ? L.nbr[(size_t)i * k + lane] : -1, nrm);
    }
}

// ---- the voting stage's candidates (ppf.cpp:273-276) --------------------------------------
// Candidate r (id cand[r], the reduced tree's r-th point): its tree position, and the squared
// distance below which a radius search of radius^2 r2 surely reaches it: the search's bound
// above the point's leaf is at most (distance + excursion)^2 (as in `reaches`).
__global__ void k_kd_cands(const int *__restrict__ cand, int n, const int *__restrict__ treePos,
                           const float4 *__restrict__ pos, const float *__restrict__ nodeBox,
                           const int *__restrict__ leafOf, float r2, int *__restrict__ posOf,
                           float *__restrict__ sure) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n)
        return;
    const int    id = cand[r], ip = treePos[id];
    posOf[r] = ip;
    sure[r]  = sure_reach(r2, excursion(nodeBox + 6 * (size_t)leafOf[ip], pos[id]));
}

// Leaves holding an active position flag themselves and their ancestors (a walk stops at
// an ancestor another walk has flagged).
__global__ void k_kd_nonempty(const int4 *__restrict__ nd, const int *__restrict__ parent,
                              int nnodes, const int *__restrict__ vacc, int *__restrict__ flags) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nnodes)
        return;
    const int4 n = nd[v];
    if (!smk::is_leaf(n))
        return;
    bool any = false;
    for (int i = n.x; i < n.y && !any; i++)
        any = vacc[i] >= 0;
    for (int u = v; any && u >= 0; u = parent[u])
        if (atomicExch(&flags[u], 1) == 1)
            break;
}

// Leaf records, and with excMax (zeroed) the largest distance of a listed point from its
// leaf's build-time box, rounded up (as float bits: they order like the floats).
__global__ void k_kd_tpos(const int *__restrict__ vacc, int m, const float4 *__restrict__ pos,
                          const float *__restrict__ nodeBox, const int *__restrict__ leafOf,
                          float4 *__restrict__ tpos, float *__restrict__ excMax) {
    const int i  = blockIdx.x * blockDim.x + threadIdx.x;
    const int id = i < m ? vacc[i] : -1;
    float     e  = 0.0f;
    if (id >= 0) {
        const float4 p = pos[id];
        tpos[i]        = make_float4(p.x, p.y, p.z, __int_as_float(id));
        if (excMax)
            e = (float)(excursion(nodeBox + 6 * (size_t)leafOf[i], p) * (1.0 + 1e-6));
    } else if (i < m) {
        tpos[i] = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
    }
    if (excMax) {
        const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(e));
        if ((threadIdx.x & 31) == 0 && w)
            atomicMax((unsigned *)excMax, w);
    }
}

} // namespace

// =======================================================================================
void build_kdtree(Ctx &c, const float4 *pos, int npoints, const int *ids, int m, const Box &box,
                  KdTree &T, const std::string &tag) {
    if (m >= (1 << 28))
        throw Error(SM_ERR_CAPACITY, "k-d tree over more than 2^28 points is not supported");
    T.m       = m;
    T.npoints = npoints;
    const int cap = std::max(2 * m, 1);
    T.nd      = c.arena.get<int4>(tag + ".nd", cap);
    T.box     = c.arena.get<float>(tag + ".box", (size_t)6 * cap);
    T.vacc    = c.arena.get<int>(tag + ".vacc", std::max(m, 1));
    T.leafOf  = c.arena.get<int>(tag + ".leaf", std::max(m, 1));
    T.treePos = c.arena.get<int>(tag + ".tpos", std::max(npoints, 1));
    T.rec     = c.arena.get<float4>(tag + ".rec", std::max(m, 1));
    int *parent  = c.arena.get<int>(tag + ".par", cap);
    T.parent     = parent;
    int *arrive  = c.arena.get<int>(tag + ".arr", cap);
    int *ctl     = c.arena.get<int>(tag + ".ctl", kKdCtl);
    int *segOf   = c.arena.get<int>(tag + ".segof", std::max(m, 1));
    int *g1      = c.arena.get<int>(tag + ".g1", (size_t)m + 1);
    int *g2      = c.arena.get<int>(tag + ".g2", (size_t)m + 1);
    int *badR    = c.arena.get<int>(tag + ".badr", std::max(m, 1));
    const int maxSeg = std::max(m / (smk::kLeafMax + 1) + 2, 2);
    const int maxOpen = m / (kSmall + 1) + 1; // open ranges of a level: above kSmall points each
    Seg *segs[2] = {c.arena.get<Seg>(tag + ".segA", maxSeg), c.arena.get<Seg>(tag + ".segB", maxSeg)};
    Seg *small   = c.arena.get<Seg>(tag + ".small", maxSeg);
    SM_CUDA(cudaMemsetAsync(ctl, 0, kKdCtl * sizeof(int), c.stream));
    SM_CUDA(cudaMemsetAsync(T.treePos, 0xff, (size_t)std::max(npoints, 1) * 4, c.stream));
    if (m == 0)
        return;
    k_kd_root<<<1, 1, 0, c.stream>>>(segs[0], small, m, box, T.nd, parent, ctl);
    SM_LAUNCH_CHECK();
    k_kd_init<<<nblocks(m, 256), 256, 0, c.stream>>>(pos, ids, m, T.rec, segOf, segs[0]);
    SM_LAUNCH_CHECK();
    const int       gm    = nblocks(m, 256), go = nblocks(maxOpen, 128);
    const long long n1    = (long long)m + 1;
    const int       parts = (int)((n1 + kScanTile - 1) / kScanTile);
    auto            read  = [&](int first, int n) { // control words to the host
        SM_CUDA(cudaMemcpyAsync(c.hostCounts, ctl + first, n * sizeof(int), cudaMemcpyDeviceToHost,
                                c.stream));
        c.sync_checked();
    };
    // (a level above kMaxDepth has no open range: its parents set the error and the host stops)
    bool open = m > kSmall;
    for (int level = 0; open; level++) {
        Seg *cur = segs[level & 1], *nxt = segs[(level + 1) & 1];
        int *nseg = ctl + kKdOpen + level, *onCut = ctl + kKdOnCut + level;
        launch_chained(c, k_kd_cut, go, 128, 0, cur, nseg);
        for (int pass = 1; pass <= 2; pass++) {
            int    *g = pass == 1 ? g1 : g2;
            KdFlags F{T.rec, segOf, cur, nseg, g1, onCut, pass, m};
            const unsigned epoch = scan_state(c, parts);
            launch_chained(c, k_scan_lookback<KdFlags, kPrefix>, parts, kScanBs, 0, F, g, n1,
                           (const int *)nullptr, c.scan.status, c.scan.ticket, parts, epoch,
                           (int *)nullptr);
            launch_chained(c, k_kd_rank, gm, 256, 0, F, g, badR);
            launch_chained(c, k_kd_swap, gm, 256, 0, F, T.rec, g, badR);
        }
        launch_chained(c, k_kd_children, go, 128, 0, cur, nseg, onCut, g1, g2, T.nd, parent, ctl, nxt,
                       nseg + 1, small);
        launch_chained(c, k_kd_advance, gm, 256, 0, T.rec, segOf, m, cur, nseg, nxt);
        if ((level + 1) % kKdLevels == 0) {
            read(0, kKdOpen + level + 2);
            open = c.hostCounts[kKdOpen + level + 1] > 0;
            if (c.hostCounts[kKdErr])
                throw Error(SM_ERR_CAPACITY, "k-d tree deeper than " + std::to_string(smk::kMaxDepth));
        }
    }
    read(0, kKdOpen);
    const int nsmall = c.hostCounts[kKdSmallN];
    if (nsmall > 0) {
        k_kd_small<<<nsmall, kSmall, 0, c.stream>>>(small, T.rec, T.nd, parent, ctl + kKdNodes,
                                                    ctl + kKdErr);
        SM_LAUNCH_CHECK();
    }
    SM_CUDA(cudaMemsetAsync(arrive, 0, (size_t)cap * 4, c.stream));
    k_kd_finish<<<nblocks(cap, 256), 256, 0, c.stream>>>(T.nd, parent, ctl + kKdNodes, T.rec, T.box,
                                                         arrive, T.vacc, T.leafOf, T.treePos);
    SM_LAUNCH_CHECK();
    read(0, kKdOpen);
    T.nnodes = c.hostCounts[kKdNodes];
    if (c.hostCounts[kKdErr] == 1)
        throw Error(SM_ERR_CAPACITY, "k-d tree deeper than " + std::to_string(smk::kMaxDepth));
    if (c.hostCounts[kKdErr] == 2)
        throw Error(SM_ERR_CAPACITY, "k-d tree build: too many open ranges in a small range");
}

int kd_sample(Ctx &c, const KdTree &T, const int *vaccActive, const float4 *pos, float step,
              const Box &box, int *outIds, int *ioi, const std::string &tag, const int **before) {
    const int m = T.m;
    if (m <= 0)
        return 0;
    const int *vaccA = vaccActive ? vaccActive : T.vacc;
    float      ext[3] = {box.ext(0), box.ext(1), box.ext(2)};
    unsigned   ring   = 1024;
    while (ring < 2u * (unsigned)m)
        ring <<= 1;
    GridParamsK gp;
    // a dense table where cells just above the step fit it (5 % faster than hashed ones on 0.9 M
    // points: 1.59 against 1.68 ms), else hashed ones (0.9 M points in an extent of twice and four
    // times what fits: 1.76 and 1.58 ms; cells of twice and four times the side 2.15 and 4.87)
    gp.g = smg::sample_cell(step, ext, kSpCells);
    for (int a = 0; a < 3; a++) {
        gp.org[a] = box.mn[a];
        gp.dim[a] = smg::dim_of(ext[a], gp.g);
    }
    const float     want   = step * (1.0f + 1.0f / 1024.0f);
    const bool      hashed = gp.g > kSpCoarse * want;
    const long long nc     = hashed ? (long long)ring : (long long)gp.dim[0] * gp.dim[1] * gp.dim[2];
    const uint32_t  noCell = (uint32_t)nc;
    int             bits   = 1;
    while ((nc >> bits) != 0)
        bits++;
    uint32_t *key   = c.arena.get<uint32_t>(tag + ".key", m);
    uint32_t *val   = c.arena.get<uint32_t>(tag + ".val", m);
    int      *head  = c.arena.get<int>(tag + ".head", (size_t)m + 1);
    int      *rank  = c.arena.get<int>(tag + ".rank", (size_t)m + 1);
    int      *cRank = c.arena.get<int>(tag + ".crank", nc);
    int      *cList = c.arena.get<int>(tag + ".clist", m); // at most a cell per point
    int      *cEnd  = c.arena.get<int>(tag + ".cend", m);
    float4   *ent   = c.arena.get<float4>(tag + ".ent", m);
    float    *sure  = c.arena.get<float>(tag + ".sure", m);
    int      *flag  = c.arena.get<int>(tag + ".flag", (size_t)m + 1);
    int      *ctl   = c.arena.get<int>(tag + ".ctl", 4 * kSpCtl); // head, tail, open cells, error
    SampleArgs a{};
    a.t = T.view(vaccA, pos);
    for (int d = 0; d < 3; d++)
        a.dim[d] = gp.dim[d];
    a.ent      = ent;
    a.sure     = sure;
    a.cellRank = cRank;
    a.cellList = cList;
    a.cellEnd  = cEnd;
    a.cur      = c.arena.get<unsigned long long>(tag + ".cur", m);
    a.dec      = c.arena.get<int>(tag + ".dec", m);
    a.filed    = c.arena.get<int>(tag + ".filed", m);
    a.nextCell = c.arena.get<int>(tag + ".next", m);
    a.ring     = c.arena.get<int>(tag + ".ring", ring);
    a.ringMask = ring - 1;
    a.head     = ctl;
    a.tail     = ctl + kSpCtl;
    a.open     = ctl + 2 * kSpCtl;
    a.r2       = step * step;
    a.keptFlag = flag;
    a.err      = ctl + 3 * kSpCtl;
    if (hashed) {
        auto *keys = c.arena.get<unsigned long long>(tag + ".keys", nc);
        a.keys     = keys;
        a.slotMask = (uint32_t)(nc - 1);
        SM_CUDA(cudaMemsetAsync(keys, 0xff, (size_t)nc * 8, c.stream));
        k_sp_keys_hashed<<<nblocks(m, 256), 256, 0, c.stream>>>(vaccA, pos, m, 1.0 / (double)want, keys,
                                                                a.slotMask, noCell, key, val);
    } else {
        k_sp_keys<<<nblocks(m, 256), 256, 0, c.stream>>>(vaccA, pos, m, gp, noCell, key, val);
    }
    SM_LAUNCH_CHECK();
    radix_sort_pairs(c, key, val, m, bits, tag);
    k_sp_heads<<<nblocks((long long)m + 1, 256), 256, 0, c.stream>>>(key, m, noCell, head);
    SM_LAUNCH_CHECK();
    scan_excl(c, head, rank, (long long)m + 1, tag + ".hs", false);
    SM_CUDA(cudaMemsetAsync(cRank, 0xff, (size_t)nc * 4, c.stream));
    SM_CUDA(cudaMemsetAsync(flag, 0, ((size_t)m + 1) * 4, c.stream));
    SM_CUDA(cudaMemsetAsync(ctl, 0, 4 * kSpCtl * sizeof(int), c.stream));
    SM_CUDA(cudaMemsetAsync(a.ring, 0xff, (size_t)ring * 4, c.stream));
    k_sp_cells<<<nblocks(m, 256), 256, 0, c.stream>>>(key, val, m, noCell, head, rank, T.box,
                                                     T.leafOf, cRank, cList, cEnd, ent, sure, a);
    SM_LAUNCH_CHECK();
    int nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    const int gFirst = std::min(nblocks(m, kSpBs / 32), nsm * 8);
    const int gRun   = std::min(nblocks(m, kSpBs / 32), nsm * kSpCtas);
    if (hashed)
        k_sp_first<true><<<gFirst, kSpBs, 0, c.stream>>>(a);
    else
        k_sp_first<false><<<gFirst, kSpBs, 0, c.stream>>>(a);
    SM_LAUNCH_CHECK();
    if (hashed)
        k_sp_run<true><<<gRun, kSpBs, 0, c.stream>>>(a);
    else
        k_sp_run<false><<<gRun, kSpBs, 0, c.stream>>>(a);
    SM_LAUNCH_CHECK();
    int *pre = c.arena.get<int>(tag + ".pre", (size_t)m + 1);
    scan_excl(c, flag, pre, (long long)m + 1, tag + ".os", false);
    if (before)
        *before = pre;
    k_sp_out<<<nblocks(m, 256), 256, 0, c.stream>>>(flag, pre, m, vaccA, outIds, ioi);
    SM_LAUNCH_CHECK();
    SM_CUDA(cudaMemcpyAsync(c.hostCounts, pre + m, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    SM_CUDA(cudaMemcpyAsync(c.hostCounts + 1, a.err, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    c.sync_checked();
    if (c.hostCounts[1])
        throw Error(SM_ERR_RUNTIME, "tree-order sampler: a bounded wait expired");
    return c.hostCounts[0];
}

void kd_knn(Ctx &c, const KdTree &T, const int *vaccActive, const float4 *pos,
            const float4 *qpos, const int *nq, int nqMax, int k, int *nbr, float *dist) {
    if (nqMax <= 0 || T.m <= 0)
        return;
    if (k < 1 || k > kMaxKnn)
        throw Error(SM_ERR_RANGE, "knnNormal larger than " + std::to_string(kMaxKnn) + " is not supported");
    float4 *tpos = c.arena.get<float4>("kd.knn.tpos", T.m);
    kd_tree_positions(c, T, vaccActive, pos, tpos);
    k_kd_knn<<<nblocks(nqMax, 128), 128, 0, c.stream>>>(T.view(vaccActive, pos, nullptr, tpos), qpos,
                                                        nq, k, nbr, dist);
    SM_LAUNCH_CHECK();
}

void kd_knn_points(Ctx &c, const KdTree &T, const HGrid &g, const float4 *pos,
                   const smd::NormalList &L, int part, int nqMax, int k, bool grow,
                   const float4 *nrm) {
    if (nqMax <= 0 || T.m <= 0)
        return;
    if (g.coarse) {
        k_kd_knn_list<<<nblocks(nqMax, 128), 128, 0, c.stream>>>(T.view(nullptr, pos), L, part, k, grow,
                                                                 nrm);
        SM_LAUNCH_CHECK();
        return;
    }
    k_kd_knn_grid<<<nblocks((long long)nqMax * 32, kKnnBs), kKnnBs, 0, c.stream>>>(
        T.view(nullptr, pos), T.m, g.view(), T.treePos, L, part, k, grow, nrm);
    SM_LAUNCH_CHECK();
}

void kd_vote_tree(Ctx &c, const KdTree &T, const int *vaccActive, const float4 *pos,
                  const int *cand, int ncand, const int *before, float r2, VoteTree &V,
                  const std::string &tag) {
    int   *posOf = c.arena.get<int>(tag + ".pos", std::max(ncand, 1));
    float *sure  = c.arena.get<float>(tag + ".sure", std::max(ncand, 1));
    V.view       = T.view(vaccActive, pos);
    V.m          = T.m;
    V.treePos    = T.treePos;
    V.posOf      = posOf;
    V.before     = before;
    V.sure       = sure;
    if (ncand <= 0)
        return;
    k_kd_cands<<<nblocks(ncand, 256), 256, 0, c.stream>>>(cand, ncand, T.treePos, pos, T.box,
                                                          T.leafOf, r2, posOf, sure);
    SM_LAUNCH_CHECK();
}

void kd_mark_nonempty(Ctx &c, const KdTree &T, const int *vaccActive, int *flags) {
    if (T.nnodes <= 0)
        return;
    SM_CUDA(cudaMemsetAsync(flags, 0, (size_t)T.nnodes * 4, c.stream));
    k_kd_nonempty<<<nblocks(T.nnodes, 256), 256, 0, c.stream>>>(T.nd, T.parent, T.nnodes,
                                                                vaccActive ? vaccActive : T.vacc,
                                                                flags);
    SM_LAUNCH_CHECK();
}

void kd_tree_positions(Ctx &c, const KdTree &T, const int *vaccActive, const float4 *pos,
                       float4 *tpos, float *excMax) {
    if (excMax)
        SM_CUDA(cudaMemsetAsync(excMax, 0, sizeof(float), c.stream));
    if (T.m <= 0)
        return;
    k_kd_tpos<<<nblocks(T.m, 256), 256, 0, c.stream>>>(vaccActive ? vaccActive : T.vacc, T.m, pos,
                                                        T.box, T.leafOf, tpos, excMax);
    SM_LAUNCH_CHECK();
}

} // namespace sm
