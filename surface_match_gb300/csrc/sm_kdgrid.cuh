// sm_kdgrid.cuh - the reference-order nearest searches answered on a uniform grid.
//
// A k-d tree search by one thread is a chain of some hundred dependent loads; a warp finds
// the nearest points on a grid in a few rounds of independent ones. The reference's search
// differs from the exact nearest points only through its order (which of equally distant
// points it meets first) and its pruning (normal estimation moves points out of their
// leaves' boxes, and the search bounds the boxes). Both are decided here by the search
// itself, restricted to the points that can matter:
//
//   Let B be a squared distance and C all points with squared distance <= B. Run the
//   reference's search on the tree that holds only C (subtrees without a point of C are
//   skipped: sm_kdtree.cuh). Leaving points farther than B out changes its worst distance
//   only where that is above B. So every decision "lower bound md <= worst" comes out as in
//   the full search unless it passes with md > B; if none does, the points found are exactly
//   those of the full search that lie within B. Otherwise B grows to the largest such md and
//   the search runs again.
//
// With B the k-th smallest distance, C is the k nearest points and the restricted search
// visits little more than their root paths. Measured with a thread per query on the tree against
// a warp per query here: correspondences of the large scene's dense refinement 750 -> 220 us a
// launch, of the sparse one 340 -> 48 us; its 140,000 k-nearest searches 1970 -> 430 us;
// the whole large scene in reference order 29.5 -> 22.1 ms, the small one 12.3 -> 9.7 ms.
// Lane j of the warp holds point j of C; the
// pending far children's frames live one per lane (each splits C, so there are at most 31).
#pragma once

#include "sm_device.cuh"
#include "sm_kdtree.cuh"

namespace smk {

constexpr int kMaxRaise = 4; // times B may grow before the full search by one lane decides

// The restricted search by a warp. Lane j < count holds a point of C: tree position pos,
// squared distance d; the lanes ascend in d. k results are kept (worst distance: the k-th
// smallest met so far). Returns the mask of lanes whose point was met; *seq = the lane's place
// in the order of meeting; *over = the largest md > B that passed (0: none).
__device__ __forceinline__ unsigned warp_kd_restricted(const int4 *__restrict__ nd, int m,
                                                       const KdView &t, const float q[3], int count,
                                                       int pos, float d, int k, float B, int *seq,
                                                       float *over) {
    const int  lane = threadIdx.x & 31;
    const bool have = lane < count;
    unsigned   met  = 0u;
    int        sp = 0, leaves = 0;
    float      worst = 3.402823466e38f, big = 0.0f;
    float      ds[3];
    float      mind = init_dists(t, q, ds);
    int        v = 0, l = 0, r = m;
    // this lane's frame of the stack
    int   fOther = 0, fIdx = 0, fL = 0, fR = 0;
    float fCut = 0.f, fMind = 0.f, f0 = 0.f, f1 = 0.f, f2 = 0.f;
    *seq        = 0;
    bool resume = false;
    for (;;) {
        if (resume) {
            // the deepest pending far child that passes its bound
            bool found = false;
            while (sp > 0 && !found) {
                sp--;
                const int   idx = __shfl_sync(0xffffffffu, fIdx, sp);
                const float cut = __shfl_sync(0xffffffffu, fCut, sp);
                const float fm  = __shfl_sync(0xffffffffu, fMind, sp);
                float       e[3];
                e[0]            = __shfl_sync(0xffffffffu, f0, sp);
                e[1]            = __shfl_sync(0xffffffffu, f1, sp);
                e[2]            = __shfl_sync(0xffffffffu, f2, sp);
                const float dst = idx == 0 ? e[0] : idx == 1 ? e[1] : e[2];
                const float md  = fm + cut - dst;
                if (md * 1.0f <= worst) {
                    if (md > B)
                        big = fmaxf(big, md);
                    ds[0] = idx == 0 ? cut : e[0];
                    ds[1] = idx == 1 ? cut : e[1];
                    ds[2] = idx == 2 ? cut : e[2];
                    mind  = md;
                    v     = __shfl_sync(0xffffffffu, fOther, sp);
                    l     = __shfl_sync(0xffffffffu, fL, sp);
                    r     = __shfl_sync(0xffffffffu, fR, sp);
                    found = true;
                }
            }
            if (!found)
                break;
            resume = false;
        }
        const int4 n = nd[v];
        if (is_leaf(n)) {
            const bool     in = have && pos >= n.x && pos < n.y && d < worst;
            const unsigned mk = __ballot_sync(0xffffffffu, in);
            if (in)
                *seq = leaves * 16 + (pos - n.x); // (a leaf has at most 10 entries)
            leaves++;
            met |= mk;
            if (__popc(met) >= k) {
                unsigned w = met; // the k-th smallest met: the lanes ascend in d
                for (int j = 1; j < k; j++)
                    w &= w - 1u;
                worst = __shfl_sync(0xffffffffu, d, __ffs(w) - 1);
            }
            resume = true;
            continue;
        }
        const int   idx = divfeat_of(n);
        const float val = idx == 0 ? q[0] : idx == 1 ? q[1] : q[2];
        const float dlow = __int_as_float(n.x), dhigh = __int_as_float(n.y);
        const int   c1   = child1_of(n);
        const bool  low  = ((val - dlow) + (val - dhigh)) < 0.0f; // child 1 is the nearer
        const float cut  = low ? (val - dhigh) * (val - dhigh) : (val - dlow) * (val - dlow);
        const bool  in1  = __any_sync(0xffffffffu, have && pos >= l && pos < n.w);
        const bool  in2  = __any_sync(0xffffffffu, have && pos >= n.w && pos < r);
        const bool  nearIn = low ? in1 : in2, farIn = low ? in2 : in1;
        const int   nearV = low ? c1 : c1 + 1, farV = low ? c1 + 1 : c1;
        const int   farL = low ? n.w : l, farR = low ? r : n.w;
        const int   nearL = low ? l : n.w, nearR = low ? n.w : r;
        if (nearIn) {
            if (farIn) {
                if (lane == sp) {
                    fOther = farV;
                    fIdx   = idx;
                    fL     = farL;
                    fR     = farR;
                    fCut   = cut;
                    fMind  = mind;
                    f0     = ds[0];
                    f1     = ds[1];
                    f2     = ds[2];
                }
                sp++;
            }
            v = nearV;
            l = nearL;
            r = nearR;
            continue;
        }
        // only the far child holds a point of C: checked now (the near one's search returns
        // at once)
        const float dst = idx == 0 ? ds[0] : idx == 1 ? ds[1] : ds[2];
        const float md  = mind + cut - dst;
        if (farIn && md * 1.0f <= worst) {
            if (md > B)
                big = fmaxf(big, md);
            if (idx == 0)
                ds[0] = cut;
            else if (idx == 1)
                ds[1] = cut;
            else
                ds[2] = cut;
            mind = md;
            v    = farV;
            l    = farL;
            r    = farR;
            continue;
        }
        resume = true;
    }
    *over = big;
    return met;
}

// Rings that a walk here goes out to before it leaves the query to the tree's own search: the
// rings' cubes grow with the fourth power of the distance, so a lone point some hundred cells from
// its neighbours would keep its warp for seconds.
constexpr int kMaxShell = smd::kTreeShell;
constexpr int kFar      = -2; // a nearest search that gave up there

// All points of grid g within squared distance B of q (<=), ascending by (distance, index) over
// the lanes: lane j gets the j-th key. Returns their number; above 32, or where B reaches beyond
// kMaxShell rings, 33 and no points.
__device__ __forceinline__ int warp_collect(const smd::HGridView &g, float qx, float qy, float qz,
                                            float B, unsigned long long *key) {
    unsigned long long best = ~0ull;
    int                n    = 0;
    auto               visit = [&](const float4 &p, bool valid) {
        unsigned long long kk = ~0ull;
        if (valid) {
            const float dd = smm::dist2(qx, qy, qz, p.x, p.y, p.z);
            if (dd <= B)
                kk = ((unsigned long long)__float_as_uint(dd) << 32) | (unsigned)__float_as_int(p.w);
        }
        const int c = __popc(__ballot_sync(0xffffffffu, kk != ~0ull));
        if (c) {
            n += c;
            best = smd::warp_merge_low(best, smd::warp_bitonic_sort(kk));
        }
        return n > 32;
    };
    int c[3];
    smd::grid_cc(g, qx, qy, qz, c);
    const int ms = max(smd::grid_max_shell(g, c), 1);
    bool      over = smd::warp_block27(g, qx, qy, qz, c, B, visit);
    for (int done = 1; !over;) {
        const float rb = smg::ring_bound(done, g.g, g.slack);
        if (rb * rb > B || done >= ms)
            break;
        const int hi = smd::band_end(done, ms, B, g);
        over = done >= kMaxShell ||
               smd::warp_band(g, qx, qy, qz, c, done + 1, hi, [&]() { return B; }, visit);
        done = hi;
    }
    *key = best;
    return over ? 33 : n;
}

// Nearest point of g by squared distance as smd::warp_nn_walk (bounded by limit2), and whether
// another point lies at the same distance. kFar: not found within kMaxShell rings.
__device__ __forceinline__ int warp_nn_tie(const smd::HGridView &g, float qx, float qy, float qz,
                                           float limit2, float &outd, bool &tie) {
    unsigned long long gb = ~0ull, mine = ~0ull; // warp's best so far; lane's since then
    bool               dup = false;
    tie                    = false;
    auto visit = [&](const float4 &p, bool valid) {
        if (valid) {
            const float dd = smm::dist2(qx, qy, qz, p.x, p.y, p.z);
            const unsigned long long key =
                ((unsigned long long)__float_as_uint(dd) << 32) | (unsigned)__float_as_int(p.w);
            if ((unsigned)(key >> 32) == (unsigned)(mine >> 32))
                dup = true;
            else if (key < mine)
                dup = false;
            mine = key < mine ? key : mine;
        }
        return false;
    };
    auto fold = [&]() {
        const unsigned long long m  = smd::warp_min_u64(mine);
        const unsigned           hm = (unsigned)(m >> 32), hg = (unsigned)(gb >> 32);
        const bool same = m != ~0ull && (unsigned)(mine >> 32) == hm;
        const bool t    = __any_sync(0xffffffffu, same && (mine != m || dup));
        if (m != ~0ull) {
            if (hm < hg)
                tie = t;
            else if (hm == hg)
                tie = true;
            gb = m < gb ? m : gb;
        }
        mine = ~0ull;
        dup  = false;
        return gb == ~0ull ? __int_as_float(0x7f800000) : __uint_as_float((unsigned)(gb >> 32));
    };
    int c[3];
    smd::grid_cc(g, qx, qy, qz, c);
    const int ms = max(smd::grid_max_shell(g, c), 1);
    smd::warp_block27(g, qx, qy, qz, c, limit2, visit);
    for (int done = 1;;) {
        const float d  = fold();
        const float rb = smg::ring_bound(done, g.g, g.slack);
        if (d < rb * rb || rb * rb > limit2 || done >= ms)
            break;
        if (done >= kMaxShell)
            return kFar;
        const int hi = smd::band_end(done, ms, fminf(d, limit2), g);
        smd::warp_band(g, qx, qy, qz, c, done + 1, hi, [&]() { return fminf(fold(), limit2); }, visit);
        done = hi;
    }
    fold();
    if (gb == ~0ull) {
        outd = 3.402823466e+38f;
        return -1;
    }
    outd = __uint_as_float((unsigned)(gb >> 32));
    return (int)(unsigned)(gb & 0xffffffffu);
}

// Whether the nearest point's squared distance d is one that the reference's search returns and
// its caller asks for (the search starts from the largest float: d may have overflowed).
__device__ __forceinline__ bool in_limit(float d, float limit2) {
    return d <= limit2 && d < 3.402823466e38f;
}

// The search itself, by one lane: the point's name (-1: none, or one farther than limit2) and its
// squared distance.
__device__ __forceinline__ int tree_nearest(const KdView &t, const int *__restrict__ nameOf, float exc,
                                            float qx, float qy, float qz, float limit2, float *d) {
    const float q[3] = {qx, qy, qz};
    NnSet       rs;
    rs.init(nn_bound(nn_bound(limit2, exc), exc));
    kd_search(t, q, rs);
    *d = rs.dist;
    return !rs.count ? -1 : nameOf ? nameOf[rs.idx] : rs.idx;
}

// What the reference's one-nearest search of tree `t` (m positions, reduced to the points of
// grid g; t.tpos their leaf records) returns from q, provided its squared distance is at most
// limit2: the point's name in g (pts.w) and its squared distance *d. Else -1, or a point farther
// than limit2. posOf[name] = the point's tree position, nameOf[id] = the name of point id
// (nullptr: the name is the id); exc = the points' largest excursion (nn_bound). A whole warp
// calls it for one query.
__device__ __forceinline__ int warp_kd_nearest(const KdView &t, int m, const smd::HGridView &g,
                                               const int *__restrict__ posOf,
                                               const int *__restrict__ nameOf, float exc, float qx,
                                               float qy, float qz, float limit2, float *d) {
    const int   lane = threadIdx.x & 31;
    const float q[3] = {qx, qy, qz};
    if (!isfinite(qx) || !isfinite(qy) || !isfinite(qz))
        return -1; // no distance from it is below the search's start
    bool tie;
    const int   j = warp_nn_tie(g, qx, qy, qz, limit2, *d, tie);
    if (j != kFar && (j < 0 || !in_limit(*d, limit2)))
        return -1; // the reference's result is no nearer
    float B     = *d;
    float dl    = *d;
    int   name  = j;
    int   count = 1;
    for (int it = 0; j != kFar && it < kMaxRaise; it++) {
        if (it > 0 || tie) {
            unsigned long long key;
            count = warp_collect(g, qx, qy, qz, B, &key);
            if (count > 32)
                break;
            name = (int)(unsigned)key;
            dl   = __uint_as_float((unsigned)(key >> 32));
        }
        const int      pos = lane < count ? posOf[name] : -1;
        int            seq;
        float          over;
        const unsigned met =
            warp_kd_restricted(t.nd, m, t, q, count, pos, dl, 1, B, &seq, &over);
        if (over > B) {
            B = over;
            continue;
        }
        // the nearest met, of equals the first met
        const unsigned long long kk =
            (met >> lane) & 1u
                ? ((unsigned long long)__float_as_uint(dl) << 32) | (unsigned)seq
                : ~0ull;
        const unsigned long long w = smd::warp_min_u64(kk);
        if (w == ~0ull)
            return -1; // (C was never empty: unreachable)
        const int src = __ffs(__ballot_sync(0xffffffffu, kk == w)) - 1;
        *d            = __shfl_sync(0xffffffffu, dl, src);
        return __shfl_sync(0xffffffffu, name, src);
    }
    // the search itself, by one lane
    int   id = -1;
    float dd = 0.0f;
    if (lane == 0)
        id = tree_nearest(t, nameOf, exc, qx, qy, qz, limit2, &dd);
    *d = __shfl_sync(0xffffffffu, dd, 0);
    return __shfl_sync(0xffffffffu, id, 0);
}

// The same for up to 32 queries of a warp, a lane's own each (`need`: it has one): the nearest
// points on the grid by the whole warp, query after query, then the root paths of those that
// are the only ones at their distance by their lanes at once (a point that is reached even with
// its own distance as the bound is the one that is returned), and the search above for the rest.
// (A warp's restricted search per query took two thirds of the time of the reference order's
// correspondences.)
__device__ __forceinline__ int lanes_kd_nearest(const KdView &t, int m, const smd::HGridView &g,
                                                const int *__restrict__ posOf,
                                                const int *__restrict__ nameOf, float exc, float qx,
                                                float qy, float qz, float limit2, bool need, float *d) {
    const int lane = threadIdx.x & 31;
    int       j    = -1;
    bool      tied = false;
    float     dd;
    *d = 3.402823466e+38f;
    // (no distance from a point that is not finite is below the search's start)
    need = need && isfinite(qx) && isfinite(qy) && isfinite(qz);
    if (g.coarse) { // (uniform) the search itself, a lane for each query
        if (need)
            j = tree_nearest(t, nameOf, exc, qx, qy, qz, limit2, d);
        __syncwarp();
        return j;
    }
    for (unsigned w = __ballot_sync(0xffffffffu, need); w; w &= w - 1u) {
        const int src = __ffs(w) - 1;
        bool      tie;
        const int r = warp_nn_tie(g, __shfl_sync(0xffffffffu, qx, src), __shfl_sync(0xffffffffu, qy, src),
                                  __shfl_sync(0xffffffffu, qz, src),
                                  __shfl_sync(0xffffffffu, limit2, src), dd, tie);
        if (lane == src) {
            j    = r;
            *d   = dd;
            tied = tie;
        }
    }
    bool open = false;
    if (j == kFar) {
        open = true;
    } else if (j >= 0 && !in_limit(*d, limit2)) {
        j  = -1; // the reference's result is no nearer
        *d = 3.402823466e38f;
    } else if (j >= 0) {
        uint64_t    key;
        const float q[3] = {qx, qy, qz};
        open             = tied || !kd_reaches(t, q, posOf[j], *d, &key);
    }
    for (unsigned w = __ballot_sync(0xffffffffu, open); w; w &= w - 1u) {
        const int src = __ffs(w) - 1;
        const int r   = warp_kd_nearest(t, m, g, posOf, nameOf, exc, __shfl_sync(0xffffffffu, qx, src),
                                        __shfl_sync(0xffffffffu, qy, src), __shfl_sync(0xffffffffu, qz, src),
                                        __shfl_sync(0xffffffffu, limit2, src), &dd);
        if (lane == src) {
            j  = r;
            *d = dd;
        }
    }
    return j;
}

// The k nearest (k <= 32) that the reference's search of tree `t` (m positions; the points of
// grid g) returns from q, in its order: lane j < the returned count gets the j-th point's id.
// -1: not decided here (the caller runs the search itself).
__device__ __forceinline__ int warp_kd_knearest(const KdView &t, int m, const smd::HGridView &g,
                                                const int *__restrict__ treePos, float qx, float qy,
                                                float qz, int k, int *id) {
    const int   lane = threadIdx.x & 31;
    const float q[3] = {qx, qy, qz};
    float       d;
    const int   n = smd::warp_knn_sorted<true>(g, qx, qy, qz, k, id, &d);
    if (n < 0)
        return -1; // far from its neighbours
    // fewer than k points in all: the search's worst distance stays at the start
    float B = n < k ? 3.402823466e38f : __shfl_sync(0xffffffffu, d, k - 1);
    if (__any_sync(0xffffffffu, lane < n && !(d < 3.402823466e38f)))
        return -1; // (distances that overflow: a search from the largest float leaves them out)
    int   pos = lane < n ? treePos[*id] : -1;
    {
        // every one of them reached even with the final worst distance, and no two at one
        // distance (nor a further point at the last one's): the order is that of the distances
        uint64_t    key;
        const bool  in    = lane >= n || kd_sure(t, q, pos, B) || kd_reaches(t, q, pos, B, &key);
        const float dn    = __shfl_down_sync(0xffffffffu, d, 1);
        const int   idn   = __shfl_down_sync(0xffffffffu, *id, 1);
        const bool  equal = lane < n && lane < 31 && idn != -1 && dn == d;
        if (__all_sync(0xffffffffu, in && !equal) && k < 32)
            return n;
    }
    for (int it = 0; it < kMaxRaise; it++) {
        unsigned long long key;
        const int          count = warp_collect(g, qx, qy, qz, B, &key);
        if (count > 32)
            return -1;
        const int   name = (int)(unsigned)key;
        const float dl   = __uint_as_float((unsigned)(key >> 32));
        int         seq;
        float       over;
        pos = lane < count ? treePos[name] : -1;
        const unsigned met = warp_kd_restricted(t.nd, m, t, q, count, pos, dl, k, B, &seq, &over);
        if (over > B) {
            B = over;
            continue;
        }
        unsigned long long kk = ~0ull;
        if ((met >> lane) & 1u)
            kk = ((unsigned long long)__float_as_uint(dl) << 32) | (unsigned)((seq << 5) | lane);
        kk            = smd::warp_bitonic_sort(kk);
        const int src = (int)(kk & 31u);
        *id           = __shfl_sync(0xffffffffu, name, src);
        return min(k, __popc(met));
    }
    return -1;
}

} // namespace smk
