// sm_vote.cuh - device pieces of the voting stage shared by the multi-kernel pipeline
// (vote_pipe.cu) and the single-kernel variant (vote.cu): model table probe, the
// shared-memory vote loop, peak extraction and the per-keypoint result (ppf.cpp:247-409).
#pragma once

#include <algorithm>
#include <climits>
#include <type_traits>

#include "sm_device.cuh"
#include "sm_icp.h"

namespace sm {
namespace vt {

using namespace smd;

constexpr int kVoteU     = 8;           // bucket entries each lane has in flight
constexpr int kItem      = 32 * kVoteU; // bucket entries per warp work item
constexpr int kNarrowMax = 65535;       // 16-bit counters are exact up to this many votes

// Everything a voting kernel reads or writes.
struct VoteArgs {
    // model
    const float4 *sp, *sn;
    int           ns;
    const uint4  *htab;
    uint32_t      hmask;
    const uint2  *entries;
    int           A;
    float         angleStep, distStep, smax, sqDiam, voteThreshold;
    // scene
    const float4 *pos, *nrm;
    const int    *kp;
    int           K;
    const int    *nbrOff, *nbrIds; // CSR neighbour lists, or
    const int    *cand;            // radius mode: candidate point ids (ascending)
    int           ncand;
    // accumulator sizing
    int refChunk;     // reference points per accumulator pass with 16-bit counters
    int refChunkWide; // the same with 32-bit counters
    // outputs
    long long *stats; // K x 8
    float     *cands, *poses;
    int       *poseOk;
    int       *acc;
    int        dumpK;
    int        forceWide;   // 32-bit counters for every keypoint (a test switch)
    int        fingerprint; // fold the accumulators into stats column 4 (a test switch)
};

struct Cand {
    float v;
    int   r, j;
};

__device__ __forceinline__ bool before(const Cand &a, const Cand &b) {
    return a.v > b.v || (a.v == b.v && a.r < b.r);
}

__device__ __forceinline__ void top3_insert(Cand t[3], const Cand &c) {
    if (!before(c, t[2]))
        return;
    if (before(c, t[1])) {
        t[2] = t[1];
        if (before(c, t[0])) {
            t[1] = t[0];
            t[0] = c;
        } else {
            t[1] = c;
        }
    } else {
        t[2] = c;
    }
}

// Open-addressed model table of uint4 {key, first entry, entry count, 0}; count 0 = empty.
__device__ __forceinline__ uint32_t probe(const uint4 *__restrict__ tab, uint32_t mask, uint32_t key,
                                          uint32_t &off, uint32_t &mult) {
    uint32_t i = key & mask;
    for (uint32_t n = 0; n <= mask; n++) {
        const uint4 s = tab[i];
        if (s.z == 0)
            return 0;
        if (s.x == key) {
            off  = s.y;
            mult = s.w;
            return s.z;
        }
        i = (i + 1) & mask;
    }
    return 0;
}

// One vote in cell c of the accumulator at shared address acc. One increment per vote: a warp's
// votes rarely share a cell (a bucket's entries are different pairs), so aggregating them first
// measured 2.8x slower on the large scene.
template <bool NARROW> __device__ __forceinline__ void cast_vote(uint32_t acc, uint32_t c) {
    const uint32_t at = NARROW ? acc + ((c * 2u) & ~3u) : acc + c * 4u;
    const uint32_t by = NARROW ? (c & 1u) * 65535u + 1u : 1u;
    asm volatile("red.relaxed.cta.shared.add.u32 [%0], %1;" : : "r"(at), "r"(by) : "memory");
}

// Votes of the hits hOff/hCnt/hAs/hAsT[0..nHits) into the shared accumulator of reference
// points [r0, r1) (ALL: of every one). A hit's bucket is cut into items of kItem consecutive
// entries (cPre: prefix of items per hit, T in all) and each warp takes a contiguous range of
// items. Within an item the hit's values are warp-uniform registers, lane l owns entries l, l+32,
// ..., so the loads coalesce, and issues up to kVoteU of them before the first use. NARROW: two
// 16-bit counters per 32-bit word. Bound by a vote's instructions and the bank conflicts of its
// increments (5.4 wavefronts a round of 32 random cells): a round inside the bucket's 8-lane
// blocks has no tests of its own, whole batches of rounds no predicated loads, and the bin is
// smm::vote_bin's of such an entry (whose floor the conversion to an unsigned number is). With
// tests and predicates on every entry (39 instructions a round) 2.9e9 votes of 3,349 keypoints
// took 4.36 ms, now 2.65; the large scene's 35e6 0.125 ms, now 0.098. Loads of the next item
// taken over vote by vote (a fuller pipeline) measured slower, 3.7 against 3.5 ms at that point.
template <bool ALL, bool NARROW>
__device__ __forceinline__ void cast_items(const VoteArgs &a, uint32_t acc, const int *hOff,
                                           const int *hCnt, const float *hAs, const float *hAsT,
                                           const int *cPre, int h, int i0, int i1, int r0, int r1) {
    const int      lane = threadIdx.x & 31;
    const uint32_t A = (uint32_t)a.A, last = A - 1u;
    const float    smax = a.smax;
    for (int item = i0; item < i1; item++) {
        while (cPre[h + 1] <= item)
            h++;
        const int    B   = hCnt[h], e0 = (item - cPre[h]) * kItem;
        const int    n   = min(B - e0, kItem);                // entries of the item
        const int    vec = B - B % smm::kLanes - e0;          // and those inside the blocks
        const float  as  = hAs[h], vs = as - smm::kPiF;
        const uint2 *src = a.entries + hOff[h] + e0 + lane;
        auto         fast = [&](const uint2 &ent) {
            float v = __uint_as_float(ent.y) - vs;
            if (v > smm::k2PiF)
                v = v - smm::k2PiF;
            if (v < 0.0f)
                v = v + smm::k2PiF;
            // (at most A - 1: the bound keeps the index in range whatever the entry)
            const uint32_t bin = min(__float2uint_rz(smax * v), last);
            if (ALL || ((int)ent.x >= r0 && (int)ent.x < r1))
                cast_vote<NARROW>(acc, (ALL ? ent.x : ent.x - (uint32_t)r0) * A + bin);
        };
        auto batch = [&](auto rounds, int u0) {
            uint2 ent[rounds.value];
#pragma unroll
            for (int u = 0; u < rounds.value; u++)
                ent[u] = src[(u0 + u) * 32];
#pragma unroll
            for (int u = 0; u < rounds.value; u++)
                fast(ent[u]);
        };
        const int full = min(n, vec) >> 5; // rounds inside the blocks
        if (full == kVoteU) {
            batch(std::integral_constant<int, kVoteU>(), 0);
            continue;
        }
        // the last entries' load goes out first
        uint2 end = make_uint2(0u, 0u);
        if (full * 32 + lane < n)
            end = src[full * 32];
        if (full & 4)
            batch(std::integral_constant<int, 4>(), 0);
        if (full & 2)
            batch(std::integral_constant<int, 2>(), full & 4);
        if (full & 1)
            batch(std::integral_constant<int, 1>(), full & 6);
        for (int t = full * 32 + lane; t < n; t += 32) {
            const int ref = (int)end.x;
            if (ALL || (ref >= r0 && ref < r1)) {
                const uint32_t bin =
                    smm::vote_bin(t < vec, __uint_as_float(end.y), as, hAsT[h], smax);
                cast_vote<NARROW>(acc, (uint32_t)(ALL ? ref : ref - r0) * A + min(bin, last));
            }
            if (t + 32 < n) // (a round cut by the end of the blocks, and what is beyond it)
                end = src[t + 32 - lane];
        }
    }
}

// The rarer forms, out of line: inlined they take the common one's registers.
template <bool NARROW>
static __device__ __noinline__ void cast_items_call(const VoteArgs &a, uint32_t acc, const int *hOff,
                                                    const int *hCnt, const float *hAs,
                                                    const float *hAsT, const int *cPre, int h, int i0,
                                                    int i1, int r0, int r1) {
    cast_items<false, NARROW>(a, acc, hOff, hCnt, hAs, hAsT, cPre, h, i0, i1, r0, r1);
}

__device__ __forceinline__ void cast_votes(const VoteArgs &a, uint32_t *acc, const int *hOff,
                                           const int *hCnt, const float *hAs, const float *hAsT,
                                           const int *cPre, int nHits, int T, int r0, int r1,
                                           bool narrow) {
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int i0 = (int)((long long)T * w / nw), i1 = (int)((long long)T * (w + 1) / nw);
    if (i0 >= i1)
        return;
    int lo = 0, hi = nHits - 1; // the hit holding item i0: last h with cPre[h] <= i0
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (cPre[mid] <= i0)
            lo = mid;
        else
            hi = mid - 1;
    }
    const uint32_t at  = (uint32_t)__cvta_generic_to_shared(acc);
    const bool     all = r0 == 0 && r1 == a.ns; // one pass holds every reference point
    if (all && narrow)
        cast_items<true, true>(a, at, hOff, hCnt, hAs, hAsT, cPre, lo, i0, i1, r0, r1);
    else if (narrow)
        cast_items_call<true>(a, at, hOff, hCnt, hAs, hAsT, cPre, lo, i0, i1, r0, r1);
    else
        cast_items_call<false>(a, at, hOff, hCnt, hAs, hAsT, cPre, lo, i0, i1, r0, r1);
}

__device__ __forceinline__ int acc_get(const uint32_t *acc, int e, bool narrow) {
    return narrow ? (int)((acc[e >> 1] >> ((e & 1) * 16)) & 0xffffu) : (int)acc[e];
}

// Peaks of the accumulator rows of reference points [r0, r1) (ppf.cpp:363-389): first
// argmax, both circular neighbours added; rows whose total or maximum is below half the
// vote threshold are skipped. A thread per row; 16-bit rows of an even length are read two
// counters per 32-bit word. With FP, every non-zero cell is also folded into the
// fingerprint (a check of the whole accumulator, for tests).
template <bool FP>
__device__ __forceinline__ void peaks_rows(const VoteArgs &a, const uint32_t *acc, bool narrow,
                                           int r0, int r1, Cand top[3],
                                           unsigned long long &myHash) {
    const int   A     = a.A;
    const float thre  = a.voteThreshold / 2.0f;
    const bool  pairs = narrow && (A & 1) == 0;
    for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) {
        const int e0    = (i - r0) * A;
        int       total = 0, j = 0, best = -1;
        auto      cell  = [&](int t, int v) {
            total += v;
            if (v > best) {
                best = v;
                j    = t;
            }
            if (FP && v)
                myHash += smm::mix64(((unsigned long long)(i * A + t) << 32) | (uint32_t)v);
        };
        if (pairs) {
            const uint32_t *w = acc + (e0 >> 1);
            for (int t = 0; t < A; t += 2) {
                const uint32_t x = w[t >> 1];
                cell(t, (int)(x & 0xffffu));
                cell(t + 1, (int)(x >> 16));
            }
        } else {
            for (int t = 0; t < A; t++)
                cell(t, acc_get(acc, e0 + t, narrow));
        }
        if ((float)total < thre || (float)best < thre)
            continue;
        int vote = best;
        vote += acc_get(acc, e0 + ((j == 0) ? A - 1 : j - 1), narrow);
        vote += acc_get(acc, e0 + ((j == A - 1) ? 0 : j + 1), narrow);
        top3_insert(top, Cand{(float)vote, i, j});
    }
}

__device__ __forceinline__ void peaks_chunk(const VoteArgs &a, const uint32_t *acc, bool narrow,
                                            int r0, int r1, Cand top[3],
                                            unsigned long long &myHash) {
    if (a.fingerprint)
        peaks_rows<true>(a, acc, narrow, r0, r1, top, myHash);
    else
        peaks_rows<false>(a, acc, narrow, r0, r1, top, myHash);
}

__device__ __forceinline__ void dump_chunk(const VoteArgs &a, int c, const uint32_t *acc,
                                           bool narrow, int r0, int r1) {
    if (c >= a.dumpK)
        return;
    int      *d     = a.acc + ((size_t)c * a.ns + r0) * a.A;
    const int nElem = (r1 - r0) * a.A;
    for (int i = threadIdx.x; i < nElem; i += blockDim.x)
        d[i] = acc_get(acc, i, narrow);
}

// The keypoint's result: the block's top-3 candidates by (votes desc, reference asc), the
// poses of those within 95% of the best (ppf.cpp:391-409) and its statistics row
// {searched, 0, hits, votes, fingerprint, candidates, poses, counter bound}. wc needs
// blockDim/32 x 3 Cand, shash one zeroed word; both in shared memory.
__device__ __forceinline__ void finish_keypoint(const VoteArgs &a, int c, const smm::RT &rt,
                                                Cand top[3], unsigned long long myHash,
                                                long long searched, long long nHits,
                                                long long V, long long bound, Cand (*wc)[3],
                                                unsigned long long *shash) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        Cand other[3];
        for (int t = 0; t < 3; t++) {
            other[t].v = __shfl_xor_sync(0xffffffffu, top[t].v, o);
            other[t].r = __shfl_xor_sync(0xffffffffu, top[t].r, o);
            other[t].j = __shfl_xor_sync(0xffffffffu, top[t].j, o);
        }
        for (int t = 0; t < 3; t++)
            top3_insert(top, other[t]);
        myHash += __shfl_xor_sync(0xffffffffu, myHash, o);
    }
    if (lane == 0) {
        for (int t = 0; t < 3; t++)
            wc[w][t] = top[t];
        atomicAdd(shash, myHash);
    }
    __syncthreads();
    if (tid != 0)
        return;
    Cand t3[3];
    for (int t = 0; t < 3; t++)
        t3[t] = Cand{-1.0f, INT_MAX, 0};
    for (int ww = 0; ww < nw; ww++)
        for (int t = 0; t < 3; t++)
            if (wc[ww][t].r != INT_MAX)
                top3_insert(t3, wc[ww][t]);
    int nc = 0;
    for (int t = 0; t < 3; t++)
        nc += t3[t].r != INT_MAX ? 1 : 0;
    for (int t = 0; t < 3; t++) {
        float *cc = a.cands + (size_t)c * 9 + t * 3;
        cc[0]     = t < nc ? t3[t].v : -1.0f;
        cc[1]     = t < nc ? (float)t3[t].r : -1.0f;
        cc[2]     = t < nc ? (float)t3[t].j : -1.0f;
    }
    int npose = 0;
    if (nc > 0) {
        const float thr2 = (float)((double)t3[0].v * 0.95);
        for (int t = 0; t < nc; t++) {
            if (t3[t].v < thr2)
                continue;
            const float4  pm = a.sp[t3[t].r], nm = a.sn[t3[t].r];
            const smm::RT rm = smm::transform_rt(pm.x, pm.y, pm.z, nm.x, nm.y, nm.z);
            const float   al = smm::candidate_angle(t3[t].j, a.A - 1);
            smi::candidate_pose(rt, rm, al, t3[t].v,
                                a.poses + ((size_t)c * 3 + npose) * smi::kPoseFloats);
            npose++;
        }
    }
    for (int t = 0; t < 3; t++)
        a.poseOk[(size_t)c * 3 + t] = t < npose ? 1 : 0;
    long long *st = a.stats + (size_t)c * 8;
    st[0]         = searched;
    st[1]         = 0;
    st[2]         = nHits;
    st[3]         = V;
    st[4]         = (long long)*shash;
    st[5]         = nc;
    st[6]         = npose;
    st[7]         = bound;
}

// A keypoint that casts no votes: its normal is not finite (flag 1) or fewer neighbours
// than the vote threshold were found (flag 2).
__device__ __forceinline__ void skip_keypoint(const VoteArgs &a, int c, long long searched,
                                              bool nanN) {
    const int tid = threadIdx.x;
    long long *st = a.stats + (size_t)c * 8;
    if (tid < 8)
        st[tid] = tid == 0 ? searched : (tid == 1 ? (nanN ? 1 : 2) : 0);
    if (tid < 3) {
        a.poseOk[(size_t)c * 3 + tid] = 0;
        for (int e = 0; e < 3; e++)
            a.cands[(size_t)c * 9 + tid * 3 + e] = -1.0f;
    }
}

// Shared-memory sizing of the accumulator (host): 16-bit counters for all reference points
// when two CTAs of `staticBytes` then fit an SM, else as many reference points per pass as
// one CTA can hold; the 32-bit passes reuse the same bytes. Returns the dynamic bytes.
inline size_t acc_sizing(int ns, int A, long long staticBytes, int optin, int perSM,
                         int *refChunk, int *refChunkWide) {
    const long long narrowAll = ((long long)ns * A + 1) / 2 * 4;
    const long long cap       = optin - staticBytes;
    long long dyn = narrowAll + staticBytes + 1024 <= perSM / 2 ? narrowAll : std::min(narrowAll, cap);
    dyn           = std::max<long long>(dyn, (long long)A * 4) & ~3ll;
    if (dyn > cap)
        return 0;
    *refChunk     = (int)std::max<long long>(1, std::min<long long>(ns, dyn / 4 * 2 / A));
    *refChunkWide = (int)std::max<long long>(1, std::min<long long>(ns, dyn / 4 / A));
    return (size_t)dyn;
}

} // namespace vt
} // namespace sm
