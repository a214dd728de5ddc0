// vote_pipe.cu - the voting stage of matchScene (ppf.cpp:247-409) as a pipeline of
// kernels, each shaped for what it spends its time on.
//
//  1. k_kp_radius + k_kp_info, or k_kp_csr + k_rows_count: per keypoint its neighbour count, its
//     rows (neighbours other than itself) and the list position of its first "tail" row - the
//     reference computes a keypoint's rows in 8-lane blocks and the last (rows mod 8) one by
//     one, with different float rounding. In radius mode (all candidates within the model
//     diameter, in ascending order) the rows are kept as a bitmask over the candidate list,
//     computed from candidate tiles staged in shared memory and shared by 32 keypoints. In
//     reference order a candidate is a neighbour when the k-d tree's radius search reaches it,
//     and the tail rows are the last ones in the search's depth-first order.
//  2. A prefix sum over the rows gives every keypoint a segment of the hit list.
//  3. k_ppf: a CTA per keypoint (several where keypoints are few), each warp packing rows from
//     its share of the candidates until it has 32: quantised PPF key and model table probe by a
//     lane per row; the hits, packed again, pay for the scene alpha; a hit (bucket, count,
//     alpha) is appended to the keypoint's segment.
//  4. k_lpt: keypoints ordered by their vote count, largest first, so the heaviest
//     accumulators start first and the tail of the next kernel stays short.
//  5. k_vote_acc: one CTA per keypoint votes its hits into a shared-memory (reference
//     point x angle bin) accumulator - 16-bit counters when the keypoint's vote count
//     allows - then extracts peaks, the top three candidates and their poses.
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "sm_kdtree.cuh"
#include "sm_stages.h"
#include "sm_vote.cuh"

namespace sm {
using namespace smd;
using namespace vt;

void fill_vote_model(const Model &m, float minScore, VoteArgs &a);

namespace {

constexpr int kKpWarps   = 8;    // warps per CTA of the radius kernel
constexpr int kKpPer     = 4;    // keypoints per warp of it
constexpr int kTile      = 1024; // candidates per shared-memory tile
constexpr int kPpfBs     = 256;
// vote accumulation launch shapes the launch tuner chooses between - CTA size, and one CTA per
// keypoint or a persistent grid that takes keypoints from a device counter in LPT order;
// every one computes the same accumulators, peaks and candidates
constexpr int kAccBs[3]  = {256, 512, 1024};
constexpr int kAccShapes = 6; // shape s: CTA size kAccBs[s % 3], persistent when s >= 3
constexpr int kHitChunk  = 1024; // hits staged in shared memory per round
constexpr int kLptBins   = 40;

struct PipeBufs {
    int4               *info;    // K: {searched, rows voted (0 when skipped), first tail row, flags}
    smm::RT            *rt;      // K: transform of the keypoint
    uint32_t           *mask;    // K x words: row bits over the candidate list (radius mode)
    int                 words;
    int                 splits;  // radius mode: parts of the candidate list
    int2               *part;    // splits x K: {neighbours, rows} in the part
    VoteTree            tree;    // reference order
    int                *tail;    // reference order: K x 8, the tail rows' candidates (else -1)
    int                *rowOff;  // K + 1
    unsigned long long *rowSum;  // reference order: all rows (their 32-bit prefixes may wrap)
    int4               *hits;    // per row segment: {bucket offset, count, alpha bits, 0}
    int                *hitCnt;  // K
    unsigned long long *votes;   // K
    unsigned long long *bound;   // K: sum of the hits' bucket multiplicities (cell bound)
    int                *order;   // K
    int                *next;    // persistent accumulation: the next place in `order` to take
};

// flags: bit 0 = keypoint votes, bit 1 = its normal is not finite
__device__ __forceinline__ int4 kp_info(const VoteArgs &a, int searched, int R, int tail,
                                        const float4 &n1) {
    const bool nanN   = !(isfinite(n1.x) && isfinite(n1.y) && isfinite(n1.z));
    const bool active = !nanN && !((float)searched < a.voteThreshold);
    return make_int4(searched, active ? R : 0, tail, (active ? 1 : 0) | (nanN ? 2 : 0));
}

// Position of the first of the last `need` set bits of the warp's mask words [0, nw) (the
// first tail row); `n` when need == 0. All lanes return the same value.
__device__ __forceinline__ int tail_from_mask(const uint32_t *m, int nw, int need, int n) {
    const int lane  = threadIdx.x & 31;
    int       found = n;
    for (int base = nw - 1; base >= 0 && need > 0; base -= 32) {
        const int      wi = base - lane; // lane 0 = last word
        const uint32_t wv = wi >= 0 ? m[wi] : 0u;
        const int      k  = __popc(wv);
        // rows in words after this lane's word (lanes before it in this round)
        int incl = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += t;
        }
        const int      excl = incl - k;
        const bool     mine = excl < need && incl >= need;
        const uint32_t who  = __ballot_sync(0xffffffffu, mine);
        if (who) {
            const int src = __ffs(who) - 1;
            int       pos = 0;
            if (lane == src) {
                uint32_t b = wv; // the (need - excl)-th highest set bit of wv
                for (int t = 1; t < need - excl; t++)
                    b &= ~(0x80000000u >> __clz(b));
                pos = wi * 32 + (31 - __clz(b));
            }
            found = __shfl_sync(0xffffffffu, pos, src);
            need  = 0;
        } else {
            need -= __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    return found;
}

// Radius mode, part blockIdx.y of the candidates: kKpPer keypoints per warp over shared-memory
// tiles of the candidates' positions. The parts make CTAs enough: with one CTA per eight
// keypoints over all candidates, 2390 keypoints x 18,069 candidates took 145 us, now 54 us.
//
// TREE: a candidate nearer than its `sure` distance is reached; one between that and the radius
// waits in the warp's queue for the walk down its root path (smk::kd_reaches), a lane each 32 at
// a time. (A CTA per keypoint walking the path of every candidate within the radius took 1470 us
// for 2489 keypoints x 18,248 candidates, and the neighbour lists made from it another 170 us.)
template <bool TREE>
__global__ void __launch_bounds__(kKpWarps * 32) k_kp_radius(VoteArgs a, PipeBufs b, int per) {
    smd::chain_enter(); // launched chained
    __shared__ float4   tp[kTile]; // w: candidate id, TREE: its sure distance
    __shared__ uint32_t words[kKpWarps][kKpPer][TREE ? kTile / 32 : 1];
    __shared__ int      queue[kKpWarps][TREE ? 32 * kKpPer + 32 : 1]; // keypoint << 16 | place
    __shared__ float    kx[kKpWarps][kKpPer][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c0   = (blockIdx.x * kKpWarps + w) * kKpPer;
    const int i0 = blockIdx.y * per, i1 = min(a.ncand, i0 + per);
    if (TREE && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        *b.rowSum = 0ull; // (k_kp_info adds to it)
    int       self[kKpPer], S[kKpPer], R[kKpPer]; // self: the keypoint's id, TREE: its candidate
    float     x[kKpPer], y[kKpPer], z[kKpPer];
#pragma unroll
    for (int k = 0; k < kKpPer; k++) {
        const int    pid = c0 + k < a.K ? a.kp[c0 + k] : -1;
        const float4 p   = pid >= 0 ? a.pos[pid] : make_float4(0.f, 0.f, 0.f, 0.f);
        self[k]          = TREE && pid >= 0 ? b.tree.before[b.tree.treePos[pid]] : pid;
        x[k]             = p.x;
        y[k]             = p.y;
        z[k]             = p.z;
        S[k] = R[k] = 0;
        if (TREE && lane == 0) {
            kx[w][k][0] = p.x;
            kx[w][k][1] = p.y;
            kx[w][k][2] = p.z;
        }
    }
    for (int t0 = i0; t0 < i1; t0 += kTile) {
        const int tn = min(kTile, i1 - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < tn; i += blockDim.x) {
            const int    id = a.cand[t0 + i];
            const float4 q  = a.pos[id];
            tp[i] = make_float4(q.x, q.y, q.z, TREE ? b.tree.sure[t0 + i] : __int_as_float(id));
        }
        __syncthreads();
        if (c0 >= a.K)
            continue;
        int  nq   = 0;
        auto walk = [&](int n) { // the queue's last n <= 32 pairs
            if (lane < n) {
                const int e = queue[w][nq - n + lane], k = e >> 16, j = e & 0xffff;
                uint64_t  key;
                const int at = b.tree.posOf[t0 + j];
                if (smk::kd_sure(b.tree.view, kx[w][k], at, a.sqDiam) ||
                    smk::kd_reaches(b.tree.view, kx[w][k], at, a.sqDiam, &key))
                    atomicOr(&words[w][k][j >> 5], 1u << (j & 31));
            }
            nq -= n;
            __syncwarp();
        };
        for (int j = 0; j < tn; j += 32) {
            const bool   ok = j + lane < tn;
            const float4 q  = tp[ok ? j + lane : 0];
            uint32_t     word = 0;
#pragma unroll
            for (int k = 0; k < kKpPer; k++) {
                const float d  = smm::dist2(x[k], y[k], z[k], q.x, q.y, q.z);
                const bool  in = ok && d < a.sqDiam;
                if (TREE) {
                    const bool     sure = in && d < q.w;
                    const uint32_t row  = __ballot_sync(0xffffffffu, sure);
                    const uint32_t ask  = __ballot_sync(0xffffffffu, in && !sure && c0 + k < a.K);
                    if (in && !sure && c0 + k < a.K)
                        queue[w][nq + __popc(ask & ((1u << lane) - 1u))] = (k << 16) | (j + lane);
                    nq += __popc(ask); // (below 32 before the round)
                    word = lane == k ? row : word;
                } else {
                    S[k] += __popc(__ballot_sync(0xffffffffu, in));
                    const uint32_t row =
                        __ballot_sync(0xffffffffu, in && __float_as_int(q.w) != self[k]);
                    R[k] += __popc(row);
                    word = lane == k ? row : word;
                }
            }
            if (TREE) {
                if (lane < kKpPer)
                    words[w][lane][j >> 5] = word;
                __syncwarp();
                while (nq >= 32)
                    walk(32);
            } else if (lane < kKpPer && c0 + lane < a.K) {
                b.mask[(size_t)(c0 + lane) * b.words + ((t0 + j) >> 5)] = word;
            }
        }
        if (TREE) {
            if (nq > 0)
                walk(nq);
#pragma unroll
            for (int k = 0; k < kKpPer; k++) { // a word per lane: counts, the keypoint taken out
                if (c0 + k >= a.K || lane * 32 >= tn)
                    continue;
                uint32_t m = words[w][k][lane];
                S[k] += __popc(m);
                if ((self[k] - t0) >> 5 == lane)
                    m &= ~(1u << ((self[k] - t0) & 31));
                R[k] += __popc(m);
                b.mask[(size_t)(c0 + k) * b.words + (t0 >> 5) + lane] = m;
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int k = 0; k < kKpPer; k++) {
        if (TREE) {
            S[k] = __reduce_add_sync(0xffffffffu, S[k]);
            R[k] = __reduce_add_sync(0xffffffffu, R[k]);
        }
        if (lane == k && c0 + k < a.K)
            b.part[(size_t)blockIdx.y * a.K + c0 + k] = make_int2(S[k], R[k]);
    }
}

// Set bits of the mask row in [l, r), by a warp.
__device__ __forceinline__ int mask_count(const uint32_t *mask, int l, int r) {
    int n = 0;
    if (l < r)
        for (int w = (l >> 5) + (int)(threadIdx.x & 31); w <= (r - 1) >> 5; w += 32) {
            uint32_t m = mask[w];
            if (w == l >> 5)
                m &= ~0u << (l & 31);
            if (w == (r - 1) >> 5)
                m &= ~0u >> (31 - ((r - 1) & 31));
            n += __popc(m);
        }
    return __reduce_add_sync(0xffffffffu, n);
}

// The last n set bits of the mask row in [l, r) (at least n are set), to out[0..n), by a warp.
__device__ __forceinline__ void mask_last(const uint32_t *mask, int l, int r, int n, int *out) {
    const int lane = threadIdx.x & 31;
    int       at   = 0;
    for (int w1 = (r - 1) >> 5; at < n && w1 >= l >> 5; w1 -= 32) {
        const int w = w1 - lane; // lane 0: the last word
        uint32_t  m = w >= l >> 5 ? mask[w] : 0u;
        if (w == l >> 5)
            m &= ~0u << (l & 31);
        if (w == (r - 1) >> 5)
            m &= ~0u >> (31 - ((r - 1) & 31));
        const int incl = warp_incl_scan(__popc(m));
        int       k    = at + incl - __popc(m);
        while (m && k < n) {
            const int bit = 31 - __clz(m);
            m ^= 1u << bit;
            out[k++] = w * 32 + bit;
        }
        at += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// The last `need` of a keypoint's rows in the depth-first order of its radius search (nearer
// child first): from the root, a far child that holds as many is where they lie, one that holds
// fewer gives all of its own. Rows of a subtree are a range of the mask, as the candidates are
// in tree order.
__device__ __forceinline__ void tree_tail(const VoteTree &T, const uint32_t *mask, const float q[3],
                                          int need, int *out) {
    int v = 0, l = 0, r = T.m;
    while (need > 0) {
        const int4 n = T.view.nd[v];
        if (smk::is_leaf(n)) {
            mask_last(mask, T.before[n.x], T.before[n.y], need, out);
            return;
        }
        const int   f     = smk::divfeat_of(n);
        const float val   = f == 0 ? q[0] : f == 1 ? q[1] : q[2];
        const bool  near1 = ((val - __int_as_float(n.x)) + (val - __int_as_float(n.y))) < 0.0f;
        const int   fl = near1 ? n.w : l, fr = near1 ? r : n.w; // the far child's positions
        const int   cl = T.before[fl], cr = T.before[fr];
        const int   c  = mask_count(mask, cl, cr);
        const int   c1 = smk::child1_of(n);
        if (c >= need) {
            v = near1 ? c1 + 1 : c1;
            l = fl;
            r = fr;
            continue;
        }
        mask_last(mask, cl, cr, c, out);
        out += c;
        need -= c;
        v = near1 ? c1 : c1 + 1;
        l = near1 ? l : n.w;
        r = near1 ? n.w : r;
    }
}

// Radius mode, a warp per keypoint: its counts over the parts, its tail rows, its transform; the
// row counts (cnt[K] = 0 closes the scan's input), and the per-keypoint hit counters and vote
// totals cleared for k_ppf.
template <bool TREE> __global__ void k_kp_info(VoteArgs a, PipeBufs b, int *__restrict__ cnt) {
    smd::chain_enter(); // launched chained
    const int lane = threadIdx.x & 31;
    const int c    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= a.K)
        return;
    int S = 0, R = 0;
    for (int s = lane; s < b.splits; s += 32) {
        const int2 v = b.part[(size_t)s * a.K + c];
        S += v.x;
        R += v.y;
    }
    S = __reduce_add_sync(0xffffffffu, S);
    R = __reduce_add_sync(0xffffffffu, R);
    const int       pid  = a.kp[c];
    const float4    p1   = a.pos[pid];
    const uint32_t *mask = b.mask + (size_t)c * b.words;
    int             tail = 0;
    if (TREE) {
        const float q[3] = {p1.x, p1.y, p1.z};
        if (lane < 8)
            b.tail[(size_t)c * 8 + lane] = -1;
        __syncwarp();
        tree_tail(b.tree, mask, q, R % smm::kLanes, b.tail + (size_t)c * 8);
    } else {
        tail = tail_from_mask(mask, b.words, R % smm::kLanes, a.ncand);
    }
    if (lane != 0)
        return;
    const float4 n1   = a.nrm[pid];
    const int4   info = kp_info(a, S, R, tail, n1);
    b.info[c]         = info;
    b.rt[c]           = smm::transform_rt(p1.x, p1.y, p1.z, n1.x, n1.y, n1.z);
    cnt[c]            = info.y;
    if (TREE)
        atomicAdd(b.rowSum, (unsigned long long)info.y);
    b.hitCnt[c]       = 0;
    b.votes[c]        = 0ull;
    b.bound[c]        = 0ull;
    if (c == 0)
        cnt[a.K] = 0;
}

// CSR mode: one warp per keypoint over its list.
__global__ void k_kp_csr(VoteArgs a, PipeBufs b) {
    smd::chain_enter(); // launched chained
    const int lane = threadIdx.x & 31;
    const int c    = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (c >= a.K)
        return;
    const int  pid = a.kp[c];
    const int  beg = a.nbrOff[c], len = a.nbrOff[c + 1] - beg;
    const int *L   = a.nbrIds + beg;
    int        R   = 0;
    for (int i = lane; i < len; i += 32)
        R += L[i] != pid ? 1 : 0;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
        R += __shfl_xor_sync(0xffffffffu, R, o);
    int need = R % smm::kLanes, found = len;
    for (int end = len; end > 0 && need > 0; end -= 32) {
        const int i = end - 1 - lane;
        uint32_t  m = __ballot_sync(0xffffffffu, i >= 0 && L[i] != pid);
        const int k = __popc(m);
        if (k >= need) {
            for (int t = 1; t < need; t++)
                m &= m - 1;
            found = end - 1 - (__ffs(m) - 1);
            need  = 0;
        } else {
            need -= k;
        }
    }
    if (lane == 0) {
        const float4 p1 = a.pos[pid], n1 = a.nrm[pid];
        b.info[c]       = kp_info(a, len, R, found, n1);
        b.rt[c]         = smm::transform_rt(p1.x, p1.y, p1.z, n1.x, n1.y, n1.z);
    }
}

// Row counts per keypoint (cnt[K] = 0 closes the scan's input), and the per-keypoint hit
// counters and vote totals cleared for k_ppf.
__global__ void k_rows_count(const int4 *__restrict__ info, int K, int *__restrict__ cnt,
                             PipeBufs b) {
    smd::chain_enter(); // launched chained
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0)
        cnt[K] = 0;
    if (c < K) {
        cnt[c]      = info[c].y;
        b.hitCnt[c] = 0;
        b.votes[c]  = 0ull;
        b.bound[c]  = 0ull;
    }
}

// Keypoint blockIdx.x; its 8 x gridDim.y warps take its candidates (CSR: list entries) 128 at a
// time in turn. A warp packs the rows it finds into its queue (a few of 32 candidates are rows:
// a lane per candidate would idle) and takes 32 at a time, a lane each, for the PPF key and the
// table probe; the few hits wait in a second queue for the scene alpha. No barriers: the warps of
// a CTA share nothing. (8.4 M rows: through a row list in global memory, with the alpha of every
// row, 51 + 248 us; packed by the whole CTA between barriers 532 us; now 267 us, mostly the
// issue of the keys' arithmetic, some 700 instructions a row with its divisions and arc tangents.)
enum RowSource { kRowsMask, kRowsTree, kRowsCsr }; // tree: a mask with listed tail rows

template <RowSource SRC>
__global__ void __launch_bounds__(kPpfBs, 5) k_ppf(VoteArgs a, PipeBufs b) {
    smd::chain_enter(); // launched chained
    constexpr int  W   = kPpfBs / 32;
    constexpr bool CSR = SRC == kRowsCsr;
    __shared__ int  rowQ[W][160]; // point * 2 + block lane
    __shared__ int4 hitQ[W][64];  // {row, bucket offset, count, multiplicity}
    const int  c    = blockIdx.x;
    const int4 info = b.info[c];
    if (info.y == 0)
        return;
    const int       lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t  below = (1u << lane) - 1u;
    const int       pid   = a.kp[c];
    const float4    p1 = a.pos[pid], n1 = a.nrm[pid];
    const int       beg = CSR ? a.nbrOff[c] : 0;
    const int       len = CSR ? a.nbrOff[c + 1] - beg : a.ncand;
    const uint32_t *mask = CSR ? nullptr : b.mask + (size_t)c * b.words;
    int            *rq   = rowQ[w];
    int4           *hq   = hitQ[w];
    int             nr = 0, nh = 0;
    unsigned long long votes = 0, bound = 0;

    auto take_hits = [&](int n) { // the queue's last n <= 32 hits
        const int4 v  = lane < n ? hq[nh - n + lane] : make_int4(0, 0, 0, 0);
        float      as = 0.0f;
        bool       ok = lane < n;
        if (ok) {
            const float4  q  = a.pos[v.x >> 1];
            const smm::RT rt = b.rt[c];
            as               = smm::alpha_of((v.x & 1) != 0, rt, q.x, q.y, q.z);
            ok               = !smm::fisnan(as);
        }
        nh -= n;
        const uint32_t m    = __ballot_sync(0xffffffffu, ok);
        int            base = 0;
        if (lane == 0 && m)
            base = atomicAdd(&b.hitCnt[c], __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (ok) {
            b.hits[b.rowOff[c] + base + __popc(m & below)] =
                make_int4(v.y, v.z, __float_as_int(as), 0);
            votes += (unsigned)v.z;
            bound += (unsigned)v.w;
        }
    };
    auto take_rows = [&](int n) { // the queue's last n <= 32 rows
        uint32_t off = 0, mult = 0;
        int      cnt = 0, row = 0;
        if (lane < n) {
            row                = rq[nr - n + lane];
            const float4   p2 = a.pos[row >> 1], n2 = a.nrm[row >> 1];
            const uint32_t key =
                smm::ppf_key((row & 1) != 0, p1.x, p1.y, p1.z, n1.x, n1.y, n1.z, p2.x, p2.y, p2.z,
                             n2.x, n2.y, n2.z, a.angleStep, a.distStep);
            cnt = (int)probe(a.htab, a.hmask, key, off, mult);
        }
        nr -= n;
        const uint32_t m = __ballot_sync(0xffffffffu, cnt > 0);
        if (cnt > 0)
            hq[nh + __popc(m & below)] = make_int4(row, (int)off, cnt, (int)mult);
        nh += __popc(m); // (below 32 before: 64 entries hold it)
        __syncwarp();
        if (nh >= 32)
            take_hits(32);
        __syncwarp(); // (the queues' places are written again after their reads)
    };

    const int tail = SRC == kRowsTree ? b.tail[(size_t)c * 8 + (lane & 7)] : -1;
    const int step = gridDim.y * W * 128;
    for (int i0 = (blockIdx.y * W + w) * 128; i0 < len; i0 += step) {
        uint32_t m[4];
        int      id[4];
#pragma unroll
        for (int k = 0; k < 4; k++) { // the loads of 128 candidates in flight
            const int i = i0 + k * 32 + lane;
            if (CSR)
                id[k] = i < len ? a.nbrIds[beg + i] : pid;
            else
                m[k] = i0 + k * 32 < len ? mask[(i0 >> 5) + k] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (CSR)
                m[k] = __ballot_sync(0xffffffffu, id[k] != pid);
            else if ((m[k] >> lane) & 1u)
                id[k] = a.cand[i0 + k * 32 + lane];
        }
        // the lane's rows that the reference computes one by one
        unsigned single = 0u;
        if (SRC == kRowsTree) {
            uint32_t here = __ballot_sync(0xffffffffu, lane < 8 && tail >= 0 && (tail ^ i0) < 128);
            while (here) {
                const int t = __shfl_sync(0xffffffffu, tail, __ffs(here) - 1) - i0;
                here &= here - 1u;
                if ((t & 31) == lane)
                    single |= 1u << (t >> 5);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const bool block =
                SRC == kRowsTree ? !((single >> k) & 1u) : i0 + k * 32 + lane < info.z;
            if ((m[k] >> lane) & 1u)
                rq[nr + __popc(m[k] & below)] = id[k] * 2 + (block ? 1 : 0);
            nr += __popc(m[k]); // (below 32 before: 160 entries hold 128 more)
        }
        __syncwarp();
        while (nr >= 32)
            take_rows(32);
    }
    if (nr > 0)
        take_rows(nr);
    if (nh > 0)
        take_hits(nh);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        votes += __shfl_xor_sync(0xffffffffu, votes, o);
        bound += __shfl_xor_sync(0xffffffffu, bound, o);
    }
    if (lane == 0 && votes) {
        atomicAdd(&b.votes[c], votes);
        atomicAdd(&b.bound[c], bound);
    }
}

__device__ __forceinline__ int lpt_bin(unsigned long long v) {
    return v == 0 ? 0 : min(kLptBins - 1, 64 - __clzll((long long)v));
}

// Keypoints by vote count, largest first (binned by powers of two).
__global__ void k_lpt(const unsigned long long *__restrict__ votes, int K, int *__restrict__ order,
                      int *__restrict__ next) {
    smd::chain_enter(); // launched chained
    __shared__ int hist[kLptBins], start[kLptBins];
    if (threadIdx.x == 0)
        *next = 0; // the persistent vote grid's work counter
    if (threadIdx.x < kLptBins)
        hist[threadIdx.x] = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < K; c += blockDim.x)
        atomicAdd(&hist[lpt_bin(votes[c])], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int k = kLptBins - 1; k >= 0; k--) {
            start[k] = s;
            s += hist[k];
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < K; c += blockDim.x)
        order[atomicAdd(&start[lpt_bin(votes[c])], 1)] = c;
}

// One CTA per keypoint (in LPT order by block index), or with PERSIST a resident grid whose
// CTAs take the next keypoint of the LPT order from a device counter until none is left.
template <int BS, bool PERSIST>
__global__ void __launch_bounds__(BS, BS >= 1024 ? 1 : 2) k_vote_acc(VoteArgs a, PipeBufs b) {
    smd::chain_enter(); // launched chained
    extern __shared__ uint32_t acc[];
    __shared__ int       hOff[kHitChunk], hCnt[kHitChunk], cPre[kHitChunk + 1];
    __shared__ float     hAs[kHitChunk], hAsT[kHitChunk];
    __shared__ int       sh[33];
    __shared__ Cand      wc[BS / 32][3];
    __shared__ unsigned long long shash;
    __shared__ int       sNext;

    const int tid = threadIdx.x;
    for (int it = 0;; it++) {
        int idx = blockIdx.x;
        if (PERSIST) {
            if (tid == 0)
                sNext = atomicAdd(b.next, 1);
            __syncthreads();
            idx = sNext;
            __syncthreads();
            if (idx >= a.K)
                return;
        } else if (it > 0) {
            return;
        }
        const int  c    = b.order[idx];
        const int4 info = b.info[c];
        if (!(info.w & 1)) {
            skip_keypoint(a, c, info.x, (info.w & 2) != 0);
            continue;
        }
        if (tid == 0)
            shash = 0;
        const long long V      = (long long)b.votes[c];
        const long long bound  = (long long)b.bound[c];
        const int       nH     = b.hitCnt[c];
        const int4     *H      = b.hits + b.rowOff[c];
        const bool      narrow = bound <= kNarrowMax && !a.forceWide; // no cell can pass 65535
        const int       chunk  = narrow ? a.refChunk : a.refChunkWide;
        Cand            top[3];
        for (int t = 0; t < 3; t++)
            top[t] = Cand{-1.0f, INT_MAX, 0};
        unsigned long long myHash = 0;
        for (int r0 = 0; r0 < a.ns; r0 += chunk) {
            const int r1     = min(r0 + chunk, a.ns);
            const int nElem  = (r1 - r0) * a.A;
            const int nWords = narrow ? (nElem + 1) >> 1 : nElem;
            for (int i = tid; i < nWords; i += BS)
                acc[i] = 0u;
            for (int h0 = 0; h0 < nH; h0 += kHitChunk) {
                const int n = min(kHitChunk, nH - h0);
                __syncthreads();
                int T = 0;
                for (int j0 = 0; j0 < n; j0 += BS) {
                    const int j   = j0 + tid;
                    int       nit = 0;
                    if (j < n) {
                        const int4 hv = H[h0 + j];
                        hOff[j]       = hv.x;
                        hCnt[j]       = hv.y;
                        hAs[j]        = __int_as_float(hv.z);
                        hAsT[j]       = smm::alpha_tail_shift(__int_as_float(hv.z));
                        nit           = (hv.y + kItem - 1) / kItem;
                    }
                    int       tot;
                    const int pre = block_excl_scan(nit, sh, &tot);
                    if (j < n)
                        cPre[j] = T + pre;
                    T += tot;
                }
                if (tid == 0)
                    cPre[n] = T;
                __syncthreads();
                cast_votes(a, acc, hOff, hCnt, hAs, hAsT, cPre, n, T, r0, r1, narrow);
            }
            __syncthreads();
            peaks_chunk(a, acc, narrow, r0, r1, top, myHash);
            dump_chunk(a, c, acc, narrow, r0, r1);
            __syncthreads();
        }
        finish_keypoint(a, c, b.rt[c], top, myHash, info.x, nH, V, bound, wc, &shash);
        __syncthreads(); // the shared buffers serve the CTA's next keypoint
    }
}

const void *vote_acc_fn(int shape) {
    switch (shape) {
    case 0: return (const void *)k_vote_acc<kAccBs[0], false>;
    case 1: return (const void *)k_vote_acc<kAccBs[1], false>;
    case 2: return (const void *)k_vote_acc<kAccBs[2], false>;
    case 3: return (const void *)k_vote_acc<kAccBs[0], true>;
    case 4: return (const void *)k_vote_acc<kAccBs[1], true>;
    default: return (const void *)k_vote_acc<kAccBs[2], true>;
    }
}

// Dynamic shared memory of the accumulator for launch shape `shape` (its static shared
// memory differs a little by CTA size); 0 when it does not fit.
size_t vote_acc_smem(int shape, const Ctx &c, VoteArgs &a) {
    int optin = 0, perSM = 0;
    SM_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    SM_CUDA(cudaDeviceGetAttribute(&perSM, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c.device));
    cudaFuncAttributes fa;
    SM_CUDA(cudaFuncGetAttributes(&fa, vote_acc_fn(shape)));
    const size_t smem = acc_sizing(a.ns, a.A, (long long)fa.sharedSizeBytes, optin, perSM,
                                   &a.refChunk, &a.refChunkWide);
    if (smem && smem > allow_dynamic_smem(vote_acc_fn(shape), c.device))
        return 0;
    return smem;
}

// counterClear: the persistent grid's work counter is zero already (k_lpt clears it; each
// of the tuner's timed launches uses it up).
void launch_vote_acc(int shape, const Ctx &c, const VoteArgs &a, const PipeBufs &b, int K,
                     size_t smem, bool counterClear) {
    const int bs = kAccBs[shape % 3];
    int       g  = K;
    if (shape >= 3) {
        // one resident wave, keypoints from the counter
        int per = 0, nsm = 0;
        SM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, vote_acc_fn(shape), bs, smem));
        SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
        g = std::max(1, std::min(K, std::max(per, 1) * nsm));
        if (!counterClear)
            SM_CUDA(cudaMemsetAsync(b.next, 0, sizeof(int), c.stream));
    }
    switch (shape) {
    case 0: launch_chained(c, k_vote_acc<kAccBs[0], false>, g, bs, smem, a, b); break;
    case 1: launch_chained(c, k_vote_acc<kAccBs[1], false>, g, bs, smem, a, b); break;
    case 2: launch_chained(c, k_vote_acc<kAccBs[2], false>, g, bs, smem, a, b); break;
    case 3: launch_chained(c, k_vote_acc<kAccBs[0], true>, g, bs, smem, a, b); break;
    case 4: launch_chained(c, k_vote_acc<kAccBs[1], true>, g, bs, smem, a, b); break;
    default: launch_chained(c, k_vote_acc<kAccBs[2], true>, g, bs, smem, a, b); break;
    }
}

// The launch tuner: per device, the vote accumulation shape measured fastest on the first
// call with at least kTuneMinK keypoints (each shape timed twice with CUDA events on the
// call's own data, the faster of the two runs kept), then used for every later call.
// SM_VOTE_SHAPE=256|512|1024, with a trailing 'p' for the persistent grid, in the
// environment fixes the shape instead (tests).
constexpr int    kTuneMinK = 512;
std::atomic<int> g_voteShape[64] = {};     // 0 untuned, else 1 + shape index
std::mutex       g_tuneMu;

int forced_vote_shape() {
    const char *e = std::getenv("SM_VOTE_SHAPE");
    if (!e)
        return -1;
    const int  v       = std::atoi(e);
    const bool persist = std::strchr(e, 'p') != nullptr;
    for (int s = 0; s < 3; s++)
        if (kAccBs[s] == v)
            return s + (persist ? 3 : 0);
    return -1;
}

} // namespace

int vote_tuned_shape(int device, int *persistent) {
    *persistent = 0;
    if (device < 0 || device >= 64)
        return 0;
    const int t = g_voteShape[device].load();
    if (t <= 0)
        return 0;
    *persistent = t - 1 >= 3 ? 1 : 0;
    return kAccBs[(t - 1) % 3];
}

void vote(Ctx &c, const Model &m, const float4 *pos, const float4 *nrm, const int *kp, int K,
          const int *nbrOff, const int *nbrIds, const int *cand, int ncand, float minScore,
          const VoteOut &out, int dumpK, const VoteTree *tree) {
    if (K <= 0)
        return;
    // rows (keypoint, neighbour) are counted and offset in 32-bit ints: at most K x ncand in
    // radius mode (every candidate a neighbour of every keypoint). Grid order refuses what could
    // be more, reference order what is.
    const char *const tooMany = "too many keypoint x sampled point pairs for one call";
    const bool        many    = !nbrOff && (long long)K * (long long)ncand > 0x7fffffffll;
    if (many && !tree)
        throw Error(SM_ERR_CAPACITY, tooMany);
    VoteArgs a{};
    fill_vote_model(m, minScore, a);
    a.pos    = pos;
    a.nrm    = nrm;
    a.kp     = kp;
    a.K      = K;
    a.nbrOff = nbrOff;
    a.nbrIds = nbrIds;
    a.cand   = cand;
    a.ncand  = ncand;
    a.stats  = out.stats;
    a.cands  = out.cands;
    a.poses  = out.poses;
    a.poseOk = out.poseOk;
    a.acc    = out.acc;
    a.dumpK  = out.acc ? dumpK : 0;
    // SM_VOTE_FORCE_WIDE=1 runs every keypoint on 32-bit counters, a regime that the cell
    // bound otherwise reserves for extreme inputs, so that tests reach it
    const char *fw = std::getenv("SM_VOTE_FORCE_WIDE");
    a.forceWide    = (fw && fw[0] == '1') ? 1 : 0;
    // SM_VOTE_FINGERPRINT=1 folds every accumulator into stats column 4 (checked by tests
    // against the oracle); without it the column is 0 and the peak scan skips the work
    const char *fp = std::getenv("SM_VOTE_FINGERPRINT");
    a.fingerprint  = (fp && fp[0] == '1') ? 1 : 0;

    const bool csr = nbrOff != nullptr;

    // the accumulation's launch shape: forced, tuned on this device, or the default (512)
    const int dev    = c.device >= 0 && c.device < 64 ? c.device : 0;
    const int forced = forced_vote_shape();
    int       shape  = forced >= 0 ? forced : (g_voteShape[dev].load() > 0 ? g_voteShape[dev].load() - 1 : 1);
    const bool tune  = forced < 0 && g_voteShape[dev].load() == 0 && K >= kTuneMinK;
    size_t     smem  = vote_acc_smem(shape, c, a);
    if (!smem)
        throw Error(SM_ERR_CAPACITY, "featAngleResolution too large for the vote accumulator");

    PipeBufs b{};
    b.info   = c.arena.get<int4>("v.info", K);
    b.rt     = c.arena.get<smm::RT>("v.rt", K);
    b.words  = csr ? 0 : (ncand + 31) / 32;
    b.mask   = csr ? nullptr : c.arena.get<uint32_t>("v.mask", (size_t)K * std::max(b.words, 1));
    b.rowOff = c.arena.get<int>("v.rowoff", (size_t)K + 1);
    b.hitCnt = c.arena.get<int>("v.hitcnt", K);
    b.votes  = c.arena.get<unsigned long long>("v.votes", K);
    b.bound  = c.arena.get<unsigned long long>("v.bound", K);
    b.order  = c.arena.get<int>("v.order", K);
    b.next   = c.arena.get<int>("v.next", 1);
    int *cnt = c.arena.get<int>("v.rowcnt", (size_t)K + 1);
    int  nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    if (csr) {
        launch_chained(c, k_kp_csr, nblocks((long long)K * 32, 256), 256, 0, a, b);
        launch_chained(c, k_rows_count, nblocks(K, 256), 256, 0, b.info, K, cnt, b);
    } else {
        // parts of the candidate list (whole mask words, 256 candidates at least) so that some
        // four CTAs per SM run
        const int gx   = nblocks(K, kKpPer * kKpWarps);
        const int want = std::max(1, std::min(nblocks(ncand, 256), nblocks(4LL * nsm, gx)));
        const int per  = nblocks(nblocks(ncand, want), 32) * 32;
        b.splits       = std::max(1, nblocks(ncand, per));
        b.part         = c.arena.get<int2>("v.part", (size_t)b.splits * K);
        const int gi   = nblocks((long long)K * 32, 256);
        if (tree) {
            b.tree = *tree;
            b.tail = c.arena.get<int>("v.tail", (size_t)K * 8);
            b.rowSum = c.arena.get<unsigned long long>("v.rowsum", 1);
            launch_chained(c, k_kp_radius<true>, dim3(gx, b.splits), kKpWarps * 32, 0, a, b, per);
            launch_chained(c, k_kp_info<true>, gi, 256, 0, a, b, cnt);
        } else {
            launch_chained(c, k_kp_radius<false>, dim3(gx, b.splits), kKpWarps * 32, 0, a, b, per);
            launch_chained(c, k_kp_info<false>, gi, 256, 0, a, b, cnt);
        }
    }
    unsigned long long *rowSum = reinterpret_cast<unsigned long long *>(c.hostCounts + 2);
    *rowSum                    = 0ull;
    if (many) // (read with the scan's total)
        SM_CUDA(cudaMemcpyAsync(rowSum, b.rowSum, sizeof(*rowSum), cudaMemcpyDeviceToHost, c.stream));
    const int rtot = scan_excl(c, cnt, b.rowOff, (long long)K + 1, "v.scan", true);
    if (*rowSum > 0x7fffffffull)
        throw Error(SM_ERR_CAPACITY, tooMany);
    b.hits = c.arena.get<int4>("v.hits", std::max(rtot, 1));
    SM_CUDA(cudaEventRecord(c.ev[10], c.stream));
    if (rtot > 0) {
        // several CTAs per keypoint where the keypoints would not fill the SMs (for CSR lists as
        // far as the rows could need them)
        const int most = nblocks(csr ? rtot : ncand, 128 * (kPpfBs / 32));
        const int gy   = std::max(1, std::min(most, nblocks(4LL * nsm, K)));
        if (csr)
            launch_chained(c, k_ppf<kRowsCsr>, dim3(K, gy), kPpfBs, 0, a, b);
        else if (tree)
            launch_chained(c, k_ppf<kRowsTree>, dim3(K, gy), kPpfBs, 0, a, b);
        else
            launch_chained(c, k_ppf<kRowsMask>, dim3(K, gy), kPpfBs, 0, a, b);
    }
    SM_CUDA(cudaEventRecord(c.ev[11], c.stream));
    launch_chained(c, k_lpt, 1, 1024, 0, b.votes, K, b.order, b.next);
    if (tune) {
        // every shape computes the same outputs: time each on this call's keypoints, keep
        // the fastest for the device (one process-wide decision, taken once)
        std::lock_guard<std::mutex> lk(g_tuneMu);
        if (g_voteShape[dev].load() == 0) {
            cudaEvent_t e0, e1;
            SM_CUDA(cudaEventCreate(&e0));
            SM_CUDA(cudaEventCreate(&e1));
            float best[kAccShapes];
            for (int sh = 0; sh < kAccShapes; sh++)
                best[sh] = 1e30f;
            for (int rep = 0; rep < 2; rep++)
                for (int sh = 0; sh < kAccShapes; sh++) {
                    VoteArgs     at = a;
                    const size_t sm = vote_acc_smem(sh, c, at);
                    if (!sm)
                        continue;
                    SM_CUDA(cudaEventRecord(e0, c.stream));
                    launch_vote_acc(sh, c, at, b, K, sm, false);
                    SM_CUDA(cudaEventRecord(e1, c.stream));
                    SM_CUDA(cudaEventSynchronize(e1));
                    float ms = 0.0f;
                    SM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                    best[sh] = std::min(best[sh], ms);
                }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            int pick = 1;
            for (int sh = 0; sh < kAccShapes; sh++)
                if (best[sh] < best[pick])
                    pick = sh;
            g_voteShape[dev].store(1 + pick);
        }
        shape = g_voteShape[dev].load() - 1;
        smem  = vote_acc_smem(shape, c, a);
    }
    SM_CUDA(cudaEventRecord(c.ev[12], c.stream));
    launch_vote_acc(shape, c, a, b, K, smem, !tune);
    SM_CUDA(cudaEventRecord(c.ev[13], c.stream));
}

} // namespace sm
