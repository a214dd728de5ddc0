// cluster.cu - pose clustering of matchScene (ppf.cpp:414-418): sortPoses, clusterPose,
// avgClusters, sortPoses, clusterPose2 (util.cpp:486-601).
//
// Both clusterings are greedy first fits: in order, an entry joins the first earlier head (leader)
// it is compatible with, or becomes one. Taken one after the other they are a chain as long as the
// list (a warp's walk over 8083 poses took 9 ms; all the clustering takes 0.33 ms now), so they
// are resolved a chunk of kClBs entries at a time from the compatibility bits of the chunk's pairs,
// in parallel rounds that reproduce the sequential decisions (greedy_chunk), after the entries that
// fit a head of an earlier chunk were taken out.
//
// k_cluster_rank (all CTAs): stable rank-by-counting sort on (votes desc, list position).
// k_cluster_bits (all CTAs): the compatibility of every pose with the earlier ones of its chunk.
// Per chunk k_cluster_heads (one CTA): its heads and their members in it; k_cluster_join (all
// CTAs): the later poses' first fit among its heads - first in creation order, since the earlier
// chunks' heads were tried before. k_cluster_avg: one block per cluster sums its members in pose
// order (FP32 translation, FP64 quaternion moments) and averages them, so the clusters' FP64 work
// spreads over the SMs. k_cluster_b (one CTA): the second sort (k_cluster_rank2 for long lists)
// and clusterPose2. Results are identical to the oracle's sequential restatement.
#include <cmath>
#include <cstring>

#include "sm_icp.h"
#include "sm_stages.h"

namespace sm {

namespace {

constexpr int kClBs   = 1024;
constexpr int PF      = smi::kPoseFloats;
struct ClArgs {
    const float *poses;
    int          np;
    float        sqThr, angThr, cx, cy, cz, thr2;
    float       *sorted;    // np x PF
    float       *avg;       // np x PF (cluster creation order)
    float       *avgSorted; // np x PF
    float4      *tr;        // np
    float       *out;       // np x PF
    int         *outCount;
    float4      *key;       // np: sorted {tx, ty, tz, angle}
    float       *sum;       // np: the leaders' vote sums
    float4      *tv, *qv;   // np each: sorted {tx, ty, tz, votes} and quaternions
    int         *clu;       // np: cluster number per sorted pose (-1: none yet)
    int         *heads;     // np: pose index of each cluster head; later the leaders
    int         *nh;        // clusters, and how many there were before the last chunk
    uint32_t    *bits;      // per chunk 32 kClBs compatibility words (k_cluster_bits)
};

// clusterPose compatibility of pose a with head b (util.cpp:499-520); the distance test
// sqrt(v) < distThr is evaluated as v < sqThr (exact: see sqrt_lt_bound).
__device__ __forceinline__ bool compat(const float4 &a, const float4 &b, float sqThr, float angThr) {
    const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    return x * x + (y * y + z * z) < sqThr && smm::fabs_(a.w - b.w) < angThr;
}

// sortPoses (util.cpp:486-491) as a stable rank by votes (float 17) descending: the rank of entry i
// of n of `in`, by P neighbouring lanes of a block whose threads all call it (i >= n: none). The
// votes are staged in shared memory, a run at a time.
constexpr int kRankRun = 2048;
template <int P>
__device__ __forceinline__ int rank_by_votes(const float *in, int n, int i, float *sv) {
    const int   sub  = threadIdx.x % P;
    const float v    = i < n ? in[(size_t)i * PF + 17] : 0.0f;
    int         rank = 0;
    for (int j0 = 0; j0 < n; j0 += kRankRun) {
        const int m = min(n - j0, kRankRun);
        for (int j = threadIdx.x; j < m; j += blockDim.x)
            sv[j] = in[(size_t)(j0 + j) * PF + 17];
        __syncthreads();
        if (i < n)
#pragma unroll 8
            for (int j = sub; j < m; j += P) {
                const float u = sv[j];
                rank += (u > v || (u == v && j0 + j < i)) ? 1 : 0;
            }
        __syncthreads();
    }
#pragma unroll
    for (int o = 1; o < P; o <<= 1)
        rank += __shfl_xor_sync(0xffffffffu, rank, o);
    return rank;
}

// The poses sorted, with their {tx, ty, tz, angle} keys, {tx, ty, tz, votes} and quaternions:
// kRankP lanes a pose (with one, 8083 poses took 88 us, 21 cycles a comparison).
constexpr int kRankP = 8, kRankBs = 128;
__global__ void __launch_bounds__(kRankBs) k_cluster_rank(ClArgs a) {
    smd::chain_enter(); // launched chained
    __shared__ float sv[kRankRun];
    const int        i    = (blockIdx.x * blockDim.x + threadIdx.x) / kRankP, sub = threadIdx.x % kRankP;
    const int        rank = rank_by_votes<kRankP>(a.poses, a.np, i, sv);
    if (i >= a.np)
        return;
    const float *P = a.poses + (size_t)i * PF;
    for (int e = sub; e < PF; e += kRankP)
        a.sorted[(size_t)rank * PF + e] = P[e];
    if (sub == 0) {
        a.key[rank] = make_float4(P[3], P[7], P[11], P[16]);
        a.tv[rank]  = make_float4(P[3], P[7], P[11], P[17]);
        a.qv[rank]  = make_float4(P[12], P[13], P[14], P[15]);
        a.clu[i]    = -1;
    }
}

// The model box's centre under an averaged pose, as a key of clusterPose2.
__device__ __forceinline__ float4 centre_key(const ClArgs &a, const float *P) {
    smi::Pose34 T;
    for (int e = 0; e < 12; e++)
        T.m[e] = P[e];
    float x, y, z;
    smi::pose_apply(T, a.cx, a.cy, a.cz, x, y, z);
    return make_float4(x, y, z, 0.f);
}

// The averaged clusters sorted likewise, with their centres' keys (lists too long for
// k_cluster_b's one CTA).
__global__ void __launch_bounds__(kRankBs) k_cluster_rank2(ClArgs a) {
    smd::chain_enter(); // launched chained
    __shared__ float sv[kRankRun];
    const int        nh = a.nh[0], per = blockDim.x / kRankP;
    if ((int)blockIdx.x * per >= nh)
        return; // (uniform)
    const int i    = blockIdx.x * per + threadIdx.x / kRankP, sub = threadIdx.x % kRankP;
    const int rank = rank_by_votes<kRankP>(a.avg, nh, i, sv);
    if (i >= nh)
        return;
    const float *P = a.avg + (size_t)i * PF;
    for (int e = sub; e < PF; e += kRankP)
        a.avgSorted[(size_t)rank * PF + e] = P[e];
    if (sub == 0)
        a.key[rank] = centre_key(a, P); // (the poses' keys are read no more)
}

// The compatibility word w of entry i of a chunk (keys k): bit b set when it is compatible with
// the chunk's earlier entry 32 w + b.
__device__ __forceinline__ uint32_t compat_word(const float4 *k, int i, int w, float sqThr, float angThr) {
    const float4 P = k[i];
    uint32_t     m = 0;
    if (w * 32 < i)
        for (int b = 0; b < 32; b++) {
            const int j = w * 32 + b;
            if (j < i && compat(P, k[j], sqThr, angThr))
                m |= 1u << b;
        }
    return m;
}

// The words of all chunks (blockIdx.y) over all CTAs: word w of entry i of a chunk of n at w n + i;
// of the poses, or (centres) of the averaged clusters.
__global__ void k_cluster_bits(ClArgs a, int centres) {
    smd::chain_enter(); // launched chained
    const int c0 = blockIdx.y * kClBs, n = min((centres ? a.nh[0] : a.np) - c0, kClBs);
    const int W = (n + 31) >> 5, idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (n > 0 && idx < n * W)
        a.bits[(size_t)blockIdx.y * 32 * kClBs + idx] =
            compat_word(a.key + c0, idx % n, idx / n, centres ? a.thr2 : a.sqThr,
                        centres ? __int_as_float(0x7f800000) : a.angThr);
}

struct ClMasks {
    uint32_t head[32], unk[32], newH[32], newM[32];
    int      pre[33];
};

// The greedy first fit of a chunk of n entries by a block of kClBs threads, a thread each, from the
// words `bits` (shared memory; as k_cluster_bits lays them out): `open` says whether the
// thread's entry takes part. Returns the number of the entry's head among the chunk's (heads in
// order; -1: takes no part); M.head has the heads' bits, M.pre[32] their number. By rounds: an
// undecided entry compatible with a head is a member; one whose compatible earlier entries are all
// decided members is a head. The smallest undecided entry is decided in every round, and
// each decision is the sequential one; a member's head is its lowest compatible one.
__device__ __forceinline__ int greedy_chunk(const uint32_t *bits, int n, bool open, ClMasks &M) {
    const int      tid = threadIdx.x, lane = tid & 31, own = tid >> 5, W = (n + 31) >> 5;
    const unsigned ob = __ballot_sync(0xffffffffu, open);
    if (lane == 0) {
        M.unk[own]  = ob;
        M.head[own] = M.newH[own] = M.newM[own] = 0u;
    }
    __syncthreads();
    bool undecided = open;
    for (;;) {
        if (undecided) {
            bool hitHead = false, hitUnk = false;
            for (int w = 0; w <= own && !hitHead; w++) {
                const uint32_t r = bits[(size_t)w * n + tid];
                hitHead          = (r & M.head[w]) != 0u;
                hitUnk           = hitUnk || (r & M.unk[w]) != 0u;
            }
            if (hitHead)
                atomicOr(&M.newM[own], 1u << lane);
            else if (!hitUnk)
                atomicOr(&M.newH[own], 1u << lane);
        }
        if (!__syncthreads_or(undecided))
            break;
        if (tid < W) {
            M.head[tid] |= M.newH[tid];
            M.unk[tid] &= ~(M.newH[tid] | M.newM[tid]);
            M.newH[tid] = M.newM[tid] = 0u;
        }
        __syncthreads();
        undecided = undecided && ((M.unk[own] >> lane) & 1u);
    }
    if (own == 0) {
        const int c    = lane < W ? __popc(M.head[lane]) : 0;
        const int incl = smd::warp_incl_scan(c);
        M.pre[lane]    = incl - c;
        if (lane == 31)
            M.pre[32] = incl;
    }
    __syncthreads();
    if (!open)
        return -1;
    const uint32_t hb = M.head[own];
    if ((hb >> lane) & 1u)
        return M.pre[own] + __popc(hb & ((1u << lane) - 1u));
    for (int w = 0; w <= own; w++) {
        const uint32_t r = bits[(size_t)w * n + tid] & M.head[w];
        if (r)
            return M.pre[w] + __popc(M.head[w] & ((r & (0u - r)) - 1u));
    }
    return -1; // (a decided entry is a head or has one: unreachable)
}

// clusterPose: the heads of the chunk at c0 and its poses' clusters.
__global__ void __launch_bounds__(kClBs) k_cluster_heads(ClArgs a, int c0) {
    smd::chain_enter(); // launched chained
    extern __shared__ uint32_t bits[];
    __shared__ ClMasks         M;
    const int                  tid = threadIdx.x, n = min(a.np - c0, kClBs), W = (n + 31) >> 5;
    const int                  nh = c0 ? a.nh[0] : 0;
    const uint32_t            *src = a.bits + (size_t)c0 * 32;
    for (int k = tid; k < n * W; k += kClBs)
        bits[k] = src[k];
    const bool open = tid < n && (c0 == 0 || a.clu[c0 + tid] < 0);
    const int  h    = greedy_chunk(bits, n, open, M); // (begins with a barrier)
    if (open) {
        a.clu[c0 + tid] = nh + h;
        if ((M.head[tid >> 5] >> (tid & 31)) & 1u)
            a.heads[nh + h] = c0 + tid;
    }
    if (tid == 0) {
        a.nh[0] = nh + M.pre[32];
        a.nh[1] = nh;
    }
}

// The poses from c1 on that fit none of the earlier heads: the first of the last chunk's that each
// fits.
__global__ void k_cluster_join(ClArgs a, int c1) {
    smd::chain_enter(); // launched chained
    __shared__ float4 sk[128];
    const int         i   = c1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int         nh1 = a.nh[0], nh0 = a.nh[1];
    bool              open = i < a.np && a.clu[i] < 0;
    const float4      P    = open ? a.key[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h0 = nh0; h0 < nh1; h0 += 128) {
        const int m = min(nh1 - h0, 128);
        if ((int)threadIdx.x < m)
            sk[threadIdx.x] = a.key[a.heads[h0 + threadIdx.x]];
        __syncthreads();
        for (int k = 0; k < m && open; k++)
            if (compat(P, sk[k], a.sqThr, a.angThr)) {
                a.clu[i] = h0 + k;
                open     = false;
            }
        if (!__syncthreads_or(open))
            return;
    }
}

// avgClusters: one block per cluster (grid-stride); the warp finds the members in pose
// order (cluster numbers read 256 poses ahead) and sums them in that order, one sum per lane:
// lane e < 10 the FP64 quaternion moment e, lanes 10..13 the FP32 translation and votes (the
// same additions in the same order as one thread summing all of them); then the Markley
// quaternion average in FP64.
__global__ void k_cluster_avg(ClArgs a) {
    smd::chain_enter(); // launched chained
    const int lane = threadIdx.x & 31;
    const int nh   = a.nh[0];
    // moment e of lane e: q[r] * q[s] over the upper triangle in row order
    int er = 0, es = 0;
    for (int r = 0, e = 0; r < 4; r++)
        for (int s2 = r; s2 < 4; s2++, e++)
            if (e == lane) {
                er = r;
                es = s2;
            }
    for (int h = blockIdx.x; h < nh; h += gridDim.x) {
        const int head = a.heads[h];
        double    Sd   = 0.0; // lane e < 10: moment e
        float     Pf   = 0.0f; // lanes 10..13: tx, ty, tz, votes
        int       cnt  = 0;
        for (int base = head; base < a.np; base += 32 * 8) {
            int cl[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int i = base + u * 32 + lane;
                cl[u]       = i < a.np ? a.clu[i] : -1;
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int      i   = base + u * 32 + lane;
                const bool     mem = cl[u] == h;
                const uint32_t m   = __ballot_sync(0xffffffffu, mem);
                if (!m)
                    continue;
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f), q4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (mem) {
                    t  = a.tv[i];
                    q4 = a.qv[i];
                }
                for (uint32_t r = m; r; r &= r - 1) {
                    const int   src = __ffs(r) - 1;
                    const float tv[4] = {__shfl_sync(0xffffffffu, t.x, src),
                                         __shfl_sync(0xffffffffu, t.y, src),
                                         __shfl_sync(0xffffffffu, t.z, src),
                                         __shfl_sync(0xffffffffu, t.w, src)};
                    const float qv[4] = {__shfl_sync(0xffffffffu, q4.x, src),
                                         __shfl_sync(0xffffffffu, q4.y, src),
                                         __shfl_sync(0xffffffffu, q4.z, src),
                                         __shfl_sync(0xffffffffu, q4.w, src)};
                    if (lane < 10)
                        Sd += (double)qv[er] * (double)qv[es];
                    else if (lane < 14)
                        Pf = Pf + tv[lane - 10];
                    cnt++;
                }
            }
        }
        double S[10];
#pragma unroll
        for (int e = 0; e < 10; e++)
            S[e] = __shfl_sync(0xffffffffu, Sd, e);
        const float px = __shfl_sync(0xffffffffu, Pf, 10), py = __shfl_sync(0xffffffffu, Pf, 11),
                    pz = __shfl_sync(0xffffffffu, Pf, 12), vs = __shfl_sync(0xffffffffu, Pf, 13);
        if (lane != 0)
            continue;
        double q[4], R[9];
        sml::quat_average_from_sum(S, cnt, q);
        sml::quat_to_mat(q, R);
        float *O = a.avg + (size_t)h * PF;
        for (int r = 0; r < 3; r++)
            for (int s = 0; s < 3; s++)
                O[r * 4 + s] = (float)R[r * 3 + s];
        const float fc = (float)cnt;
        O[3]           = smm::fdiv(px, fc);
        O[7]           = smm::fdiv(py, fc);
        O[11]          = smm::fdiv(pz, fc);
        for (int r = 0; r < 4; r++)
            O[12 + r] = (float)q[r];
        O[16] = sml::quat_angle(q);
        O[17] = vs;
    }
}

// sortPoses of the averaged clusters and clusterPose2 (overlap of the transformed model-box centres,
// util.cpp:522-551); with `ranked` the sort, the keys and the bits are there. One block, a chunk of kClBs clusters at a
// time: its clusters' first fit among the leaders so far, then greedy_chunk for the rest. A leader's
// vote sum keeps the order of the sequential walk. (A warp's walk over the clusters, 32
// leaders a step, took 22 us for 168.)
__global__ void __launch_bounds__(kClBs) k_cluster_b(ClArgs a, int ranked) {
    smd::chain_enter(); // launched chained
    extern __shared__ uint32_t bits[];
    __shared__ ClMasks         M;
    __shared__ float4          sKey[kClBs];
    __shared__ float           sVote[kRankRun];
    __shared__ int             sClu[kClBs];
    const int                  tid = threadIdx.x;
    const int                  nh  = a.nh[0];
    if (!ranked) { // (nh <= kClBs)
        const int rank = rank_by_votes<1>(a.avg, nh, tid, sVote);
        if (tid < nh)
            for (int e = 0; e < PF; e++)
                a.avgSorted[(size_t)rank * PF + e] = a.avg[(size_t)tid * PF + e];
        __syncthreads();
    }
    int nl = 0;
    for (int c0 = 0; c0 < nh; c0 += kClBs) {
        const int n = min(nh - c0, kClBs), W = (n + 31) >> 5;
        int       lead = -1;
        if (tid < n) {
            const float *P = a.avgSorted + (size_t)(c0 + tid) * PF;
            const float4 k = ranked ? a.key[c0 + tid] : centre_key(a, P);
            sKey[tid]      = k;
            sVote[tid]     = P[17];
            for (int l = 0; l < nl && lead < 0; l++)
                if (compat(k, a.key[a.heads[l]], a.thr2, __int_as_float(0x7f800000)))
                    lead = l;
        }
        __syncthreads();
        for (int k = tid; k < n * W; k += kClBs)
            bits[k] = ranked ? a.bits[(size_t)c0 * 32 + k]
                             : compat_word(sKey, k % n, k / n, a.thr2, __int_as_float(0x7f800000));
        const bool open = tid < n && lead < 0;
        const int  h    = greedy_chunk(bits, n, open, M); // (begins with a barrier)
        if (open) {
            lead = nl + h;
            if ((M.head[tid >> 5] >> (tid & 31)) & 1u)
                a.heads[lead] = c0 + tid;
        }
        sClu[tid]      = lead;
        const int nl1 = nl + M.pre[32];
        __syncthreads();
        for (int l = tid; l < nl1; l += kClBs) {
            bool  first = l >= nl; // the leader itself comes first
            float sum   = first ? 0.0f : a.sum[l];
            for (int k = 0; k < n; k++)
                if (sClu[k] == l) {
                    sum   = first ? sVote[k] : sum + sVote[k];
                    first = false;
                }
            a.sum[l] = sum;
        }
        nl = nl1;
        __syncthreads();
    }
    for (int idx = tid; idx < nl * PF; idx += kClBs) {
        const int l = idx / PF, e = idx - l * PF;
        a.out[idx]  = e == 17 ? a.sum[l] : a.avgSorted[(size_t)a.heads[l] * PF + e];
    }
    if (tid == 0)
        *a.outCount = nl;
}

// Smallest float v >= 0 with sqrtf(v) >= t (IEEE square root is correctly rounded and
// monotone, so sqrtf(v) < t <=> v < this bound, NaN included).
float sqrt_lt_bound(float t) {
    if (!(t > 0.0f))
        return 0.0f;
    uint32_t lo = 0, hi = 0x7f800000u; // +0 .. +inf
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        float          v;
        memcpy(&v, &mid, 4);
        if (std::sqrt(v) >= t)
            hi = mid;
        else
            lo = mid + 1;
    }
    float r;
    memcpy(&r, &lo, 4);
    return r;
}

} // namespace

int cluster(Ctx &c, const float *poses, int np, float distThr, float angThr, const float center[3],
            float maxOverlap, float *outCands, const std::string &tag) {
    if (np <= 0)
        return 0;
    ClArgs a;
    a.poses     = poses;
    a.np        = np;
    a.sqThr     = sqrt_lt_bound(distThr);
    a.angThr    = angThr;
    a.cx        = center[0];
    a.cy        = center[1];
    a.cz        = center[2];
    a.thr2      = maxOverlap * maxOverlap;
    a.sorted    = c.arena.get<float>(tag + ".sorted", (size_t)np * PF);
    a.avg       = c.arena.get<float>(tag + ".avg", (size_t)np * PF);
    a.avgSorted = c.arena.get<float>(tag + ".avgs", (size_t)np * PF);
    a.out       = outCands;
    a.outCount  = c.arena.get<int>(tag + ".count", 1);
    a.key       = c.arena.get<float4>(tag + ".key", np);
    a.sum       = c.arena.get<float>(tag + ".sum", np);
    a.tv        = c.arena.get<float4>(tag + ".tv", np);
    a.qv        = c.arena.get<float4>(tag + ".qv", np);
    int *ints   = c.arena.get<int>(tag + ".ints", (size_t)np * 2 + 2);
    a.clu       = ints;
    a.heads     = ints + np;
    a.nh        = ints + 2 * (size_t)np;
    const int chunks = nblocks(np, kClBs), most = std::min(np, kClBs);
    a.bits = c.arena.get<uint32_t>(tag + ".bits", (size_t)chunks * 32 * kClBs);
    const int    words = most * ((most + 31) / 32);
    const size_t smem  = (size_t)words * 4;
    if (smem > allow_dynamic_smem((const void *)k_cluster_heads, c.device) ||
        smem > allow_dynamic_smem((const void *)k_cluster_b, c.device))
        throw Error(SM_ERR_CAPACITY, "shared-memory request above the device limit");
    const int  per  = kRankBs / kRankP;
    const dim3 bits = dim3(nblocks(words, 256), chunks);
    launch_chained(c, k_cluster_rank, nblocks(np, per), kRankBs, 0, a);
    launch_chained(c, k_cluster_bits, bits, 256, 0, a, 0);
    for (int c0 = 0; c0 < np; c0 += kClBs) {
        launch_chained(c, k_cluster_heads, 1, kClBs, smem, a, c0);
        if (c0 + kClBs < np)
            launch_chained(c, k_cluster_join, nblocks(np - c0 - kClBs, 128), 128, 0, a, c0 + kClBs);
    }
    launch_chained(c, k_cluster_avg, std::min(np, 152 * 8), 32, 0, a);
    const int ranked = chunks > 1 ? 1 : 0;
    if (ranked) {
        launch_chained(c, k_cluster_rank2, nblocks(np, per), kRankBs, 0, a);
        launch_chained(c, k_cluster_bits, bits, 256, 0, a, 1);
    }
    launch_chained(c, k_cluster_b, 1, kClBs, smem, a, ranked);
    SM_CUDA(cudaMemcpyAsync(c.hostCounts, a.outCount, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    return c.hostCounts[0];
}

} // namespace sm
