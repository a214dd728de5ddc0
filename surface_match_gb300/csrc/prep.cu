// prep.cu - point preparation, scans and compaction, uniform grids, greedy sampling and
// normal estimation of the matching path.
//
// Reference counterparts: removeNan / computeBoundingBox (util.cpp:86-105, 178-207), the
// k-d tree (kdtree/kdtree.h) replaced by uniform grids, samplePointCloud (util.cpp:107-139),
// estimateNormal / computeNormal (util.cpp:234-334), normalizeNormal (util.cpp:163-176).
#include <atomic>
#include <climits>
#include <cmath>

#include "sm_icp.h"
#include "sm_linalg.h"
#include "sm_scan.cuh"
#include "sm_stages.h"

namespace sm {
using namespace smd;

namespace {


struct GridParams {
    float org[3], g;
    int   dim[3];
};

GridParams grid_params(const Box &b, float g, int dim[3]) {
    GridParams p;
    for (int a = 0; a < 3; a++) {
        p.org[a] = b.mn[a];
        p.dim[a] = dim[a];
    }
    p.g = g;
    return p;
}

__device__ __forceinline__ float4 nan4() {
    const float q = __int_as_float(0x7fc00000);
    return make_float4(q, q, q, 0.0f);
}

__device__ __forceinline__ bool finite3(float x, float y, float z) {
    return isfinite(x) && isfinite(y) && isfinite(z);
}

// ---------------------------------------------------------------------------------------
// Three floats of each of the four points 4 g .. 4 g + 3 (below n): three 16-byte loads where the
// array is aligned to them, else one by one.
__device__ __forceinline__ void load_points4(const float *__restrict__ a, int g, int n, float v[12]) {
    const size_t o = 12 * (size_t)g;
    if (((uintptr_t)a & 15) == 0 && 4 * g + 3 < n) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float4 q = reinterpret_cast<const float4 *>(a + o)[k];
            v[4 * k]       = q.x;
            v[4 * k + 1]   = q.y;
            v[4 * k + 2]   = q.z;
            v[4 * k + 3]   = q.w;
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 12; k++)
        v[k] = 4 * g + k / 3 < n ? a[o + k] : 0.0f;
}

// A thread takes four points (0.92 M points: 27.5 us with a point per thread, its three floats
// loaded one by one, and 2432 CTAs adding to the box).
__global__ void __launch_bounds__(256)
    k_prep(const float *__restrict__ xyz, const float *__restrict__ nin, int n,
           float4 *__restrict__ pos, float4 *__restrict__ nrm, int *__restrict__ valid,
           int *__restrict__ bbox, int *__restrict__ nvalid) {
    __shared__ int smn[3], smx[3], scnt;
    if (threadIdx.x < 3) {
        smn[threadIdx.x] = INT_MAX;
        smx[threadIdx.x] = INT_MIN;
    }
    if (threadIdx.x == 0)
        scnt = 0;
    __syncthreads();
    int lmn[3] = {INT_MAX, INT_MAX, INT_MAX}, lmx[3] = {INT_MIN, INT_MIN, INT_MIN}, lc = 0;
    const int groups = (n + 3) / 4;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += gridDim.x * blockDim.x) {
        float p[12], q[12];
        load_points4(xyz, g, n, p);
        if (nin)
            load_points4(nin, g, n, q);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int i = 4 * g + k;
            if (i >= n)
                break;
            const float x = p[3 * k], y = p[3 * k + 1], z = p[3 * k + 2];
            bool        ok = finite3(x, y, z);
            float4      nn = nan4();
            if (nin) {
                float a = q[3 * k], b = q[3 * k + 1], c = q[3 * k + 2];
                ok      = ok && finite3(a, b, c);
                const float sq = a * a + (b * b + c * c);
                if (sq > 0.0f) {
                    const float s = smm::fsqrt(sq);
                    a             = smm::fdiv(a, s);
                    b             = smm::fdiv(b, s);
                    c             = smm::fdiv(c, s);
                }
                nn = make_float4(a, b, c, 0.0f);
            }
            pos[i]   = make_float4(x, y, z, 0.0f);
            nrm[i]   = nn;
            valid[i] = ok ? 1 : 0;
            if (ok) {
                const int o[3] = {f2ord(x), f2ord(y), f2ord(z)};
                for (int a = 0; a < 3; a++) {
                    lmn[a] = min(lmn[a], o[a]);
                    lmx[a] = max(lmx[a], o[a]);
                }
                lc++;
            }
        }
    }
    for (int a = 0; a < 3; a++) {
        lmn[a] = __reduce_min_sync(0xffffffffu, lmn[a]);
        lmx[a] = __reduce_max_sync(0xffffffffu, lmx[a]);
    }
    lc = __reduce_add_sync(0xffffffffu, lc);
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; a++) {
            atomicMin(&smn[a], lmn[a]);
            atomicMax(&smx[a], lmx[a]);
        }
        atomicAdd(&scnt, lc);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int a = 0; a < 3; a++) {
            atomicMin(&bbox[a], smn[a]);
            atomicMax(&bbox[3 + a], smx[a]);
        }
        atomicAdd(nvalid, scnt);
    }
}

__global__ void k_init_bbox(int *bbox, int *nvalid) {
    if (threadIdx.x < 3) {
        bbox[threadIdx.x]     = INT_MAX;
        bbox[3 + threadIdx.x] = INT_MIN;
    }
    if (threadIdx.x == 0)
        *nvalid = 0;
}

// Up to four buffers of 32-bit words, each set to its value, in one chained launch (a
// cudaMemsetAsync per buffer would be one stream operation each and break the launch chain).
struct FillSet {
    uint32_t *p[4];
    long long n[4]; // words
    uint32_t  v[4];
    int       k = 0;
    void add(void *ptr, size_t bytes, uint32_t value) {
        if (k == 4)
            throw Error(SM_ERR_RUNTIME, "buffer clear: more than four buffers in one launch");
        p[k]   = (uint32_t *)ptr;
        n[k]   = (long long)(bytes / 4);
        v[k++] = value;
    }
};

__global__ void k_fill(FillSet f) {
    chain_enter(); // launched chained
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long st = (long long)gridDim.x * blockDim.x;
    for (int s = 0; s < f.k; s++) {
        uint32_t       *p = f.p[s];
        const long long n = f.n[s];
        const uint32_t  v = f.v[s];
        // 16-byte stores over an aligned buffer's body, 4-byte stores for the rest
        const long long n4 = ((uintptr_t)p & 15) == 0 ? n / 4 : 0;
        uint4          *q  = reinterpret_cast<uint4 *>(p);
        for (long long i = t0; i < n4; i += st)
            q[i] = make_uint4(v, v, v, v);
        for (long long i = n4 * 4 + t0; i < n; i += st)
            p[i] = v;
    }
}

static void fill(Ctx &c, const FillSet &f) {
    long long words = 0;
    for (int s = 0; s < f.k; s++)
        words += f.n[s];
    if (words == 0)
        return;
    int nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    const int g = (int)std::min<long long>(nblocks((words + 3) / 4, 256), 8LL * std::max(nsm, 1));
    launch_chained(c, k_fill, g, 256, 0, f);
}

// ---------------------------------------------------------------------------------------
__global__ void k_iota(int *__restrict__ out, int n) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = i;
}

// ---------------------------------------------------------------------------------------
// Sampler cells by how many points they hold: up to kSpSmall a group of eight lanes takes the
// cell, up to kSpHeavy a warp, above a CTA. (A warp for every cell up to 128 points left most
// lanes idle at the refinement's step, whose cells hold six points: 20 us a phase of 0.92 M
// points' 154,000 cells, 16 us now.) Where a phase has no more small cells than the launch has
// warps, a warp takes each: 6.5 us a phase of the 13,000-point scene against 10.5 us by groups.
constexpr int kSpSmall = 32;
constexpr int kSpHeavy = 128;
constexpr int kSpBs    = 1024; // threads of the table passes: few CTAs add to the phase counters

// The sampler's cells keep their side just above the step whatever the scene's extent
// (the work per point is then bounded by the packing of kept points, not by how coarse a
// capped grid would have to be). Their table is dense (slot = cell key) when the cell box is
// small against the points (see sample_points), else hashed: keys[slot] holds the cell key
// (open addressing, ~0 = empty), so only occupied cells are stored. cnt[slot] = the cell's
// points (0: empty); info[slot] = {first, kept}: a cell's points are contiguous in pts from
// `first`, its kept points' positions in keptPos from there too, `kept` of them so far. info is
// written for occupied cells only.
struct ThinView {
    int                       dim[3];
    const unsigned long long *keys; // nullptr: dense table
    uint32_t                  mask;
    const int                *cnt;
    int2                     *info;
    const float4             *pts;
    float4                   *keptPos;
    int                       m; // points
    // {first, kept} of the K cells with keys key[] where want[] is set, {0, 0} for a cell
    // without points: the loads of all K in flight together
    template <int K>
    __device__ __forceinline__ void find(const unsigned long long (&key)[K], const bool (&want)[K],
                                         int2 (&v)[K]) const {
        if (!keys) {
            int n[K];
#pragma unroll
            for (int r = 0; r < K; r++) {
                const unsigned long long t = want[r] ? key[r] : 0ull;
                v[r]                       = info[t];
                n[r]                       = cnt[t];
            }
#pragma unroll
            for (int r = 0; r < K; r++)
                if (!want[r] || n[r] == 0)
                    v[r] = make_int2(0, 0);
            return;
        }
        uint32_t           h[K];
        unsigned long long k[K];
#pragma unroll
        for (int r = 0; r < K; r++) {
            h[r] = (uint32_t)smm::mix64(key[r]) & mask;
            k[r] = want[r] ? keys[h[r]] : ~0ull;
        }
#pragma unroll
        for (int r = 0; r < K; r++)
            while (k[r] != key[r] && k[r] != ~0ull) { // (a free slot ends every probe)
                h[r] = (h[r] + 1) & mask;
                k[r] = keys[h[r]];
            }
#pragma unroll
        for (int r = 0; r < K; r++)
            v[r] = k[r] != ~0ull ? info[h[r]] : make_int2(0, 0);
    }
};

__device__ __forceinline__ unsigned long long cell_key(int x, int y, int z, int dim0, int dim1) {
    return ((unsigned long long)z * (unsigned)dim1 + (unsigned)y) * (unsigned)dim0 + (unsigned)x;
}

__device__ __forceinline__ void cell_coords(unsigned long long key, int dim0, int dim1, int c[3]) {
    if (key >> 32) {
        c[0] = (int)(key % (unsigned)dim0);
        c[1] = (int)((key / (unsigned)dim0) % (unsigned)dim1);
        c[2] = (int)(key / ((unsigned long long)dim0 * (unsigned)dim1));
    } else {
        const unsigned k = (unsigned)key, r = k / (unsigned)dim0;
        c[0] = (int)(k - r * (unsigned)dim0);
        c[2] = (int)(r / (unsigned)dim1);
        c[1] = (int)(r - (unsigned)c[2] * (unsigned)dim1);
    }
}

// The phases' counters: occupied cells, then the cells listed so far per class, then the heavy
// cells taken.
enum { kPhCells = 0, kPhSmall = 8, kPhMedium = 16, kPhHeavy = 24, kPhTaken = 32, kPhNext = 40, kPhWords = 41 };

// Counting pass: the point's cell enters the table and the point takes its place within the
// cell (place = {slot, place}); the point that opens a cell also counts the cell in its phase,
// in shared memory first (a global counter per phase took one update per cell: 67 us of the
// refinement's sampling). A hashed table has at least twice as many slots as points, so every
// cell finds one; a dense one (keys == nullptr) files the cell under its key.
__global__ void __launch_bounds__(kSpBs)
    k_thin_insert(const float4 *__restrict__ pos, const int *__restrict__ ids, int m, GridParams gp,
                  unsigned long long *__restrict__ keys, uint32_t mask, int2 *__restrict__ place,
                  int *__restrict__ cnt, int *__restrict__ ph) {
    chain_enter(); // launched chained
    __shared__ int h[8];
    if (threadIdx.x < 8)
        h[threadIdx.x] = 0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < m) {
        const float4             p   = pos[ids[i]];
        const int                cx  = smg::coord(p.x, gp.org[0], gp.g, gp.dim[0]);
        const int                cy  = smg::coord(p.y, gp.org[1], gp.g, gp.dim[1]);
        const int                cz  = smg::coord(p.z, gp.org[2], gp.g, gp.dim[2]);
        const unsigned long long key = cell_key(cx, cy, cz, gp.dim[0], gp.dim[1]);
        uint32_t                 t   = keys ? (uint32_t)smm::mix64(key) & mask : (uint32_t)key;
        for (uint32_t q = 0; q <= mask; q++) {
            const unsigned long long prev = keys ? atomicCAS(&keys[t], ~0ull, key) : key;
            if (prev == ~0ull || prev == key) {
                const int k = atomicAdd(&cnt[t], 1);
                place[i]    = make_int2((int)t, k);
                if (k == 0)
                    atomicAdd(&h[smg::phase_of(cx, cy, cz)], 1);
                break;
            }
            t = (t + 1) & mask;
        }
    }
    __syncthreads();
    if (threadIdx.x < 8 && h[threadIdx.x])
        atomicAdd(&ph[kPhCells + threadIdx.x], h[threadIdx.x]);
}

// First list place of phase p.
__device__ __forceinline__ int phase_off(const int *__restrict__ ph, int p) {
    int o = 0;
#pragma unroll
    for (int q = 0; q < 8; q++)
        o += q < p ? ph[kPhCells + q] : 0;
    return o;
}

// Occupied cells take their points' range from a counter (a CTA's at once; the cells' order does
// not matter) and enter their phase's lists (any order: cells of one phase do not interact):
// entries {slot, first, key}, small cells in one list, in the other medium ones from the front
// and heavy ones from the back. Four slots a thread.
__global__ void __launch_bounds__(kSpBs)
    k_thin_cells(ThinView G, uint32_t T, int *__restrict__ ph, int4 *__restrict__ small,
                 int4 *__restrict__ large) {
    chain_enter(); // launched chained
    __shared__ int sh[33], h[24], base[24], sBase;
    if (threadIdx.x < 24)
        h[threadIdx.x] = 0;
    const uint32_t t0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x);
    int            n[4], s = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        n[j] = t0 + j < T ? G.cnt[t0 + j] : 0;
        s += n[j];
    }
    int       tot;
    const int ex = block_excl_scan(s, sh, &tot); // (its barriers cover h)
    if (tot == 0)
        return; // (uniform)
    if (threadIdx.x == 0)
        sBase = atomicAdd(&ph[kPhNext], tot);
    int                cls[4], at[4];
    unsigned long long key[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        cls[j] = -1;
        if (n[j] > 0) {
            int c[3];
            key[j] = G.keys ? G.keys[t0 + j] : (unsigned long long)(t0 + j);
            cell_coords(key[j], G.dim[0], G.dim[1], c);
            cls[j] = smg::phase_of(c[0], c[1], c[2]) +
                     (n[j] <= kSpSmall ? 0 : n[j] <= kSpHeavy ? 8 : 16);
            at[j] = atomicAdd(&h[cls[j]], 1);
        }
    }
    __syncthreads();
    if (threadIdx.x < 24) {
        const int p   = threadIdx.x & 7;
        const int off = phase_off(ph, p);
        const int b   = h[threadIdx.x] ? atomicAdd(&ph[kPhSmall + threadIdx.x], h[threadIdx.x]) : 0;
        base[threadIdx.x] = threadIdx.x < 16 ? off + b : off + ph[kPhCells + p] - 1 - b;
    }
    __syncthreads();
    int first = sBase + ex;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (cls[j] < 0)
            continue;
        const int4 e = make_int4((int)(t0 + j), first, (int)(uint32_t)key[j],
                                 (int)(uint32_t)(key[j] >> 32));
        G.info[t0 + j] = make_int2(first, 0);
        if (cls[j] < 8)
            small[base[cls[j]] + at[j]] = e;
        else
            large[base[cls[j]] + (cls[j] < 16 ? at[j] : -at[j])] = e;
        first += n[j];
    }
}

// Placing pass: the point's position (its place i in the ascending id list in w: list order is
// index order) at its place in the cell; its kept flag starts clear.
__global__ void k_thin_scatter(const float4 *__restrict__ pos, const int *__restrict__ ids, int m,
                               const int2 *__restrict__ place, const int2 *__restrict__ info,
                               float4 *__restrict__ pts, int *__restrict__ keptFlag) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const int2   at = place[i];
    const float4 p  = pos[ids[i]];
    pts[info[at.x].x + at.y] = make_float4(p.x, p.y, p.z, __int_as_float(i));
    keptFlag[i]              = 0;
}

// ---------------------------------------------------------------------------------------
constexpr int kSpWarps  = 8;   // warps per CTA of the phase kernel
constexpr int kSpReg    = kSpHeavy / 32; // medium cell: points per lane, held in registers
constexpr int kSpHStage = 448; // heavy cell: neighbours' kept points staged
constexpr int kSpStage  = 128; // medium cell: neighbours' kept points staged per warp
constexpr int kSpGStage = 32;  // small cell: the same per group of eight lanes
constexpr int kSpBuf    = kSpWarps * kSpStage > kSpHStage ? kSpWarps * kSpStage : kSpHStage;
static_assert(kSpSmall == 32 && kSpStage == 4 * kSpGStage, "a small cell is four points a lane");

// Neighbours l, l + 32 / K, ... < 26 of cell c (the centre left out; none unless live): {first,
// kept}; cells of later phases have kept nothing yet, empty cells give {0, 0}.
template <int K>
__device__ __forceinline__ void sp_neighbours(const ThinView &G, const int c[3], int l, bool live,
                                              int2 (&nb)[K]) {
    unsigned long long key[K];
    bool               want[K];
#pragma unroll
    for (int r = 0; r < K; r++) {
        const int i = l + r * (32 / K), o = i < 13 ? i : i + 1;
        const int x = c[0] + o % 3 - 1, y = c[1] + (o / 3) % 3 - 1, z = c[2] + o / 9 - 1;
        want[r] = live && i < 26 && x >= 0 && y >= 0 && z >= 0 && x < G.dim[0] && y < G.dim[1] &&
                  z < G.dim[2];
        key[r] = cell_key(x, y, z, G.dim[0], G.dim[1]);
    }
    G.find(key, want, nb);
}

__device__ __forceinline__ unsigned long long entry_key(const int4 &e) {
    return ((unsigned long long)(uint32_t)e.w << 32) | (uint32_t)e.z;
}

__device__ __forceinline__ bool sp_near(const float4 &o, const float4 &q, float r2) {
    return smm::dist2(o.x, o.y, o.z, q.x, q.y, q.z) < r2;
}

// The sequential greedy visits a cell's points by ascending index and keeps a point unless a
// kept point lies within the step; the kept points of the 26 neighbour cells (earlier phases)
// are fixed, so the cell first drops every point within the step of one of them (order-free),
// then repeats "keep the smallest surviving index, drop the survivors within the step of it" -
// the same kept set as the sequential visit, at (kept points x cell size / threads) work and
// without sorting. Points are named by their place in the ascending id list (same order as the
// index), and keptFlag is over those places.

// A heavy cell by the whole CTA: neighbours' kept points staged in shared memory when they fit,
// survivors flagged in alive.
__device__ void sp_heavy(const ThinView &G, const int4 &e, float r2, int *__restrict__ keptFlag,
                         int *__restrict__ alive, float4 *stage) {
    __shared__ int    sFirst[26], sPre[27], sMin[kSpWarps];
    __shared__ float4 sKeep;
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int s = e.y, n = G.cnt[e.x];
    alive += s;
    if (wl == 0) {
        int c[3];
        cell_coords(entry_key(e), G.dim[0], G.dim[1], c);
        int2 nb[1];
        sp_neighbours(G, c, lane, true, nb);
        const int incl = warp_incl_scan(nb[0].y);
        if (lane < 26) {
            sFirst[lane] = nb[0].x;
            sPre[lane]   = incl - nb[0].y;
        }
        if (lane == 31)
            sPre[26] = incl;
    }
    __syncthreads();
    const int  NK      = sPre[26];
    const bool stageNb = NK <= kSpHStage;
    if (stageNb) {
        for (int t = tid; t < NK; t += kSpWarps * 32) {
            int j = 0;
            while (sPre[j + 1] <= t)
                j++;
            stage[t] = G.keptPos[sFirst[j] + (t - sPre[j])];
        }
    }
    __syncthreads();
    for (int i = tid; i < n; i += kSpWarps * 32) {
        const float4 q  = G.pts[s + i];
        bool         ok = true;
        if (stageNb) {
            for (int k = 0; k < NK && ok; k++)
                ok = !sp_near(stage[k], q, r2);
        } else {
            for (int j = 0; j < 26 && ok; j++)
                for (int k = 0; k < sPre[j + 1] - sPre[j] && ok; k++)
                    ok = !sp_near(G.keptPos[sFirst[j] + k], q, r2);
        }
        alive[i] = ok ? 1 : 0;
    }
    __syncthreads();
    int nk = 0;
    for (;;) {
        int    myMin = INT_MAX;
        float4 myP   = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = tid; i < n; i += kSpWarps * 32)
            if (alive[i]) {
                const float4 q  = G.pts[s + i];
                const int    id = __float_as_int(q.w);
                if (id < myMin) {
                    myMin = id;
                    myP   = q;
                }
            }
        const int wm = __reduce_min_sync(0xffffffffu, myMin);
        if (lane == 0)
            sMin[wl] = wm;
        __syncthreads();
        int m = INT_MAX;
        for (int k = 0; k < kSpWarps; k++)
            m = min(m, sMin[k]);
        if (m == INT_MAX)
            break; // (uniform: every thread read the same minima)
        if (myMin == m)
            sKeep = myP; // the unique holder
        __syncthreads();
        const float4 kp = sKeep;
        if (tid == 0) {
            keptFlag[m]          = 1;
            G.keptPos[s + nk]    = kp;
        }
        nk++;
        for (int i = tid; i < n; i += kSpWarps * 32) {
            if (!alive[i])
                continue;
            const float4 q = G.pts[s + i];
            if (__float_as_int(q.w) == m || sp_near(kp, q, r2))
                alive[i] = 0;
        }
        __syncthreads(); // drops done and sMin / sKeep read before the next round
    }
    if (tid == 0)
        G.info[e.x].y = nk;
    __syncthreads(); // the buffers are reused by the next cell
}

// A medium cell by a warp: its points in registers (kSpReg per lane), the neighbours' kept points
// staged in shared memory by the whole warp at once when they fit, else read one by one (a
// broadcast each).
__device__ __forceinline__ void sp_medium(const ThinView &G, const int4 &e, float r2,
                                          int *__restrict__ keptFlag, float4 *stage) {
    const int lane = threadIdx.x & 31;
    const int s = e.y, n = G.cnt[e.x]; // n <= kSpHeavy
    float4    q[kSpReg];
#pragma unroll
    for (int j = 0; j < kSpReg; j++) // (whatever follows the cell's points is masked below)
        q[j] = G.pts[min(s + lane + 32 * j, G.m - 1)];
    int c[3];
    cell_coords(entry_key(e), G.dim[0], G.dim[1], c);
    int2 nb1[1];
    sp_neighbours(G, c, lane, true, nb1);
    const int2 nb    = nb1[0];
    unsigned   alive = 0u; // bit j: point lane + 32 j is still a candidate
#pragma unroll
    for (int j = 0; j < kSpReg; j++)
        alive |= (lane + 32 * j < n ? 1u : 0u) << j;
    auto drop = [&](const float4 &o) {
#pragma unroll
        for (int j = 0; j < kSpReg; j++)
            if (sp_near(o, q[j], r2))
                alive &= ~(1u << j);
    };
    const int incl = warp_incl_scan(nb.y);
    const int excl = incl - nb.y;
    const int NK   = __shfl_sync(0xffffffffu, incl, 31);
    if (NK <= kSpStage) {
        for (int base = 0; base < NK; base += 32) {
            const int t  = base + lane;
            int       lo = 0; // the neighbour holding kept point t: last with excl <= t
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const int mid = lo + step;
                const int ev  = __shfl_sync(0xffffffffu, excl, mid & 31);
                if (mid < 26 && ev <= t)
                    lo = mid;
            }
            const int fj = __shfl_sync(0xffffffffu, nb.x, lo);
            const int ej = __shfl_sync(0xffffffffu, excl, lo);
            if (t < NK)
                stage[t] = G.keptPos[fj + (t - ej)];
        }
        __syncwarp();
        for (int k = 0; k < NK; k++)
            drop(stage[k]);
        __syncwarp(); // the slice is refilled by the warp's next cell
    } else {
        for (int j = 0; j < 26; j++) {
            const int fj = __shfl_sync(0xffffffffu, nb.x, j);
            const int cj = __shfl_sync(0xffffffffu, nb.y, j);
            for (int k = 0; k < cj; k++)
                drop(G.keptPos[fj + k]);
        }
    }
    // keep the smallest surviving index, drop the survivors within the step, repeat; the lane
    // that holds the kept point hands its position to the warp
    int nk = 0;
    for (;;) {
        int    myMin = INT_MAX;
        float4 myP   = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < kSpReg; j++) {
            const int id = __float_as_int(q[j].w);
            if (((alive >> j) & 1u) && id < myMin) {
                myMin = id;
                myP   = q[j];
            }
        }
        const int m = __reduce_min_sync(0xffffffffu, myMin);
        if (m == INT_MAX)
            break;
        const int    src = __ffs(__ballot_sync(0xffffffffu, myMin == m)) - 1;
        const float4 kp  = make_float4(__shfl_sync(0xffffffffu, myP.x, src),
                                       __shfl_sync(0xffffffffu, myP.y, src),
                                       __shfl_sync(0xffffffffu, myP.z, src), 0.0f);
        if (lane == 0) {
            keptFlag[m]       = 1;
            G.keptPos[s + nk] = kp;
        }
        nk++;
#pragma unroll
        for (int j = 0; j < kSpReg; j++)
            if (__float_as_int(q[j].w) == m || sp_near(kp, q[j], r2))
                alive &= ~(1u << j);
    }
    if (lane == 0)
        G.info[e.x].y = nk;
}

// Four small cells by a warp, eight lanes each (live: this group has one): four points a lane, and
// up to four neighbours a lane, whose kept points the lanes stage in parallel.
__device__ __forceinline__ void sp_small(const ThinView &G, const int4 &e, bool live, float r2,
                                         int *__restrict__ keptFlag, float4 *stage) {
    const int lane = threadIdx.x & 31, gl = lane & 7, g0 = lane & 24;
    const int s    = e.y;
    float4    q[4];
    int2      nb[4];
    const int n = live ? G.cnt[e.x] : 0;
#pragma unroll
    for (int j = 0; j < 4; j++)
        q[j] = G.pts[min(s + gl + 8 * j, G.m - 1)];
    int c[3];
    cell_coords(entry_key(e), G.dim[0], G.dim[1], c);
    sp_neighbours(G, c, gl, live, nb);
    const int mine = nb[0].y + nb[1].y + nb[2].y + nb[3].y;
    unsigned alive = 0u; // bit j: point gl + 8 j is still a candidate
#pragma unroll
    for (int j = 0; j < 4; j++)
        alive |= (gl + 8 * j < n ? 1u : 0u) << j;
    auto drop = [&](const float4 &o) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (sp_near(o, q[j], r2))
                alive &= ~(1u << j);
    };
    int incl = mine; // inclusive prefix over the group
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o, 8);
        if (gl >= o)
            incl += t;
    }
    const int NK   = __shfl_sync(0xffffffffu, incl, 7, 8);
    const int most = __reduce_max_sync(0xffffffffu, NK);
    if (most <= kSpGStage) {
        float4 kp[4]; // most neighbours have kept one point: these loads in flight together
#pragma unroll
        for (int r = 0; r < 4; r++)
            if (nb[r].y > 0)
                kp[r] = G.keptPos[nb[r].x];
        int at = incl - mine;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            if (nb[r].y > 0)
                stage[at] = kp[r];
            for (int k = 1; k < nb[r].y; k++)
                stage[at + k] = G.keptPos[nb[r].x + k];
            at += nb[r].y;
        }
        __syncwarp();
        for (int k = 0; k < most; k++)
            if (k < NK)
                drop(stage[k]);
        __syncwarp(); // the slice is refilled by the group's next cell
    } else {
#pragma unroll
        for (int r = 0; r < 4; r++)
            for (int l = 0; l < 8; l++) {
                const int f  = __shfl_sync(0xffffffffu, nb[r].x, l, 8);
                const int cj = __shfl_sync(0xffffffffu, nb[r].y, l, 8);
                for (int k = 0; k < cj; k++)
                    drop(G.keptPos[f + k]);
            }
    }
    int nk = 0;
    for (;;) {
        int    myMin = INT_MAX;
        float4 myP   = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int id = __float_as_int(q[j].w);
            if (((alive >> j) & 1u) && id < myMin) {
                myMin = id;
                myP   = q[j];
            }
        }
        int m = myMin;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
            m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (__all_sync(0xffffffffu, m == INT_MAX))
            break; // no group has a survivor
        const unsigned who = __ballot_sync(0xffffffffu, myMin == m && m != INT_MAX) & (0xffu << g0);
        const int      src = who ? __ffs(who) - 1 : lane;
        const float4   kp  = make_float4(__shfl_sync(0xffffffffu, myP.x, src),
                                         __shfl_sync(0xffffffffu, myP.y, src),
                                         __shfl_sync(0xffffffffu, myP.z, src), 0.0f);
        if (m == INT_MAX)
            continue; // (the group waits for the others)
        if (gl == 0) {
            keptFlag[m]       = 1;
            G.keptPos[s + nk] = kp;
        }
        nk++;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (__float_as_int(q[j].w) == m || sp_near(kp, q[j], r2))
                alive &= ~(1u << j);
    }
    if (live && gl == 0)
        G.info[e.x].y = nk;
}

// The cells of the current phase: heavy ones first, one at a time from a counter, then medium and
// small ones by stride.
__global__ void __launch_bounds__(kSpWarps * 32, 4)
    k_sample_phase(ThinView G, const int4 *__restrict__ small, const int4 *__restrict__ large,
                   int *__restrict__ ph, int phase, float r2, int *__restrict__ keptFlag,
                   int *__restrict__ aliveTmp) {
    smd::chain_enter(); // phases are chained launches: the previous phase's cells are final
    __shared__ float4 stageBuf[kSpBuf]; // heavy cell: [0, kSpHStage); warp w: its slice
    __shared__ int    sCell;
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int off = phase_off(ph, phase);
    const int nS = ph[kPhSmall + phase], nM = ph[kPhMedium + phase], nH = ph[kPhHeavy + phase];
    while (nH > 0) {
        if (threadIdx.x == 0)
            sCell = atomicAdd(&ph[kPhTaken + phase], 1);
        __syncthreads();
        const int hc = sCell;
        __syncthreads(); // every thread has read sCell before it is taken again
        if (hc >= nH)
            break;
        sp_heavy(G, large[off + ph[kPhCells + phase] - 1 - hc], r2, keptFlag, aliveTmp, stageBuf);
    }
    float4   *stage = stageBuf + wl * kSpStage;
    const int w0    = blockIdx.x * kSpWarps + wl, nw = gridDim.x * kSpWarps;
    for (int w = w0; w < nM; w += nw)
        sp_medium(G, large[off + w], r2, keptFlag, stage);
    // (from the other end of the grid: the warps without a medium cell start)
    if (nS <= nw) { // a warp for each: the shortest chain where there are warps enough
        for (int w = nw - 1 - w0; w < nS; w += nw)
            sp_medium(G, small[off + w], r2, keptFlag, stage);
        return;
    }
    for (int w = nw - 1 - w0; 4 * w < nS; w += nw) {
        const int  k    = 4 * w + (lane >> 3);
        const bool live = k < nS;
        sp_small(G, live ? small[off + k] : make_int4(0, 0, 0, 0), live, r2, keptFlag,
                 stage + (lane >> 3) * kSpGStage);
    }
}

// ---------------------------------------------------------------------------------------
__global__ void k_mark_todo(const int *__restrict__ ids, int m, const float4 *__restrict__ nrm,
                            NormalList L) {
    chain_enter(); // launched chained
    const int i   = blockIdx.x * blockDim.x + threadIdx.x;
    const int id  = i < m ? ids[i] : 0;
    bool      add = false;
    if (i < m) {
        const float4 n = nrm[id];
        add            = !finite3(n.x, n.y, n.z);
        if (add)
            atomicOr(&L.seen[id >> 5], 1u << (id & 31));
    }
    warp_append(add, id, L.list, L.count);
}

// One warp per query (exact k nearest neighbours, sm_device.cuh warp_knn_sorted) of part `part`
// of the list; lane j writes the j-th neighbour, and with `grow` lists it when it still needs a
// normal. Five CTAs an SM: at six the ring search spills, at four the large scene's queries took
// 85 + 82 us, at five 77 + 74.
__global__ void __launch_bounds__(256, 5)
    k_knn(NormalList L, int part, HGridView G, const float4 *__restrict__ pos, int k, bool grow,
          const float4 *__restrict__ nrm) {
    chain_enter(); // launched chained
    const int lane = threadIdx.x & 31;
    const int t    = L.begin(part) +
                  (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (t >= L.end(part))
        return;
    const float4 q = pos[L.list[t]];
    int          id;
    float        d;
    const int    n = warp_knn_sorted(G, q.x, q.y, q.z, k, &id, &d);
    if (lane < k)
        L.nbr[(size_t)t * k + lane] = lane < n ? id : -1;
    if (lane == 0)
        L.nbrCnt[t] = n;
    if (grow)
        L.add_neighbour(lane < n, id, nrm);
}

// ---- hashed grid build -----------------------------------------------------------------
__device__ __forceinline__ unsigned long long hkey(const float4 &p, const GridParams &gp) {
    const int cx = smg::coord(p.x, gp.org[0], gp.g, gp.dim[0]);
    const int cy = smg::coord(p.y, gp.org[1], gp.g, gp.dim[1]);
    const int cz = smg::coord(p.z, gp.org[2], gp.g, gp.dim[2]);
    return ((unsigned long long)cz * (unsigned)gp.dim[1] + (unsigned)cy) * (unsigned)gp.dim[0] +
           (unsigned)cx;
}

// Grid, three passes over one table: points count themselves into their cell's entry, then every
// occupied cell takes its points' range from a counter (a CTA's at once; the cells' order in the
// point arrays does not matter), then the points go to their places. The table is a direct one
// where the cell box is small (DIRECT: {first, count}), else hashed: slots of {key low, key high,
// first point, points - 1}, all ones where empty (so that one fill clears it), claimed by the
// cell's 64-bit key, half as many again as points. Bounded by the table's bytes and two atomics a
// point. (A key table, a count table, their scan, a copy of the scan and a pack into the slots
// moved twice the bytes; the slots rounded up to a power of two, with a CTA and its add to the
// counter per 256 of them, took 25 us in the second pass of 0.92 M points' grid, now 10, and 71 us
// in all, now 55. Both tables beside each other cost the small clouds, which read the direct one
// only, a third more.)
constexpr int kHgRun = 8; // entries a thread of the second pass
template <bool DIRECT>
__global__ void k_hg_insert(const float4 *__restrict__ pos, const int *__restrict__ ids, int m,
                            GridParams gp, uint4 *__restrict__ slot, uint32_t slots,
                            int2 *__restrict__ dense, int2 *__restrict__ place) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const unsigned long long key = hkey(pos[ids[i]], gp);
    if (DIRECT) {
        place[i] = make_int2((int)key, atomicAdd(&dense[key].y, 1));
        return;
    }
    uint32_t h = hg_slot(key, slots);
    for (uint32_t p = 0; p < slots; p++) {
        unsigned long long      *k    = reinterpret_cast<unsigned long long *>(&slot[h]);
        const unsigned long long prev = atomicCAS(k, ~0ull, key);
        if (prev == ~0ull || prev == key) {
            // (the count starts at all ones: the first point takes place 0)
            place[i] = make_int2((int)h, (int)(atomicAdd(&slot[h].w, 1u) + 1u));
            return;
        }
        h = h + 1 < slots ? h + 1 : 0;
    }
}

// Ranges of the occupied cells (of T entries), and the hashed ones' occupancy bits.
template <bool DIRECT>
__global__ void __launch_bounds__(256)
    k_hg_ranges(uint4 *__restrict__ slot, uint32_t T, int2 *__restrict__ dense,
                int *__restrict__ next, uint32_t *__restrict__ occ) {
    chain_enter(); // launched chained
    __shared__ int sh[33];
    __shared__ int sBase;
    const uint32_t     t0 = blockIdx.x * (256u * kHgRun) + threadIdx.x;
    int                cnt[kHgRun], sum = 0;
    unsigned long long key[kHgRun];
#pragma unroll
    for (int r = 0; r < kHgRun; r++) {
        const uint32_t t = t0 + 256u * r;
        if (DIRECT) {
            cnt[r] = t < T ? dense[t].y : 0;
        } else {
            const uint4 v = t < T ? slot[t] : make_uint4(~0u, ~0u, ~0u, ~0u);
            cnt[r]        = (int)(v.w + 1u);
            key[r]        = ((unsigned long long)v.y << 32) | v.x;
        }
    }
#pragma unroll
    for (int r = 0; r < kHgRun; r++)
        sum += cnt[r];
    int       tot;
    const int ex = block_excl_scan(sum, sh, &tot);
    if (tot == 0)
        return; // (uniform)
    if (threadIdx.x == 0)
        sBase = atomicAdd(next, tot);
    __syncthreads();
    int first = sBase + ex;
#pragma unroll
    for (int r = 0; r < kHgRun; r++) {
        if (cnt[r] == 0)
            continue;
        const uint32_t t = t0 + 256u * r;
        if (DIRECT) {
            dense[t].x = first;
        } else {
            slot[t].z = (uint32_t)first;
            if (occ)
                atomicOr(&occ[key[r] >> 5], 1u << (key[r] & 31));
        }
        first += cnt[r];
    }
}

template <bool DIRECT>
__global__ void k_hg_scatter(const float4 *__restrict__ pos, const int *__restrict__ ids,
                             const uint4 *__restrict__ slot, const int2 *__restrict__ dense,
                             const int2 *__restrict__ place, int m, float4 *__restrict__ pts,
                             int wIsRank) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const int    id = ids[i];
    const float4 p  = pos[id];
    const int2   at = place[i];
    const int    first = DIRECT ? dense[at.x].x : (int)slot[at.x].z;
    pts[first + at.y]  = make_float4(p.x, p.y, p.z, __int_as_float(wIsRank ? i : id));
}

// Rank-ordered copies of a subset's positions and normals: out[r] = in[ids[r]].
__global__ void k_gather_subset(const float4 *__restrict__ pos, const float4 *__restrict__ nrm,
                                const int *__restrict__ ids, int m, float4 *__restrict__ subPos,
                                float4 *__restrict__ subNrm) {
    chain_enter(); // launched chained
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= m)
        return;
    const int id = ids[r];
    subPos[r]    = pos[id];
    subNrm[r]    = nrm[id];
}

// Phase A: centroid and FP32-Kahan covariance of the neighbourhood, FP64 eigensolve, for the
// whole list.
__global__ void k_pca(NormalList L, int k, const float4 *__restrict__ pos, float4 *__restrict__ cen,
                      float4 *__restrict__ nout) {
    chain_enter(); // launched chained
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.end(1))
        return;
    const int  m = L.nbrCnt[t];
    const int *N = L.nbr + (size_t)t * k;
    if (m < 3) {
        cen[t]  = make_float4(0.f, 0.f, 0.f, -1.0f); // w < 0: no estimate
        nout[t] = make_float4(0.f, 0.f, 0.f, -1.0f);
        return;
    }
    smi::KahanF sx, sy, sz;
    sx.init();
    sy.init();
    sz.init();
    for (int j = 0; j < m; j++) {
        const float4 p = pos[N[j]];
        sx.add(p.x);
        sy.add(p.y);
        sz.add(p.z);
    }
    const float cx = smm::fdiv(sx.value(), (float)m), cy = smm::fdiv(sy.value(), (float)m),
                cz = smm::fdiv(sz.value(), (float)m);
    smi::KahanF a[6];
    for (int e = 0; e < 6; e++)
        a[e].init();
    for (int j = 0; j < m; j++) {
        const float4 p  = pos[N[j]];
        const float  dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
        a[0].add(dx * dx);
        a[1].add(dx * dy);
        a[2].add(dx * dz);
        a[3].add(dy * dy);
        a[4].add(dy * dz);
        a[5].add(dz * dz);
    }
    double C[6];
    for (int e = 0; e < 6; e++)
        C[e] = (double)a[e].value();
    float n3[3];
    sml::normal_from_cov(C, n3);
    cen[t]  = make_float4(cx, cy, cz, 1.0f);
    nout[t] = make_float4(n3[0], n3[1], n3[2], 1.0f);
}

__global__ void k_pca_write(NormalList L, const float4 *__restrict__ cen,
                            const float4 *__restrict__ nin, float4 *__restrict__ pos,
                            float4 *__restrict__ nrm) {
    chain_enter(); // launched chained
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.end(1) || cen[t].w < 0.0f)
        return;
    const int id = L.list[t];
    pos[id]      = make_float4(cen[t].x, cen[t].y, cen[t].z, 0.0f);
    nrm[id]      = make_float4(nin[t].x, nin[t].y, nin[t].z, 0.0f);
}

// Phase B: sign-aligned sum of the raw neighbourhood normals (util.cpp:292-306) of the points
// to estimate.
__global__ void k_smooth(NormalList L, int k, const float4 *__restrict__ nrm,
                         float4 *__restrict__ out) {
    chain_enter(); // launched chained
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.end(0))
        return;
    const int m = L.nbrCnt[t];
    if (m < 3) {
        out[t] = make_float4(0.f, 0.f, 0.f, -1.0f);
        return;
    }
    const float4 n0 = nrm[L.list[t]];
    float        sx = 0.f, sy = 0.f, sz = 0.f;
    for (int j = 0; j < m; j++) {
        const float4 n = nrm[L.nbr[(size_t)t * k + j]];
        const float  d = n.x * n0.x + (n.y * n0.y + n.z * n0.z);
        if (d > 0.0f) {
            sx = sx + n.x;
            sy = sy + n.y;
            sz = sz + n.z;
        } else {
            sx = sx - n.x;
            sy = sy - n.y;
            sz = sz - n.z;
        }
    }
    const float sq = sx * sx + (sy * sy + sz * sz);
    if (sq > 0.0f) {
        const float s = smm::fsqrt(sq);
        sx            = smm::fdiv(sx, s);
        sy            = smm::fdiv(sy, s);
        sz            = smm::fdiv(sz, s);
    }
    out[t] = make_float4(sx, sy, sz, 1.0f);
}

__global__ void k_smooth_write(NormalList L, const float4 *__restrict__ sm,
                               float4 *__restrict__ nrm) {
    chain_enter(); // launched chained
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= L.end(0) || sm[t].w < 0.0f)
        return;
    nrm[L.list[t]] = make_float4(sm[t].x, sm[t].y, sm[t].z, 0.0f);
}

// Phase C: orientation toward the viewpoint, or +z (util.cpp:309-333).
__global__ void k_orient(const int *__restrict__ ids, int m, const float4 *__restrict__ pos,
                         float4 *__restrict__ nrm, int hasVp, float vx, float vy, float vz,
                         int invert) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    const int id = ids[i];
    float4    n  = nrm[id];
    float     d;
    if (hasVp) {
        const float4 p = pos[id];
        const float  ax = vx - p.x, ay = vy - p.y, az = vz - p.z;
        d               = n.x * ax + (n.y * ay + n.z * az);
    } else {
        d = n.x * 0.0f + (n.y * 0.0f + n.z * 1.0f);
    }
    const bool flip = invert ? (d > 0.0f) : (d < 0.0f);
    if (flip)
        nrm[id] = make_float4(-n.x, -n.y, -n.z, 0.0f);
}

__global__ void k_normalize(float4 *__restrict__ nrm, int n) {
    chain_enter(); // launched chained
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    float4      v  = nrm[i];
    const float sq = v.x * v.x + (v.y * v.y + v.z * v.z);
    if (sq > 0.0f) {
        const float s = smm::fsqrt(sq);
        nrm[i]        = make_float4(smm::fdiv(v.x, s), smm::fdiv(v.y, s), smm::fdiv(v.z, s), 0.0f);
    }
}

} // namespace

// =======================================================================================
int prep_points(Ctx &c, const float *xyz, const float *nin, int n, float4 *pos, float4 *nrm,
                int *validFlag, Box &box) {
    int *dev = c.arena.get<int>("prep.bbox", 8);
    k_init_bbox<<<1, 32, 0, c.stream>>>(dev, dev + 6);
    SM_LAUNCH_CHECK();
    const int bs = 256;
    const int nb = std::max(1, std::min(nblocks(nblocks(n, 4), bs), 152 * 8));
    k_prep<<<nb, bs, 0, c.stream>>>(xyz, nin, n, pos, nrm, validFlag, dev, dev + 6);
    SM_LAUNCH_CHECK();
    SM_CUDA(cudaMemcpyAsync(c.hostCounts, dev, 7 * sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    for (int a = 0; a < 3; a++) {
        box.mn[a] = ord2f(c.hostCounts[a]);
        box.mx[a] = ord2f(c.hostCounts[3 + a]);
    }
    return c.hostCounts[6];
}

// The context's look-back state, grown to at least nparts tiles (zeroed when allocated);
// returns the next scan epoch.
unsigned scan_state(Ctx &c, int nparts) {
    Ctx::ScanState &S = c.scan;
    if (nparts > S.cap || S.epoch >= (1u << 30) - 1) {
        const int cap = std::max(nparts, std::max(S.cap, 1024));
        S.status      = c.arena.get<unsigned long long>("scan.status", cap);
        S.ticket      = c.arena.get<int>("scan.ticket", 2);
        SM_CUDA(cudaMemsetAsync(S.status, 0, (size_t)cap * 8, c.stream));
        SM_CUDA(cudaMemsetAsync(S.ticket, 0, 2 * sizeof(int), c.stream));
        S.cap   = cap;
        S.epoch = 0;
    }
    return ++S.epoch;
}

// A scan of n values (see ScanOut); the total goes to *total (device) when given.
template <ScanOut MODE>
static void scan_launch(Ctx &c, const int *in, int *out, long long n, const int *ids, int *total) {
    const int nparts = (int)((n + kScanTile - 1) / kScanTile);
    if (nparts == 0) {
        if (total)
            SM_CUDA(cudaMemsetAsync(total, 0, sizeof(int), c.stream));
        return;
    }
    const unsigned epoch = scan_state(c, nparts);
    cudaEvent_t    t0    = c.clock.begin(c.stream);
    launch_chained(c, k_scan_lookback<ScanInts, MODE>, nparts, kScanBs, 0, ScanInts{in}, out, n, ids,
                   c.scan.status, c.scan.ticket, nparts, epoch, total);
    c.clock.end(c.stream, t0, KernelClock::kScan, 8.0 * (double)n); // 4-byte value in, 4 out
}

// *total (device) to the host.
static int read_total(Ctx &c, const int *total) {
    SM_CUDA(cudaMemcpyAsync(c.hostCounts, total, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    c.sync_checked();
    return c.hostCounts[0];
}

int scan_excl(Ctx &c, const int *in, int *out, long long n, const std::string &tag, bool wantTotal) {
    int *total = c.arena.get<int>(tag + ".scantot", 1);
    scan_launch<kPrefix>(c, in, out, n, nullptr, total);
    return wantTotal ? read_total(c, total) : -1;
}

int compact(Ctx &c, const int *flags, int n, int *outIds, const std::string &tag) {
    if (n <= 0)
        return 0;
    int *total = c.arena.get<int>(tag + ".scantot", 1);
    scan_launch<kSelect>(c, flags, outIds, n, nullptr, total);
    return read_total(c, total);
}

void compact_known(Ctx &c, const int *flags, int n, int count, int *outIds) {
    if (n <= 0)
        return;
    if (count == n) // every flag is set
        launch_chained(c, k_iota, nblocks(n, 256), 256, 0, outIds, n);
    else
        scan_launch<kSelect>(c, flags, outIds, n, nullptr, nullptr);
}

// With a tree beside it a grid is not built where the extent (a stray point some 2^20 cells off, or a
// huge number in the place of a missing value) makes its cells more than kCoarse times the wanted
// ones: a cell's points grow with their square, and the tree's own searches, a thread each, do not
// depend on the extent. (0.92 M points with strays 4, 8, 16, 32 and 64 km and 1000 km away: on the
// grid 10.6, 12.5, 21.9, 48, 113 and 868 ms a call, on the tree 16.6 to 18.1 up to 64 km; 0.1 M
// points 4.6, 4.7, 5.6, 8.7, 23 and 61 against 6.3 to 6.5. Far less than four times, the grid is
// faster; without a stray it takes 7.5 against 13.4 ms.)
constexpr float kCoarse = 4.0f;

void build_hgrid(Ctx &c, const float4 *pos, const int *ids, int m, const Box &box, float g,
                 HGrid &H, const std::string &tag, bool wIsRank, bool tree) {
    // (any cell side gives the same results: without a wanted one, some 1000 cells an axis)
    if (!(g > 0.0f))
        g = std::max(std::max(box.ext(0), box.ext(1)), std::max(box.ext(2), 1e-30f)) / 1024.0f;
    const float want = g;
    // cells per axis stay below 2^20 so that cell keys fit 60 bits (coarser cells if needed; the
    // loop ends: dim_of is 1 where the side overflows)
    while (smg::dim_of(box.ext(0), g) >= (1 << 20) || smg::dim_of(box.ext(1), g) >= (1 << 20) ||
           smg::dim_of(box.ext(2), g) >= (1 << 20))
        g = g * 2.0f;
    H.g      = g;
    H.coarse = tree && g > kCoarse * want;
    for (int a = 0; a < 3; a++) {
        H.org[a] = box.mn[a];
        H.dim[a] = smg::dim_of(box.ext(a), g);
    }
    H.slack     = box.slack(g);
    H.m         = m;
    if (H.coarse)
        return;
    int  *next  = c.arena.get<int>(tag + ".next", 2);
    int2 *place = c.arena.get<int2>(tag + ".place", std::max(m, 1));
    H.pts       = c.arena.get<float4>(tag + ".pts", std::max(m, 1));
    H.next      = next;
    // a direct {first, count} table over a cell box of at most 2^22 cells (32 MB), else the hashed
    // one, with occupancy bits over a box of at most 2^28 cells (32 MB); cleared with the counter
    // in one launch
    const unsigned long long ncell  = (unsigned long long)H.dim[0] * H.dim[1] * H.dim[2];
    const size_t             words  = (size_t)((ncell + 31) / 32);
    const bool               direct = ncell <= (1ull << 22);
    H.slots = direct ? 0u : (uint32_t)m + (uint32_t)m / 2u + 64u;
    H.dense = direct ? c.arena.get<int2>(tag + ".dense", (size_t)ncell) : nullptr;
    H.slot  = direct ? nullptr : c.arena.get<uint4>(tag + ".slot", H.slots);
    H.occ   = !direct && ncell <= (1ull << 28) ? c.arena.get<uint32_t>(tag + ".occ", words) : nullptr;
    FillSet clear;
    clear.add(next, 2 * sizeof(int), 0u);
    if (H.dense)
        clear.add(H.dense, (size_t)ncell * sizeof(int2), 0u);
    if (H.slot)
        clear.add(H.slot, (size_t)H.slots * sizeof(uint4), 0xffffffffu);
    if (H.occ)
        clear.add(H.occ, words * 4, 0u);
    fill(c, clear);
    if (m <= 0)
        return;
    const GridParams gp  = grid_params(box, g, H.dim);
    const uint32_t   T   = direct ? (uint32_t)ncell : H.slots;
    const int        gm  = nblocks(m, 256), gt = nblocks(T, 256 * kHgRun);
    const int        isR = wIsRank ? 1 : 0;
    if (direct) {
        launch_chained(c, k_hg_insert<true>, gm, 256, 0, pos, ids, m, gp, H.slot, H.slots, H.dense, place);
        launch_chained(c, k_hg_ranges<true>, gt, 256, 0, H.slot, T, H.dense, next, H.occ);
        launch_chained(c, k_hg_scatter<true>, gm, 256, 0, pos, ids, H.slot, H.dense, place, m, H.pts, isR);
    } else {
        launch_chained(c, k_hg_insert<false>, gm, 256, 0, pos, ids, m, gp, H.slot, H.slots, H.dense, place);
        launch_chained(c, k_hg_ranges<false>, gt, 256, 0, H.slot, T, H.dense, next, H.occ);
        launch_chained(c, k_hg_scatter<false>, gm, 256, 0, pos, ids, H.slot, H.dense, place, m, H.pts, isR);
    }
}

void gather_subset(Ctx &c, const float4 *pos, const float4 *nrm, const int *ids, int m,
                   float4 *subPos, float4 *subNrm) {
    if (m <= 0)
        return;
    launch_chained(c, k_gather_subset, nblocks(m, 256), 256, 0, pos, nrm, ids, m, subPos,
                   subNrm);
}

int sample_points(Ctx &c, const float4 *pos, int npoints, const int *ids, int m, const Box &box,
                  float step, int *outIds, const std::string &tag) {
    if (m <= 0)
        return 0;
    if (!(step > 0.0f)) {
        // no point lies at a squared distance below zero: every point is kept (the list is
        // ascending already)
        SM_CUDA(cudaMemcpyAsync(outIds, ids, (size_t)m * sizeof(int), cudaMemcpyDeviceToDevice,
                                c.stream));
        return m;
    }
    float ext[3] = {box.ext(0), box.ext(1), box.ext(2)};
    const float g = smg::thin_cell(step, ext);
    // the cell table over the points (dense or hashed, see ThinView), its occupied cells
    // listed per phase on the device (no host round trip; at most m of them)
    int dim[3];
    for (int a = 0; a < 3; a++)
        dim[a] = smg::dim_of(ext[a], g);
    uint32_t T = 1024;
    while (T < 2u * (uint32_t)m)
        T <<= 1;
    // dense table (slot = cell key) when the cell box has at most 2^22 cells or 16 per
    // point, never above 2^27 cells: its counts are cleared and read once, 8 bytes a cell, where
    // the hashed one claims a key per point (dense tables of 24 and 45 cells a point for the
    // resampling of 0.92 M and 2.6 M points cost 1.6 and 3.3 % of the whole call)
    const unsigned long long ncell = (unsigned long long)dim[0] * dim[1] * dim[2];
    const unsigned long long dmax  = std::max<unsigned long long>(1ull << 22, 16ull * (unsigned)m);
    const bool               dense = ncell <= std::min<unsigned long long>(dmax, 1ull << 27);
    if (dense)
        T = (uint32_t)ncell;
    ThinView V;
    for (int a = 0; a < 3; a++)
        V.dim[a] = dim[a];
    auto *keys  = dense ? nullptr : c.arena.get<unsigned long long>(tag + ".g.keys", T);
    int  *cnt   = c.arena.get<int>(tag + ".g.cnt", T);
    auto *pts   = c.arena.get<float4>(tag + ".g.pts", m);
    V.keys      = keys;
    V.mask      = dense ? 0u : T - 1;
    V.cnt       = cnt;
    V.info      = c.arena.get<int2>(tag + ".g.info", T);
    V.pts       = pts;
    V.keptPos   = c.arena.get<float4>(tag + ".kp", m);
    V.m         = m;
    int2 *place = c.arena.get<int2>(tag + ".g.place", m);
    int  *ph    = c.arena.get<int>(tag + ".ph", kPhWords);
    int4 *small = c.arena.get<int4>(tag + ".phs", m); // (at most a cell per point)
    int4 *large = c.arena.get<int4>(tag + ".phl", m);
    int  *keptFlag = c.arena.get<int>(tag + ".kf", m); // over the list places
    int  *aliveTmp = c.arena.get<int>(tag + ".al", m);
    FillSet clear;
    if (!dense)
        clear.add(keys, (size_t)T * 8, 0xffffffffu);
    clear.add(cnt, (size_t)T * sizeof(int), 0u);
    clear.add(ph, kPhWords * sizeof(int), 0u);
    fill(c, clear);
    const GridParams gpar = grid_params(box, g, dim);
    launch_chained(c, k_thin_insert, nblocks(m, kSpBs), kSpBs, 0, pos, ids, m, gpar, keys, V.mask,
                   place, cnt, ph);
    launch_chained(c, k_thin_cells, nblocks(T, 4 * kSpBs), kSpBs, 0, V, T, ph, small, large);
    launch_chained(c, k_thin_scatter, nblocks(m, 256), 256, 0, pos, ids, m, place, V.info, pts,
                   keptFlag);
    const float r2 = step * step;
    // one resident wave: heavy cells are handed out by a counter, the others by stride
    static std::atomic<int> resident[64];
    const int               dev = c.device >= 0 && c.device < 64 ? c.device : 0;
    int                     per = resident[dev].load();
    if (per <= 0) {
        SM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sample_phase, kSpWarps * 32, 0));
        per = std::max(per, 1);
        resident[dev].store(per);
    }
    int nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    const int gp = (int)std::min<long long>((m + kSpWarps - 1) / kSpWarps, (long long)nsm * per);
    for (int p = 0; p < 8; p++) {
        cudaEvent_t t0 = c.clock.begin(c.stream);
        launch_chained(c, k_sample_phase, gp, kSpWarps * 32, 0, V, small, large, ph, p, r2, keptFlag,
                       aliveTmp);
        // algorithmic bytes of a sampling: each point's position read and its flag written
        // once (16 + 4 bytes), spread over the 8 phases
        c.clock.end(c.stream, t0, KernelClock::kSamplePhase, 20.0 * (double)m / 8.0);
    }
    // the kept points in index order (list order) and their number
    int *total = c.arena.get<int>(tag + ".res", 1);
    scan_launch<kSelectIds>(c, keptFlag, outIds, m, ids, total);
    SM_CUDA(cudaMemcpyAsync(c.hostCounts, total, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    c.sync();
    return c.hostCounts[0];
}

void estimate_normals(Ctx &c, float4 *pos, float4 *nrm, int npoints, const int *ids, int m,
                      const HGrid &query, int k, bool smooth, bool invert, const float *vp,
                      const std::string &tag, const KdTree *tree) {
    if (m <= 0)
        return;
    if (k < 3)
        k = 3;
    if (k > kMaxKnn)
        throw Error(SM_ERR_RANGE, "knnNormal larger than " + std::to_string(kMaxKnn) + " is not supported");
    // the list and its counts stay on the device; launches are sized by bounds
    const int  extraMax = smooth ? (int)std::min<long long>(npoints, (long long)m * k) : 0;
    const long long most = (long long)m + extraMax;
    NormalList L;
    L.list   = c.arena.get<int>(tag + ".list", (size_t)most);
    L.seen   = c.arena.get<uint32_t>(tag + ".seen", ((size_t)npoints + 31) / 32);
    L.count  = c.arena.get<int>(tag + ".count", 2);
    L.nbr    = c.arena.get<int>(tag + ".nbr", (size_t)most * k);
    L.nbrCnt = c.arena.get<int>(tag + ".nbrCnt", (size_t)most);
    FillSet clear;
    clear.add(L.seen, ((size_t)npoints + 31) / 32 * 4, 0u);
    clear.add(L.count, 2 * sizeof(int), 0u);
    fill(c, clear);
    launch_chained(c, k_mark_todo, nblocks(m, 256), 256, 0, ids, m, nrm, L);
    // with the reference's k-d tree the k nearest are those its depth-first search finds
    // (ties: first found)
    for (int part = 0; part < (extraMax > 0 ? 2 : 1); part++) {
        const int  nq   = part ? extraMax : m;
        const bool grow = part == 0 && smooth;
        if (tree)
            kd_knn_points(c, *tree, query, pos, L, part, nq, k, grow, nrm);
        else
            launch_chained(c, k_knn, nblocks((long long)nq * 32, 256), 256, 0, L, part,
                           query.view(), pos, k, grow, nrm);
    }
    float4 *cen = c.arena.get<float4>(tag + ".cen", (size_t)most);
    float4 *nn  = c.arena.get<float4>(tag + ".nn", (size_t)most);
    launch_chained(c, k_pca, nblocks(most, 128), 128, 0, L, k, pos, cen, nn);
    launch_chained(c, k_pca_write, nblocks(most, 256), 256, 0, L, cen, nn, pos, nrm);
    if (smooth) {
        launch_chained(c, k_smooth, nblocks(m, 256), 256, 0, L, k, nrm, cen);
        launch_chained(c, k_smooth_write, nblocks(m, 256), 256, 0, L, cen, nrm);
    }
    const bool hasVp = vp && std::isfinite(vp[0]) && std::isfinite(vp[1]) && std::isfinite(vp[2]);
    launch_chained(c, k_orient, nblocks(m, 256), 256, 0, ids, m, pos, nrm, hasVp ? 1 : 0,
                   hasVp ? vp[0] : 0.f, hasVp ? vp[1] : 0.f, hasVp ? vp[2] : 0.f, invert ? 1 : 0);
}

void normalize_normals(Ctx &c, float4 *nrm, int n) {
    if (n <= 0)
        return;
    launch_chained(c, k_normalize, nblocks(n, 256), 256, 0, nrm, n);
}

} // namespace sm
