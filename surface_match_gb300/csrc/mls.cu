// mls.cu - moving-least-squares normals and surface projection of listed points
// (estimateNormalMLS, util.cpp:336-457, declared in privateUtil.h:13).
//
// For each listed point p, over its neighbours closer than the radius (strict <, the k-d
// tree's radius search, util.cpp:357-362; points with fewer than 3 are left unchanged):
//   1. PCA plane: centroid c, covariance, n = eigenvector of the smallest eigenvalue
//      (util.cpp:368-381); the normal output takes n here already, as the reference writes
//      it before its later exits.
//   2. The query projected on the plane, m = p - (n.(p - c)) n, and a tangent frame:
//      v = a unit vector orthogonal to n (Eigen's unitOrthogonal), u = n x v
//      (util.cpp:385-390).
//   3. A weighted least-squares fit of the heights f = (q - m).n over the tangent
//      coordinates by the polynomial of total degree `order` with monomials u^a v^b in the
//      order a = 0..order, b = 0..order-a; weights exp(-|q - m|^2 / r^2)
//      (util.cpp:392-436). Order <= 1 with fewer neighbours than coefficients stops at 1.
//   4. The point moves to the fit's value at the origin, m + c0 n, and the normal is
//      n - c_u u - c_v v, normalised (c_u, c_v: the coefficients of u and v, indices
//      order+1 and 1), then oriented toward the viewpoint (or +z) with the invert rule of
//      the normal estimator (util.cpp:439-455).
//
// Deterministic two-phase form: neighbourhoods always read the positions at the start of
// the call, and results go to separate outputs (the reference projects points in place
// while other threads read them as neighbours). Where the weighted system is not positive
// definite (Eigen's LLT then reports a numerical issue and its solve returns an unspecified
// vector) the point keeps the PCA normal, as for a non-finite solution.
//
// Three kernels over a hashed grid of cell just above the radius, so that the 3x3x3 block holds
// every neighbour. k_mls_near, a warp per listed point, collects its neighbours; k_mls_fit, a
// thread per point, makes everything of them; k_mls_wide, a warp per point, does it for points with
// too many. The work is FP64 (eigenvector, Cholesky) and a few dozen sums, and GB300 issues an FP64
// warp instruction at the same cost for one active lane as for 32: with a warp per point for all of
// it, 50,000 points of 30 neighbours at order 2 took 2080 us of a call's 2640, now the call takes
// 340. Sums are FP32 Kahan per point, read out with their compensation in FP64; the fit runs in
// coordinates scaled by 1/r (the same polynomial, better conditioned); the small systems are solved
// in FP64.
#include <cmath>

#include "sm_device.cuh"
#include "sm_icp.h"
#include "sm_linalg.h"
#include "sm_stages.h"

namespace sm {
namespace {

constexpr int kMlsWarps = 8;       // points per CTA of the neighbour kernel
constexpr int kMlsFitBs = 64;      // threads per CTA of the fit kernel
constexpr int kMlsNear  = 128;     // neighbours listed per point; a point with more walks the grid
constexpr int kMlsCount = 288;     // neighbours counted, of a point with more than are listed
constexpr int kMlsChunk = 1 << 18; // points per launch pair (128 MB of lists)

struct MlsArgs {
    smd::HGridView g; // the finite points; cell side >= 1.02 radius
    const float4  *pos;
    const int     *ids;
    float          r, r2;
    int            invert, hasVp;
    float          vx, vy, vz;
    float         *outXyz, *outNrm; // n x 3, pre-filled with the inputs
};

__device__ __forceinline__ bool finite3f(float x, float y, float z) {
    return isfinite(x) && isfinite(y) && isfinite(z);
}

__device__ __forceinline__ float powi(float x, int e) {
    float r = 1.0f;
    for (int i = 0; i < e; i++)
        r *= x;
    return r;
}

// In-place Cholesky solve of the SPD system G c = b (G: lower triangle, rows of N); false when
// a pivot is not positive or the solution is not finite.
template <int N> __device__ bool cholesky_solve(double (&G)[N][N], double (&b)[N]) {
#pragma unroll
    for (int j = 0; j < N; j++) {
        double d = G[j][j];
#pragma unroll
        for (int k = 0; k < j; k++)
            d -= G[j][k] * G[j][k];
        if (!(d > 0.0))
            return false;
        const double s = sqrt(d);
        G[j][j]        = s;
#pragma unroll
        for (int i = j + 1; i < N; i++) {
            double v = G[i][j];
#pragma unroll
            for (int k = 0; k < j; k++)
                v -= G[i][k] * G[j][k];
            G[i][j] = v / s;
        }
    }
#pragma unroll
    for (int i = 0; i < N; i++) { // L y = b
        double v = b[i];
#pragma unroll
        for (int k = 0; k < i; k++)
            v -= G[i][k] * b[k];
        b[i] = v / G[i][i];
    }
#pragma unroll
    for (int i = N - 1; i >= 0; i--) { // L^T c = y
        double v = b[i];
#pragma unroll
        for (int k = i + 1; k < N; k++)
            v -= G[k][i] * b[k];
        b[i] = v / G[i][i];
        if (!isfinite(b[i]))
            return false;
    }
    return true;
}

// The same in loops, for a system in shared memory.
__device__ bool cholesky_solve(double *G, double *b, int n) {
    for (int j = 0; j < n; j++) {
        double d = G[j * n + j];
        for (int k = 0; k < j; k++)
            d -= G[j * n + k] * G[j * n + k];
        if (!(d > 0.0))
            return false;
        const double s = sqrt(d);
        G[j * n + j]   = s;
        for (int i = j + 1; i < n; i++) {
            double v = G[i * n + j];
            for (int k = 0; k < j; k++)
                v -= G[i * n + k] * G[j * n + k];
            G[i * n + j] = v / s;
        }
    }
    for (int i = 0; i < n; i++) { // L y = b
        double v = b[i];
        for (int k = 0; k < i; k++)
            v -= G[i * n + k] * b[k];
        b[i] = v / G[i * n + i];
    }
    for (int i = n - 1; i >= 0; i--) { // L^T c = y
        double v = b[i];
        for (int k = i + 1; k < n; k++)
            v -= G[k * n + i] * b[k];
        b[i] = v / G[i * n + i];
        if (!isfinite(b[i]))
            return false;
    }
    return true;
}

// The neighbours of listed point i0 + t (places in g.pts) in the lists' order: neighbour j of
// the points of a warp of k_mls_fit is one line of near; cnt[t] their number, counted to
// some kMlsCount. Points with more than are listed are named in wide[], counted on from base in
// nwide[0], and their numbers added to nwide[1]. (Counting on costs up to 5 %: 50,000 points of 200
// neighbours 1291 -> 1358 us. Their number estimated from what the list's end left of the block
// misses the line of mls_by by too much.)
__global__ void __launch_bounds__(kMlsWarps * 32)
    k_mls_near(MlsArgs a, int i0, int n, int *__restrict__ near, int *__restrict__ cnt,
               int *__restrict__ wide, int *__restrict__ nwide, int base) {
    smd::chain_enter(); // launched chained
    const int lane = threadIdx.x & 31;
    const int t    = blockIdx.x * kMlsWarps + (threadIdx.x >> 5);
    if (t >= n)
        return; // warp-uniform
    const float4 q   = a.pos[a.ids[i0 + t]];
    int          num = 0;
    if (finite3f(q.x, q.y, q.z)) { // (a search from a non-finite point finds nothing)
        int c[3], b = 0, e = 0;
        smd::grid_cc(a.g, q.x, q.y, q.z, c);
        if (lane < 27) {
            const int x = c[0] + lane % 3 - 1, y = c[1] + (lane / 3) % 3 - 1,
                      z = c[2] + lane / 9 - 1;
            if (x >= 0 && y >= 0 && z >= 0 && x < a.g.dim[0] && y < a.g.dim[1] &&
                z < a.g.dim[2] && smd::cell_lb2(a.g, q.x, q.y, q.z, x, y, z) <= a.r2)
                a.g.range(x, y, z, b, e);
        }
        const int incl = smd::warp_incl_scan(e - b);
        const int excl = incl - (e - b);
        const int T    = __shfl_sync(0xffffffffu, incl, 31);
        int      *L    = near + (size_t)(t >> 5) * (32 * kMlsNear) + (t & 31);
        for (int r0 = 0; r0 < T && num <= kMlsCount; r0 += 32) {
            const int r   = r0 + lane;
            int       own = 0; // the lane whose cell holds point r: last lane with excl <= r
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1)
                if (__shfl_sync(0xffffffffu, excl, own + step) <= r)
                    own += step;
            const int at = __shfl_sync(0xffffffffu, b, own) + (r - __shfl_sync(0xffffffffu, excl, own));
            bool      in = false;
            if (r < T) {
                const float4 p = a.g.pts[at];
                in             = smm::dist2(q.x, q.y, q.z, p.x, p.y, p.z) < a.r2;
            }
            const unsigned m = __ballot_sync(0xffffffffu, in);
            const int      j = num + __popc(m & ((1u << lane) - 1u));
            if (in && j < kMlsNear)
                L[32 * j] = at;
            num += __popc(m);
        }
    }
    if (lane == 0) {
        cnt[t] = num;
        if (num > kMlsNear) {
            wide[atomicAdd(nwide, 1) - base] = t;
            atomicAdd(nwide + 1, num);
        }
    }
}

// fn(p) for every neighbour p of q: the listed ones, or by a walk over the 3x3x3 block.
template <class F>
__device__ __forceinline__ void each_near(const MlsArgs &a, const float4 &q, const int *L, int cnt,
                                          F &&fn) {
    if (cnt <= kMlsNear) {
        for (int j = 0; j < cnt; j += 4) { // four neighbours' loads in flight
            float4 p[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (j + u < cnt)
                    p[u] = a.g.pts[L[32 * (j + u)]];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (j + u < cnt)
                    fn(p[u]);
        }
        return;
    }
    int c[3];
    smd::grid_cc(a.g, q.x, q.y, q.z, c);
    for (int k = 0; k < 27; k++) {
        const int x = c[0] + k % 3 - 1, y = c[1] + (k / 3) % 3 - 1, z = c[2] + k / 9 - 1;
        if (x < 0 || y < 0 || z < 0 || x >= a.g.dim[0] || y >= a.g.dim[1] || z >= a.g.dim[2] ||
            !(smd::cell_lb2(a.g, q.x, q.y, q.z, x, y, z) <= a.r2))
            continue;
        int b, e;
        a.g.range(x, y, z, b, e);
        for (int i = b; i < e; i++) {
            const float4 p = a.g.pts[i];
            if (smm::dist2(q.x, q.y, q.z, p.x, p.y, p.z) < a.r2)
                fn(p);
        }
    }
}

__device__ __forceinline__ double sum_of(const smi::KahanF &k) { return (double)k.s - (double)k.c; }

// The tangent frame of normal n.
__device__ __forceinline__ void mls_frame(const float n[3], float u[3], float v[3]) {
    if (!(fabsf(n[0]) <= fabsf(n[2]) * 1e-5f) || !(fabsf(n[1]) <= fabsf(n[2]) * 1e-5f)) {
        const float h = smm::fdiv(1.0f, smm::fsqrt(n[0] * n[0] + n[1] * n[1]));
        v[0]          = -n[1] * h;
        v[1]          = n[0] * h;
        v[2]          = 0.0f;
    } else {
        const float h = smm::fdiv(1.0f, smm::fsqrt(n[1] * n[1] + n[2] * n[2]));
        v[0]          = 0.0f;
        v[1]          = -n[2] * h;
        v[2]          = n[1] * h;
    }
    u[0] = n[1] * v[2] - n[2] * v[1];
    u[1] = n[2] * v[0] - n[0] * v[2];
    u[2] = n[0] * v[1] - n[1] * v[0];
}

// 4. The fit's coefficients b back in unscaled coordinates (c0 scales by r, the linear terms are
// slopes and do not change), and with them the point and its normal.
template <int ORDER>
__device__ __forceinline__ void mls_write(const MlsArgs &a, int id, const double *b, const float m[3],
                                          const float n[3], const float u[3], const float v[3]) {
    const float c0 = (float)(b[0] * (double)a.r);
    const float cv = (float)b[1], cu = (float)b[ORDER + 1];
    const float px = m[0] + c0 * n[0], py = m[1] + c0 * n[1], pz = m[2] + c0 * n[2];
    float       nx = n[0] - cu * u[0] - cv * v[0], ny = n[1] - cu * u[1] - cv * v[1],
          nz = n[2] - cu * u[2] - cv * v[2];
    const float nn = nx * nx + ny * ny + nz * nz;
    if (nn > 0.0f) {
        const float s = smm::fsqrt(nn);
        nx            = smm::fdiv(nx, s);
        ny            = smm::fdiv(ny, s);
        nz            = smm::fdiv(nz, s);
    }
    const float d = a.hasVp ? nx * (a.vx - px) + ny * (a.vy - py) + nz * (a.vz - pz) : nz;
    if (a.invert ? d > 0.0f : d < 0.0f) {
        nx = -nx;
        ny = -ny;
        nz = -nz;
    }
    float *outN = a.outNrm + 3 * (size_t)id;
    float *outP = a.outXyz + 3 * (size_t)id;
    outP[0]     = px;
    outP[1]     = py;
    outP[2]     = pz;
    outN[0]     = nx;
    outN[1]     = ny;
    outN[2]     = nz;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The place of moment u^i v^j (i + j <= D, i outer): rows 0 .. i - 1 come before it.
template <int D> __device__ __forceinline__ constexpr int moment_at(int i, int j) {
    return i * (D + 1) - i * (i - 1) / 2 + j;
}

// Exponents of monomial k of total degree <= order, u's outer.
__device__ __forceinline__ void monomial(int k, int order, int &i, int &j) {
    for (i = 0; k > order - i; i++)
        k -= order - i + 1;
    j = k;
}

// Which points of a launch of n a warp takes each: those with more neighbours than are listed, where
// they have enough more of them (W points, `sum` neighbours) for their warps to be done sooner than
// the threads' walks are; and all points of a small launch then, so that no thread's chain follows
// the warps'. A thread walks the 27 cells for three sums, loads one after the other, beside the other
// points' threads; the warps' kernel comes before those, with a chain of its own (a solve by one
// lane: some 130 us at order 3, 450 at order 4) and a time per point. By threads and by warps, of
// 16,000 points, W of them taken: order 2, mean 133 neighbours, W 273 350 and 369 us; 137, 3915 522
// and 576; 145, 1400 658 and 264; 182, 7300 898 and 683; 1000, 40 2695 and 603, 10,000 2685 and
// 1833. Order 3, 130, 4 332 and 458; 145, 5200 788 and 1001; 300, 8000 1331 and 1269. Order 4, 133,
// 273 518 and 1207; 300, 2000 1508 and 953. The line fits 393 such cases of clouds of 3,000 to
// 50,000 points, few of them more than 5 % slower than by threads.
enum MlsBy { kMlsThreads, kMlsWideByWarps, kMlsAllByWarps };
constexpr int kMlsSmall = 2048, kMlsWideCtas = 3; // (CTAs per SM)
__device__ __forceinline__ MlsBy mls_by(int n, const int *wide, int base, int order) {
    const int   W = wide[0] - base, sum = wide[1];
    const int   most = order == 1 ? 32768 : order == 2 ? 12288 : order == 3 ? 8192 : 6144;
    const float perWide = order == 1 ? 0.0f : order <= 3 ? 0.002f : 0.02f;
    const float perOther = order == 1 ? 0.0f : order == 2 ? 0.002f : 0.004f;
    if (W == 0 || W > most ||
        (float)sum < (float)W * ((float)kMlsNear + perWide * (float)W + perOther * (float)min(n - W, 16000)))
        return kMlsThreads;
    return n <= kMlsSmall ? kMlsAllByWarps : kMlsWideByWarps;
}

// The points that a warp takes each, which walks the 3x3x3 block for each sum: lane l owns the fit's
// sums l, l + 32, ... (the moments of the Gram matrix, then the right-hand side) and takes every
// neighbour.
template <int ORDER>
__global__ void __launch_bounds__(kMlsWarps * 32, kMlsWideCtas)
    k_mls_wide(MlsArgs a, int i0, int n, const int *__restrict__ num, const int *__restrict__ wide,
               const int *__restrict__ nwide, int base) {
    smd::chain_enter(); // launched chained
    constexpr int D = 2 * ORDER, NM = (D + 1) * (D + 2) / 2, NC = (ORDER + 1) * (ORDER + 2) / 2;
    constexpr int PER = (NM + NC + 31) / 32;
    __shared__ double sMom[kMlsWarps][NM + NC], sGram[kMlsWarps][NC * NC];
    const int         lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int         nw = *nwide - base;
    const MlsBy       by = mls_by(n, nwide, base, ORDER);
    if (by == kMlsThreads)
        return;
    const float r2 = a.r2, invR = smm::fdiv(1.0f, a.r);
    // the lane's sums: exponents of u and v, whether the term carries the height
    int  eu[PER], ev[PER];
    bool rhs[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int e = lane + 32 * k;
        rhs[k]      = e >= NM;
        monomial(rhs[k] ? min(e - NM, NC - 1) : e, rhs[k] ? ORDER : D, eu[k], ev[k]);
    }
    const int last = by == kMlsAllByWarps ? n : nw;
    for (int k0 = blockIdx.x * kMlsWarps + wid; k0 < last; k0 += gridDim.x * kMlsWarps) {
        const int t = by == kMlsAllByWarps ? k0 : wide[k0];
        if (num[t] < 3)
            continue;
        const int    id = a.ids[i0 + t];
        const float4 q  = a.pos[id];
        int          c[3];
        smd::grid_cc(a.g, q.x, q.y, q.z, c);
        auto each = [&](auto &&fn) { // fn(p, whether the lane's p is a neighbour), by all lanes
            smd::warp_block27(a.g, q.x, q.y, q.z, c, r2, [&](const float4 &p, bool valid) {
                fn(p, valid && smm::dist2(q.x, q.y, q.z, p.x, p.y, p.z) < r2);
                return false;
            });
        };
        smi::KahanF s0[3];
        int         cnt = 0;
        for (int d = 0; d < 3; d++)
            s0[d].init();
        each([&](const float4 &p, bool in) {
            if (in) {
                cnt++;
                s0[0].add(p.x - q.x);
                s0[1].add(p.y - q.y);
                s0[2].add(p.z - q.z);
            }
        });
        cnt              = __reduce_add_sync(0xffffffffu, cnt);
        const double inv = 1.0 / (double)cnt;
        const float  cx  = (float)((double)q.x + warp_sum(sum_of(s0[0])) * inv);
        const float  cy  = (float)((double)q.y + warp_sum(sum_of(s0[1])) * inv);
        const float  cz  = (float)((double)q.z + warp_sum(sum_of(s0[2])) * inv);
        smi::KahanF  s1[6];
        for (int e = 0; e < 6; e++)
            s1[e].init();
        each([&](const float4 &p, bool in) {
            if (in) {
                const float dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
                s1[0].add(dx * dx);
                s1[1].add(dx * dy);
                s1[2].add(dx * dz);
                s1[3].add(dy * dy);
                s1[4].add(dy * dz);
                s1[5].add(dz * dz);
            }
        });
        double C[6];
        for (int e = 0; e < 6; e++)
            C[e] = warp_sum(sum_of(s1[e]));
        float n3[3], u[3], v[3];
        sml::normal_from_cov(C, n3);
        if (lane < 3)
            a.outNrm[3 * (size_t)id + lane] = lane == 0 ? n3[0] : lane == 1 ? n3[1] : n3[2];
        if (ORDER <= 1 && NC > cnt)
            continue;
        const float dist = n3[0] * (q.x - cx) + n3[1] * (q.y - cy) + n3[2] * (q.z - cz);
        const float m[3] = {q.x - dist * n3[0], q.y - dist * n3[1], q.z - dist * n3[2]};
        mls_frame(n3, u, v);
        smi::KahanF acc[PER];
#pragma unroll
        for (int k = 0; k < PER; k++)
            acc[k].init();
        each([&](const float4 &p, bool in) {
            float w = 0.0f, uc = 0.0f, vc = 0.0f, fc = 0.0f;
            if (in) {
                const float dx = p.x - m[0], dy = p.y - m[1], dz = p.z - m[2];
                w  = expf(-smm::fdiv(dx * dx + dy * dy + dz * dz, r2));
                uc = (dx * u[0] + dy * u[1] + dz * u[2]) * invR;
                vc = (dx * v[0] + dy * v[1] + dz * v[2]) * invR;
                fc = (dx * n3[0] + dy * n3[1] + dz * n3[2]) * invR;
            }
            for (unsigned live = __ballot_sync(0xffffffffu, w > 0.0f); live; live &= live - 1u) {
                const int   j  = __ffs(live) - 1;
                const float wj = __shfl_sync(0xffffffffu, w, j);
                const float uj = __shfl_sync(0xffffffffu, uc, j);
                const float vj = __shfl_sync(0xffffffffu, vc, j);
                const float fj = __shfl_sync(0xffffffffu, fc, j);
#pragma unroll
                for (int k = 0; k < PER; k++) {
                    const float term = wj * powi(uj, eu[k]) * powi(vj, ev[k]);
                    acc[k].add(rhs[k] ? term * fj : term);
                }
            }
        });
        __syncwarp(); // (the last point's solve has read them)
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (lane + 32 * k < NM + NC)
                sMom[wid][lane + 32 * k] = sum_of(acc[k]);
        __syncwarp();
        for (int e = lane; e < NC * NC; e += 32) {
            int i, j, i2, j2;
            monomial(e / NC, ORDER, i, j);
            monomial(e % NC, ORDER, i2, j2);
            sGram[wid][e] = sMom[wid][moment_at<D>(i + i2, j + j2)];
        }
        __syncwarp();
        if (lane == 0) {
            double *b = &sMom[wid][NM];
            if (cholesky_solve(sGram[wid], b, NC))
                mls_write<ORDER>(a, id, b, m, n3, u, v);
        }
    }
}

// The listed points by a thread each, but for those that k_mls_wide takes.
template <int ORDER>
__global__ void __launch_bounds__(kMlsFitBs)
    k_mls_fit(MlsArgs a, int i0, int n, const int *__restrict__ near, const int *__restrict__ num,
              const int *__restrict__ nwide, int base) {
    smd::chain_enter(); // launched chained
    constexpr int D  = 2 * ORDER;               // the Gram entries are moments of degree <= D
    constexpr int NM = (D + 1) * (D + 2) / 2;   // u^i v^j, i + j <= D, i outer
    constexpr int NC = (ORDER + 1) * (ORDER + 2) / 2;
    const int t = blockIdx.x * kMlsFitBs + threadIdx.x;
    if (t >= n)
        return;
    const int   cnt = num[t];
    const MlsBy by  = mls_by(n, nwide, base, ORDER);
    if (cnt < 3 || by == kMlsAllByWarps || (by == kMlsWideByWarps && cnt > kMlsNear))
        return;
    const int    id = a.ids[i0 + t];
    const float4 q  = a.pos[id];
    const int   *L  = near + (size_t)(t >> 5) * (32 * kMlsNear) + (t & 31);

    // 1. centroid (offsets from q), then the covariance about it
    smi::KahanF s0[3];
    int         found = 0; // (cnt, where they are listed)
    for (int d = 0; d < 3; d++)
        s0[d].init();
    each_near(a, q, L, cnt, [&](const float4 &p) {
        found++;
        s0[0].add(p.x - q.x);
        s0[1].add(p.y - q.y);
        s0[2].add(p.z - q.z);
    });
    const double inv = 1.0 / (double)found;
    const float  cx  = (float)((double)q.x + sum_of(s0[0]) * inv);
    const float  cy  = (float)((double)q.y + sum_of(s0[1]) * inv);
    const float  cz  = (float)((double)q.z + sum_of(s0[2]) * inv);
    smi::KahanF  s1[6];
    for (int e = 0; e < 6; e++)
        s1[e].init();
    each_near(a, q, L, cnt, [&](const float4 &p) {
        const float dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
        s1[0].add(dx * dx);
        s1[1].add(dx * dy);
        s1[2].add(dx * dz);
        s1[3].add(dy * dy);
        s1[4].add(dy * dz);
        s1[5].add(dz * dz);
    });
    double C[6];
    for (int e = 0; e < 6; e++)
        C[e] = sum_of(s1[e]);
    float n3[3];
    sml::normal_from_cov(C, n3);
    float *outN = a.outNrm + 3 * (size_t)id;
    outN[0]     = n3[0];
    outN[1]     = n3[1];
    outN[2]     = n3[2];

    // 2. projection on the plane and the tangent frame
    const float dist = n3[0] * (q.x - cx) + n3[1] * (q.y - cy) + n3[2] * (q.z - cz);
    const float m[3] = {q.x - dist * n3[0], q.y - dist * n3[1], q.z - dist * n3[2]};
    float       u[3], v[3];
    mls_frame(n3, u, v);
    if (ORDER <= 1 && NC > cnt)
        return;

    // 3. the fit's sums
    smi::KahanF mom[NM], rhs[NC];
#pragma unroll
    for (int k = 0; k < NM; k++)
        mom[k].init();
#pragma unroll
    for (int k = 0; k < NC; k++)
        rhs[k].init();
    const float invR = smm::fdiv(1.0f, a.r);
    each_near(a, q, L, cnt, [&](const float4 &p) {
        const float dx = p.x - m[0], dy = p.y - m[1], dz = p.z - m[2];
        const float w  = expf(-smm::fdiv(dx * dx + dy * dy + dz * dz, a.r2));
        const float uc = (dx * u[0] + dy * u[1] + dz * u[2]) * invR;
        const float vc = (dx * v[0] + dy * v[1] + dz * v[2]) * invR;
        const float fc = (dx * n3[0] + dy * n3[1] + dz * n3[2]) * invR;
        float       pv[D + 1]; // powers of vc
#pragma unroll
        for (int j = 0; j <= D; j++)
            pv[j] = powi(vc, j);
        int k = 0, kr = 0;
#pragma unroll
        for (int i = 0; i <= D; i++) {
            const float wu = w * powi(uc, i);
#pragma unroll
            for (int j = 0; j <= D - i; j++) {
                const float term = wu * pv[j];
                mom[k++].add(term);
                if (i + j <= ORDER)
                    rhs[kr++].add(term * fc);
            }
        }
    });
    // monomial k of the fit: u^i v^j, i + j <= ORDER, i outer
    double G[NC][NC], b[NC];
    {
        int k = 0;
#pragma unroll
        for (int i = 0; i <= ORDER; i++)
#pragma unroll
            for (int j = 0; j <= ORDER - i; j++, k++) {
                b[k]  = sum_of(rhs[k]);
                int l = 0;
#pragma unroll
                for (int i2 = 0; i2 <= ORDER; i2++)
#pragma unroll
                    for (int j2 = 0; j2 <= ORDER - i2; j2++, l++)
                        if (l <= k) {
                            G[k][l] = sum_of(mom[moment_at<D>(i + i2, j + j2)]);
                        }
            }
    }
    if (!cholesky_solve(G, b))
        return;
    mls_write<ORDER>(a, id, b, m, n3, u, v);
}

template <int ORDER>
void fit(Ctx &c, const MlsArgs &a, int i0, int n, const int *near, const int *num, const int *wide,
         const int *nwide, int base) {
    int nsm = 0;
    SM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    launch_chained(c, k_mls_wide<ORDER>, std::min(nblocks(n, kMlsWarps), kMlsWideCtas * nsm), kMlsWarps * 32, 0, a,
                   i0, n, num, wide, nwide, base);
    launch_chained(c, k_mls_fit<ORDER>, nblocks(n, kMlsFitBs), kMlsFitBs, 0, a, i0, n, near, num, nwide,
                   base);
}

__global__ void k_fill_nan(float *x, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n)
        x[i] = __int_as_float(0x7fc00000);
}

} // namespace

void estimate_normals_mls(Ctx &c, const float4 *pos, const int *valid, int nvalid, const Box &box,
                          const int *ids, int m, float radius, int order, bool invert,
                          const float *vp, float *outXyz, float *outNrm) {
    const float r  = std::fabs(radius);
    const float r2 = radius * radius;
    if (m <= 0 || nvalid <= 0 || !(r2 > 0.0f))
        return; // no point has a neighbour within a zero radius
    // (coarser where the rounding of cell coordinates is more than the two hundredths)
    float g = r * 1.02f;
    while (box.slack(g) > smg::kCellSlack && !(r <= g * (1.0f - 2.0f * box.slack(g))) && g < 1e37f)
        g *= 1.25f;
    HGrid G;
    build_hgrid(c, pos, valid, nvalid, box, g, G, "mls.g");
    MlsArgs a;
    a.g      = G.view();
    a.pos    = pos;
    a.ids    = ids;
    a.r      = r;
    a.r2     = r2;
    a.invert = invert ? 1 : 0;
    a.hasVp  = vp && std::isfinite(vp[0]) && std::isfinite(vp[1]) && std::isfinite(vp[2]);
    a.vx     = a.hasVp ? vp[0] : 0.f;
    a.vy     = a.hasVp ? vp[1] : 0.f;
    a.vz     = a.hasVp ? vp[2] : 0.f;
    a.outXyz = outXyz;
    a.outNrm = outNrm;
    const int chunk = std::min(m, kMlsChunk);
    int      *near  = c.arena.get<int>("mls.near", (size_t)((chunk + 31) / 32) * 32 * kMlsNear);
    int      *num   = c.arena.get<int>("mls.num", (size_t)chunk * 2);
    int      *wide  = num + chunk;
    // the built grid's range counter, at the number of its points, goes on as the wide points', and
    // the word behind it, clear, as their neighbours'
    int *nwide = G.next, base = nvalid;
    for (int i0 = 0; i0 < m; i0 += chunk) {
        const int n = std::min(chunk, m - i0);
        if (i0 > 0) {
            SM_CUDA(cudaMemsetAsync(nwide, 0, 2 * sizeof(int), c.stream));
            base = 0;
        }
        launch_chained(c, k_mls_near, nblocks(n, kMlsWarps), kMlsWarps * 32, 0, a, i0, n, near, num, wide,
                       nwide, base);
        if (order == 1)
            fit<1>(c, a, i0, n, near, num, wide, nwide, base);
        else if (order == 2)
            fit<2>(c, a, i0, n, near, num, wide, nwide, base);
        else if (order == 3)
            fit<3>(c, a, i0, n, near, num, wide, nwide, base);
        else
            fit<4>(c, a, i0, n, near, num, wide, nwide, base);
    }
}

void fill_nan(Ctx &c, float *x, long long n) {
    if (n <= 0)
        return;
    k_fill_nan<<<nblocks(n, 256), 256, 0, c.stream>>>(x, n);
    SM_LAUNCH_CHECK();
}

} // namespace sm
