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
// Two kernels over a hashed grid of cell just above the radius, so that the 3x3x3 block holds
// every neighbour. k_mls_near, a warp per listed point, collects its neighbours; k_mls_fit, a
// thread per point, makes everything of them. The work is FP64 (eigenvector, Cholesky) and a
// few dozen sums, and GB300 issues an FP64 warp instruction at the same cost for one active
// lane as for 32 and has no cheap way to spread one point's sums over a warp: with a warp per
// point for all of it, 50,000 points of 30 neighbours at order 2 took 2080 us, now 300 us (the
// call 2640 -> 710 us). Sums are FP32
// Kahan per point, read out with their compensation in FP64; the fit runs in coordinates
// scaled by 1/r (the same polynomial, better conditioned); the small systems are solved in
// FP64.
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

// The neighbours of listed point i0 + t (places in g.pts) in the lists' order: neighbour j of
// the points of a warp of k_mls_fit is one line of near; cnt[t] their number, also above the
// list's length.
__global__ void __launch_bounds__(kMlsWarps * 32)
    k_mls_near(MlsArgs a, int i0, int n, int *__restrict__ near, int *__restrict__ cnt) {
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
        for (int base = 0; base < T; base += 32) {
            const int r   = base + lane;
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
    if (lane == 0)
        cnt[t] = num;
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

template <int ORDER>
__global__ void __launch_bounds__(kMlsFitBs)
    k_mls_fit(MlsArgs a, int i0, int n, const int *__restrict__ near, const int *__restrict__ num) {
    constexpr int D  = 2 * ORDER;               // the Gram entries are moments of degree <= D
    constexpr int NM = (D + 1) * (D + 2) / 2;   // u^i v^j, i + j <= D, i outer
    constexpr int NC = (ORDER + 1) * (ORDER + 2) / 2;
    const int     t  = blockIdx.x * kMlsFitBs + threadIdx.x;
    if (t >= n)
        return;
    const int cnt = num[t];
    if (cnt < 3)
        return;
    const int    id = a.ids[i0 + t];
    const float4 q  = a.pos[id];
    const int   *L  = near + (size_t)(t >> 5) * (32 * kMlsNear) + (t & 31);

    // 1. centroid (offsets from q), then the covariance about it
    smi::KahanF s0[3];
    for (int d = 0; d < 3; d++)
        s0[d].init();
    each_near(a, q, L, cnt, [&](const float4 &p) {
        s0[0].add(p.x - q.x);
        s0[1].add(p.y - q.y);
        s0[2].add(p.z - q.z);
    });
    const double inv = 1.0 / (double)cnt;
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
    float *outP = a.outXyz + 3 * (size_t)id;
    outN[0]     = n3[0];
    outN[1]     = n3[1];
    outN[2]     = n3[2];

    // 2. projection on the plane and the tangent frame
    const float dist = n3[0] * (q.x - cx) + n3[1] * (q.y - cy) + n3[2] * (q.z - cz);
    const float mx = q.x - dist * n3[0], my = q.y - dist * n3[1], mz = q.z - dist * n3[2];
    float       v[3];
    if (!(fabsf(n3[0]) <= fabsf(n3[2]) * 1e-5f) || !(fabsf(n3[1]) <= fabsf(n3[2]) * 1e-5f)) {
        const float h = smm::fdiv(1.0f, smm::fsqrt(n3[0] * n3[0] + n3[1] * n3[1]));
        v[0]          = -n3[1] * h;
        v[1]          = n3[0] * h;
        v[2]          = 0.0f;
    } else {
        const float h = smm::fdiv(1.0f, smm::fsqrt(n3[1] * n3[1] + n3[2] * n3[2]));
        v[0]          = 0.0f;
        v[1]          = -n3[2] * h;
        v[2]          = n3[1] * h;
    }
    const float u[3] = {n3[1] * v[2] - n3[2] * v[1], n3[2] * v[0] - n3[0] * v[2],
                        n3[0] * v[1] - n3[1] * v[0]};
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
        const float dx = p.x - mx, dy = p.y - my, dz = p.z - mz;
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
                            const int A = i + i2, B = j + j2; // moments of rows 0 .. A-1 before it
                            G[k][l] = sum_of(mom[A * (D + 1) - A * (A - 1) / 2 + B]);
                        }
            }
    }
    if (!cholesky_solve(G, b))
        return;
    // 4. coefficients back to unscaled coordinates: c0 scales by r, the linear terms are
    // slopes and do not change
    const float c0 = (float)(b[0] * (double)a.r);
    const float cv = (float)b[1], cu = (float)b[ORDER + 1];
    const float px = mx + c0 * n3[0], py = my + c0 * n3[1], pz = mz + c0 * n3[2];
    float       nx = n3[0] - cu * u[0] - cv * v[0], ny = n3[1] - cu * u[1] - cv * v[1],
          nz = n3[2] - cu * u[2] - cv * v[2];
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
    outP[0] = px;
    outP[1] = py;
    outP[2] = pz;
    outN[0] = nx;
    outN[1] = ny;
    outN[2] = nz;
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
    int      *num   = c.arena.get<int>("mls.num", chunk);
    void (*const fit[kMlsMaxOrder])(MlsArgs, int, int, const int *, const int *) = {
        k_mls_fit<1>, k_mls_fit<2>, k_mls_fit<3>, k_mls_fit<4>};
    for (int i0 = 0; i0 < m; i0 += chunk) {
        const int n = std::min(chunk, m - i0);
        k_mls_near<<<nblocks(n, kMlsWarps), kMlsWarps * 32, 0, c.stream>>>(a, i0, n, near, num);
        SM_LAUNCH_CHECK();
        fit[order - 1]<<<nblocks(n, kMlsFitBs), kMlsFitBs, 0, c.stream>>>(a, i0, n, near, num);
        SM_LAUNCH_CHECK();
    }
}

void fill_nan(Ctx &c, float *x, long long n) {
    if (n <= 0)
        return;
    k_fill_nan<<<nblocks(n, 256), 256, 0, c.stream>>>(x, n);
    SM_LAUNCH_CHECK();
}

} // namespace sm
