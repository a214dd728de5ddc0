// sm_scan.cuh - the single-pass scan and selection kernel shared by the point preparation
// (prep.cu) and the k-d tree build (kdtree.cu).
#pragma once

#include "sm_device.cuh"

namespace sm {

constexpr int kScanBs   = 512;
constexpr int kScanIpt  = 8;
constexpr int kScanTile = kScanBs * kScanIpt;

// Single-pass exclusive scan with decoupled look-back (Merrill & Garland, "Single-pass
// Parallel Prefix Scan with Decoupled Look-back", 2016). Tiles of kScanTile values take a
// ticket in launch order; a tile publishes its aggregate, then warp 0 walks back over the
// tiles before it, 32 at a time, summing aggregates until it meets a tile whose inclusive
// prefix is published, and publishes its own inclusive prefix. A tile waits only on tiles
// that took earlier tickets (already running or done), so every wait ends; each is bounded
// all the same and sets *err when its limit passes. Status words: epoch (30 bits, new per
// scan, so the array needs no reset) | flag (2 bits: 1 aggregate, 2 inclusive) | value.
constexpr unsigned long long kLbAgg = 1ull << 32, kLbIncl = 2ull << 32;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// An array's values: two 16-byte loads a thread where it is aligned to them.
struct ScanInts {
    const int *in;
    __device__ __forceinline__ bool skip() const { return false; }
    __device__ __forceinline__ void load(long long tile, long long n, int (&v)[kScanIpt]) const {
        const long long base = tile + (long long)threadIdx.x * kScanIpt;
        if (base + kScanIpt <= n && ((uintptr_t)in & 15) == 0) {
            *reinterpret_cast<int4 *>(&v[0]) = *reinterpret_cast<const int4 *>(in + base);
            *reinterpret_cast<int4 *>(&v[4]) = *reinterpret_cast<const int4 *>(in + base + 4);
            return;
        }
#pragma unroll
        for (int k = 0; k < kScanIpt; k++)
            v[k] = base + k < n ? in[base + k] : 0;
    }
};

// What a scan writes: kPrefix, out[i] = sum of the values before i; kSelect (0/1 flags), the
// places i of set flags packed into out; kSelectIds, ids[i] for these. A thread's eight prefixes
// are two 16-byte stores where the array is aligned to them. (Values and prefixes one by one, and
// with the selected places written by a second kernel from the stored prefixes, 0.92 M flags took
// 11 + 7 us, a table of 2 M counts 20 us.)
enum ScanOut { kPrefix, kSelect, kSelectIds };

// The values come from IN: skip(), uniform over the launch, ends it before it takes a ticket or
// writes anything; load() gives each thread its eight consecutive values of the tile from `base`
// (0 from n on), called by the whole CTA.
template <class IN, ScanOut MODE>
__global__ void __launch_bounds__(kScanBs)
    k_scan_lookback(IN in, int *__restrict__ out, long long n, const int *__restrict__ ids,
                    unsigned long long *__restrict__ status, int *__restrict__ ticket, int nparts,
                    unsigned epoch, int *__restrict__ total) {
    smd::chain_enter(); // launched chained
    if (in.skip())
        return;
    __shared__ int sh[33];
    __shared__ int sTile, sExcl;
    if (threadIdx.x == 0) {
        const int t = atomicAdd(ticket, 1);
        if (t == nparts - 1)
            ticket[0] = 0; // every ticket of this launch is taken: ready for the next scan
        sTile = t;
    }
    __syncthreads();
    const int       tile = sTile;
    const long long base = (long long)tile * kScanTile + (long long)threadIdx.x * kScanIpt;
    const bool      whole = base + kScanIpt <= n;
    alignas(16) int v[kScanIpt];
    in.load((long long)tile * kScanTile, n, v);
    int s = 0;
#pragma unroll
    for (int k = 0; k < kScanIpt; k++)
        s += v[k];
    int       agg;
    const int ex  = smd::block_excl_scan(s, sh, &agg);
    const unsigned long long tag = (unsigned long long)epoch << 34;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int       excl = 0;
        if (tile == 0) {
            if (lane == 0)
                st_relaxed_u64(&status[0], tag | kLbIncl | (unsigned)agg);
        } else {
            if (lane == 0)
                st_relaxed_u64(&status[tile], tag | kLbAgg | (unsigned)agg);
            for (int top = tile - 1;; top -= 32) {
                const int          p = top - lane; // lane 0: the nearest predecessor
                unsigned long long w = tag | kLbIncl; // lanes before tile 0: inclusive 0
                for (int it = 0;; it++) {
                    if (p >= 0)
                        w = ld_relaxed_u64(&status[p]);
                    const bool ready = (w >> 34) == epoch && ((w >> 32) & 3ull) != 0;
                    if (__all_sync(0xffffffffu, ready))
                        break;
                    if (it > (1 << 22)) {
                        if (lane == 0)
                            atomicExch(ticket + 1, 1);
                        w = tag | kLbIncl;
                        break;
                    }
                    __nanosleep(32);
                }
                const bool     isIncl = ((w >> 32) & 3ull) == 2ull;
                const unsigned incl   = __ballot_sync(0xffffffffu, isIncl);
                int            val    = (int)(unsigned)(w & 0xffffffffull);
                if (incl) {
                    const int first = __ffs(incl) - 1;
                    excl += __reduce_add_sync(0xffffffffu, lane <= first ? val : 0);
                    break;
                }
                excl += __reduce_add_sync(0xffffffffu, val);
            }
            if (lane == 0)
                st_relaxed_u64(&status[tile], tag | kLbIncl | (unsigned)(excl + agg));
        }
        if (lane == 0) {
            sExcl = excl;
            if (tile == nparts - 1 && total)
                *total = excl + agg;
        }
    }
    __syncthreads();
    int o = ex + sExcl;
    if constexpr (MODE != kPrefix) {
#pragma unroll
        for (int k = 0; k < kScanIpt; k++)
            if (v[k]) // (0 past the end)
                out[o++] = MODE == kSelectIds ? ids[base + k] : (int)(base + k);
    } else {
        alignas(16) int w[kScanIpt];
#pragma unroll
        for (int k = 0; k < kScanIpt; k++) {
            w[k] = o;
            o += v[k];
        }
        if (whole && ((uintptr_t)out & 15) == 0) {
            *reinterpret_cast<int4 *>(out + base)     = *reinterpret_cast<int4 *>(&w[0]);
            *reinterpret_cast<int4 *>(out + base + 4) = *reinterpret_cast<int4 *>(&w[4]);
        } else {
#pragma unroll
            for (int k = 0; k < kScanIpt; k++)
                if (base + k < n)
                    out[base + k] = w[k];
        }
    }
}

} // namespace sm
