// summary.cuh -- the field summary in the reference's summation order
// (2d field_summary.c:8-45, 3d field_summary.c:8-49: one serial loop, x
// fastest, then y, then z), formed in parallel with the serial loop's result
// bit for bit: vol, mass and ie equal the reference's and temp differs only
// by the solution itself.
//
// While a running sum acc of non-negative terms stays in one binade [2^E,
// 2^(E+1)), every value it takes is a multiple of u = 2^(E-52), and adding x
// raises it by a multiple of u that depends only on x and, when x / u is
// half-way between two integers, on whether acc / u is even or odd. So a run
// of terms acts on acc as a pair of increments (i0 for an even acc, i1 for an
// odd one), both exact doubles; pairs compose associatively, and the order of
// a run without half-way cases does not even matter. A term's pair is
// (B + x) - B and (B1 + x) - B1 with B = 2^E and B1 = B + u, in two roundings
// the hardware makes. The binade of a run has to be known beforehand: pass 1
// (k_summary_sums) sums tiles in any order, whose prefix sums give each
// tile's start and end to about 1e-9; pass 2 (k_summary_pairs) forms the
// pairs of the tiles that lie in one binade by a margin of 2^-20, and of
// super-tiles of kTiles tiles; the last pass (k_field_summary_ordered)
// applies super-tiles to the exact acc, 32 at a time, as long as acc is in
// their binade and stays in it, and goes through the few others (one for each
// binade crossed, and any with a negative or non-finite term) tile by tile,
// group of 32 terms by group, and term by term where a group crosses. Nothing
// rests on the estimates: a pair is applied only to an acc that is seen to be
// in its binade before and after.
//
// Two reads of four fields bound it, and one block's walk through the binades
// (about 5 us each). A whole call, against the serial chain of adds alone:
// 128^2 0.094 / 0.110 ms, 512^2 0.132 / 1.48, 4096^2 0.604 / 93.1, 8192^2
// 1.89 / 372.
#pragma once

#include "common.cuh"

namespace tl __attribute__((visibility("hidden"))) {

constexpr int kTileCells = 256;                  // cells of a tile: 8 per lane of a warp
constexpr int kTiles = 32;                       // tiles of a super-tile: one per lane of a warp
constexpr int kSuperWarps = 16;
constexpr int kSuperThreads = 32 * kSuperWarps;
constexpr long kSumDirect = 12288;               // up to this many cells the serial loop is the faster
constexpr int kAnyBinade = 1 << 20;              // pair of a run of zeros: applies to any acc
constexpr int kNoBinade = -(1 << 20);            // no pair: the run has to be gone through
constexpr int kMinBinade = -960, kMaxBinade = 1000;
constexpr double kBinadeMargin = 1.0 / (1 << 20);

struct SumFields {   // the summed cells, in order, and their fields
    int x, hd, hdz, nx, ny;
    long xy, n;
    const double *volume, *density, *energy0, *u;
};

struct SumPair {     // increments of a run of terms
    double i0, i1;
};

struct SumScratch {
    double* tile;       // [tiles][4] sums, any order; NaN where a term is negative or not finite
    double* super;      // [supers][4] sums, then their exclusive prefixes
    SumPair* tpair;     // [tiles][4]
    SumPair* spair;     // [supers][4]
    int* tbin;          // [tiles][4] binades
    int* sbin;          // [supers][4]
    unsigned* ticket;
};

inline long sum_supers(long n) { return (n + (long)kTiles * kTileCells - 1) / ((long)kTiles * kTileCells); }
// Device memory of the scratch for n cells.
inline size_t sum_scratch_bytes(long n)
{
    const size_t s = (size_t)sum_supers(n);
    return s * (kTiles + 1) * 4 * (sizeof(double) + sizeof(SumPair) + sizeof(int)) + 256;
}
inline SumScratch sum_scratch(void* base, long n)   // base zeroed once (the ticket returns to 0)
{
    const size_t s = (size_t)sum_supers(n), t = s * kTiles;
    SumScratch c;
    c.ticket = (unsigned*)base;
    c.tpair = (SumPair*)((char*)base + 256);
    c.spair = c.tpair + t * 4;
    c.tile = (double*)(c.spair + s * 4);
    c.super = c.tile + t * 4;
    c.tbin = (int*)(c.super + s * 4);
    c.sbin = c.tbin + t * 4;
    return c;
}

__device__ __forceinline__ long sum_index(const SumFields& f, long c)
{
    long r, k;
    if (f.n <= 0xffffffffL) {
        r = (unsigned)c / (unsigned)f.nx;
        k = c - r * f.nx;
    } else {
        r = c / f.nx;
        k = c % f.nx;
    }
    long z = 0;
    if (r >= f.ny) {
        z = r <= 0xffffffffL ? (long)((unsigned)r / (unsigned)f.ny) : r / f.ny;
        r -= z * f.ny;
    }
    return (f.hdz + z) * f.xy + (f.hd + r) * f.x + (f.hd + k);
}

// Terms of cell c in the reference's expressions; zeros past the end.
__device__ __forceinline__ void sum_terms(const SumFields& f, long c, double (&t)[4])
{
    t[0] = t[1] = t[2] = t[3] = 0.0;
    if (c >= f.n) return;
    const long i = sum_index(f, c);
    const double cv = f.volume[i], cm = cv * f.density[i];
    t[0] = cv;
    t[1] = cm;
    t[2] = cm * f.energy0[i];
    t[3] = cm * f.u[i];
}

// Exponent of a positive normal double with room for its ulp, else kNoBinade.
__device__ __forceinline__ int binade(double v)
{
    const int e = (int)((unsigned long long)__double_as_longlong(v) >> 52) - 1023;   // (sign set: large)
    return e >= kMinBinade && e <= kMaxBinade ? e : kNoBinade;
}
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
__device__ __forceinline__ int odd(double v) { return (int)(__double_as_longlong(v) & 1); }

// First f, then g, on sums in the binade of base = 2^E (even).
__device__ __forceinline__ SumPair then(const SumPair& f, const SumPair& g, double base)
{
    SumPair h;
    h.i0 = f.i0 + (odd(base + f.i0) ? g.i1 : g.i0);
    h.i1 = f.i1 + (odd(base + f.i1) ? g.i0 : g.i1);
    return h;
}
__device__ __forceinline__ SumPair shfl_down(const SumPair& p, int o)
{
    return {__shfl_down_sync(0xffffffffu, p.i0, o), __shfl_down_sync(0xffffffffu, p.i1, o)};
}
// Lanes 0 .. 31 in order; lane 0 has the composition.
__device__ __forceinline__ SumPair warp_then(SumPair p, double base)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) p = then(p, shfl_down(p, o), base);
    return p;
}

// Pass 1: a block per super-tile, a warp for two of its tiles.
static __global__ void __launch_bounds__(kSuperThreads) k_summary_sums(SumFields f, SumScratch s, int supers)
{
    __shared__ double part[kSuperWarps][4];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double whole[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = 0; q < kTiles / kSuperWarps; ++q) {
        const long tile = (long)blockIdx.x * kTiles + warp * (kTiles / kSuperWarps) + q;
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        bool bad[4] = {false, false, false, false};
#pragma unroll
        for (int k = 0; k < kTileCells / 32; ++k) {
            double t[4];
            sum_terms(f, tile * kTileCells + k * 32 + lane, t);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                a[m] += t[m];
                bad[m] = bad[m] || !(t[m] >= 0.0 && t[m] < 1e300);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            a[m] = warp_sum(a[m]);
            const bool b = __any_sync(0xffffffffu, bad[m]);
            whole[m] += a[m];
            if (lane == 0) s.tile[tile * 4 + m] = b ? __longlong_as_double(0x7ff8000000000000LL) : a[m];
        }
    }
    if (lane == 0)
#pragma unroll
        for (int m = 0; m < 4; ++m) part[warp][m] = whole[m];
    __syncthreads();
    if (threadIdx.x < 4) {
        double t = 0.0;
        for (int w = 0; w < kSuperWarps; ++w) t += part[w][threadIdx.x];
        s.super[(long)blockIdx.x * 4 + threadIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(s.ticket, 1u) == (unsigned)(supers - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last block: exclusive prefixes, 128 threads per sum, each a run of super-tiles
    __shared__ double run[4][4];
    const int m = warp & 3, c = (warp >> 2) * 32 + lane;
    const int per = (supers + 127) / 128, b0 = min(c * per, supers), b1 = min(b0 + per, supers);
    double t = 0.0;
    for (int b = b0; b < b1; ++b) t += __ldcg(&s.super[(long)b * 4 + m]);
    double v = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double w = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += w;
    }
    if (lane == 31) run[m][warp >> 2] = v;
    if (threadIdx.x == 0) *s.ticket = 0u;
    __syncthreads();
    t = v - t;
    for (int w = 0; w < (warp >> 2); ++w) t += run[m][w];
    for (int b = b0; b < b1; ++b) {
        const double w = __ldcg(&s.super[(long)b * 4 + m]);
        s.super[(long)b * 4 + m] = t;
        t += w;
    }
}

// Pass 2: the pairs of tiles and super-tiles.
static __global__ void __launch_bounds__(kSuperThreads) k_summary_pairs(SumFields f, SumScratch s)
{
    __shared__ double start[kTiles + 1][4];
    __shared__ SumPair pair[kTiles][4];
    __shared__ int bin[kTiles][4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long tile0 = (long)blockIdx.x * kTiles;
    if (warp < 4) {   // estimated starts of the tiles (a NaN sum spoils those after it: they have no pair)
        const double base = s.super[(long)blockIdx.x * 4 + warp];
        double v = s.tile[(tile0 + lane) * 4 + warp];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double w = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += w;
        }
        start[lane + 1][warp] = base + v;
        if (lane == 0) start[0][warp] = base;
    }
    __syncthreads();
    for (int q = 0; q < kTiles / kSuperWarps; ++q) {
        const int t = warp * (kTiles / kSuperWarps) + q;
        double x[kTileCells / 32][4];
#pragma unroll
        for (int k = 0; k < kTileCells / 32; ++k) sum_terms(f, (tile0 + t) * kTileCells + k * 32 + lane, x[k]);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const double own = s.tile[(tile0 + t) * 4 + m];
            const int lo = binade(start[t][m] * (1.0 - kBinadeMargin));
            const int hi = binade(start[t + 1][m] * (1.0 + kBinadeMargin));
            SumPair p{0.0, 0.0};
            int e = kNoBinade;
            if (own == 0.0) {
                e = kAnyBinade;
            } else if (lo == hi && lo != kNoBinade && own > 0.0) {
                e = lo;
                const double base = pow2(e), base1 = base + pow2(e - 52);
                double d0[kTileCells / 32], d1[kTileCells / 32];
                bool ties = false;
#pragma unroll
                for (int k = 0; k < kTileCells / 32; ++k) {
                    d0[k] = (base + x[k][m]) - base;
                    d1[k] = (base1 + x[k][m]) - base1;
                    ties = ties || d0[k] != d1[k];
                }
                if (__any_sync(0xffffffffu, ties)) {
                    for (int k = 0; k < kTileCells / 32; ++k) {   // groups in order, lanes in order
                        SumPair g = warp_then(SumPair{d0[k], d1[k]}, base);
                        p = then(p, g, base);
                    }
                } else {
                    double d = 0.0;
#pragma unroll
                    for (int k = 0; k < kTileCells / 32; ++k) d += d0[k];
                    d = warp_sum(d);
                    p = SumPair{d, d};
                }
            }
            if (lane == 0) {
                pair[t][m] = p;
                bin[t][m] = e;
                s.tpair[(tile0 + t) * 4 + m] = p;
                s.tbin[(tile0 + t) * 4 + m] = e;
            }
        }
    }
    __syncthreads();
    if (warp < 4) {   // the super-tile's pair, where its tiles share a binade
        const int own = bin[lane][warp];
        int e = __reduce_max_sync(0xffffffffu, own == kAnyBinade ? kNoBinade : own);
        const bool zeros = __all_sync(0xffffffffu, own == kAnyBinade);
        if (!__all_sync(0xffffffffu, own == e || own == kAnyBinade)) e = kNoBinade;
        SumPair p{0.0, 0.0};
        if (e != kNoBinade) p = warp_then(pair[lane][warp], pow2(e));
        if (lane == 0) {
            s.spair[(long)blockIdx.x * 4 + warp] = p;
            s.sbin[(long)blockIdx.x * 4 + warp] = zeros ? kAnyBinade : e;
        }
    }
}

// Applies the runs of lanes 0 .. count - 1 in order to acc, as far as acc is
// and stays in their binade; returns how many.
__device__ __forceinline__ int sum_advance(double& acc, SumPair p, int e, int count)
{
    const int lane = threadIdx.x & 31;
    const int b = binade(acc);
    bool ok = lane < count && (e == kAnyBinade || (e == b && b != kNoBinade));
    const double base = b == kNoBinade ? 1.0 : pow2(b);
    if (!ok || e == kAnyBinade) p = SumPair{0.0, 0.0};
    if (__any_sync(0xffffffffu, p.i0 != p.i1)) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const SumPair g{__shfl_up_sync(0xffffffffu, p.i0, o), __shfl_up_sync(0xffffffffu, p.i1, o)};
            if (lane >= o) p = then(g, p, base);
        }
    } else {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double g = __shfl_up_sync(0xffffffffu, p.i0, o);
            if (lane >= o) p.i0 += g;
        }
        p.i1 = p.i0;
    }
    const double end = acc + (odd(acc) ? p.i1 : p.i0);
    if (b != kNoBinade) ok = ok && end < 2.0 * base;
    const unsigned bad = ~__ballot_sync(0xffffffffu, ok);
    const int first = bad ? __ffs(bad) - 1 : 32;
    if (first > 0) acc = __shfl_sync(0xffffffffu, end, first - 1);
    return first;
}

constexpr int kGroups = kTileCells / 32;   // groups of 32 cells of a tile

// Terms of sum m of a tile's cells (zeros past the end).
__device__ __forceinline__ void tile_terms(const SumFields& f, long tile, int m, double (&x)[kGroups])
{
    const double* const c = m == 2 ? f.energy0 : f.u;
    double v[kGroups], d[kGroups], e[kGroups];
#pragma unroll
    for (int k = 0; k < kGroups; ++k) {
        const long n = tile * kTileCells + k * 32 + (threadIdx.x & 31);
        const long i = n < f.n ? sum_index(f, n) : 0;
        v[k] = n < f.n ? f.volume[i] : 0.0;
        d[k] = n < f.n && m > 0 ? f.density[i] : 1.0;
        e[k] = n < f.n && m > 1 ? c[i] : 1.0;
    }
#pragma unroll
    for (int k = 0; k < kGroups; ++k) x[k] = v[k] * d[k] * e[k];
}

// Adds the terms of a tile's cells to the exact acc: the groups' pairs in the
// binade acc has now, all at once, applied up to the group that leaves it (or
// holds a term that has no pair); that one term by term, and the rest anew.
__device__ __forceinline__ double sum_tile(double acc, const double (&x)[kGroups])
{
    int k0 = 0;
    while (k0 < kGroups) {
        const int b = binade(acc);
        const double base = b == kNoBinade ? 0.0 : pow2(b), base1 = base + (b == kNoBinade ? 0.0 : pow2(b - 52));
        SumPair p[kGroups];
        bool ties = false;
        unsigned fit = 0;
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
            fit |= __all_sync(0xffffffffu, x[k] >= 0.0 && x[k] < base) ? 1u << k : 0u;
            p[k].i0 = (base + x[k]) - base;
            p[k].i1 = (base1 + x[k]) - base1;
            ties = ties || p[k].i0 != p[k].i1;
        }
        if (__any_sync(0xffffffffu, ties)) {
#pragma unroll
            for (int k = 0; k < kGroups; ++k) p[k] = warp_then(p[k], base);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < kGroups; ++k) p[k].i0 += __shfl_down_sync(0xffffffffu, p[k].i0, o);
#pragma unroll
            for (int k = 0; k < kGroups; ++k) p[k].i1 = p[k].i0;
        }
        int stop = kGroups;   // the first group that cannot be applied
#pragma unroll
        for (int k = 0; k < kGroups; ++k) {
            if (k < k0 || k >= stop) continue;
            const double end = __shfl_sync(0xffffffffu, acc + (odd(acc) ? p[k].i1 : p[k].i0), 0);
            if ((fit >> k & 1u) && end < 2.0 * base) acc = end;
            else stop = k;
        }
        if (stop < kGroups) {
            double y = x[0];
#pragma unroll
            for (int k = 1; k < kGroups; ++k) y = k == stop ? x[k] : y;
#pragma unroll
            for (int q = 0; q < 32; ++q) acc += __shfl_sync(0xffffffffu, y, q);
        }
        k0 = stop + 1;
    }
    return acc;
}

// The last pass: warp m forms sum m.
static __global__ void __launch_bounds__(128) k_field_summary_ordered(SumFields f, SumScratch s, int supers,
                                                                     double* out_dev, double* out_host)
{
    const int lane = threadIdx.x & 31, m = threadIdx.x >> 5;
    double acc = 0.0;
    const long tiles = (f.n + kTileCells - 1) / kTileCells;
    double x[kGroups];
    for (long b = 0; b < supers;) {
        const int count = (int)min(32L, supers - b);
        const long q = (b + min(lane, count - 1)) * 4 + m;
        const int n = sum_advance(acc, s.spair[q], s.sbin[q], count);
        b += n;
        if (n == count) continue;
        const int own = (int)min((long)kTiles, tiles - b * kTiles);   // tiles of super-tile b
        const long qt = (b * kTiles + lane) * 4 + m;
        const SumPair p = s.tpair[qt];
        const int e = s.tbin[qt];
        for (int t = 0; t < own;) {
            const SumPair pt{__shfl_sync(0xffffffffu, p.i0, lane + t), __shfl_sync(0xffffffffu, p.i1, lane + t)};
            const int nt = sum_advance(acc, pt, __shfl_sync(0xffffffffu, e, lane + t), own - t);
            t += nt;
            if (t == own) break;
            tile_terms(f, b * kTiles + t, m, x);
            acc = sum_tile(acc, x);
            ++t;
        }
        ++b;
    }
    if (lane == 0) {
        out_dev[m] = acc;
        if (out_host) out_host[m] = acc;
    }
}

// The serial loop itself, for meshes of up to kSumDirect cells: each of the
// four sums is one dependent chain of adds: warp w < 4 (lane 0) advances sum w
// through a shared-memory tile of per-cell terms while the producer warps form
// the next tile's terms from coalesced loads. One block; the chains' add
// latency bounds it (5.6 ns per cell: 23 us at 64^2, where the three passes
// above take 60; they meet at about 12000 cells).
constexpr int kSumTile = 1024;              // cells per tile
constexpr int kSumProducers = 256;          // producer threads (8 warps)
constexpr int kSumThreads = 128 + kSumProducers;
constexpr size_t kSumSmem = 2 * 4 * kSumTile * sizeof(double);

static __global__ void __launch_bounds__(kSumThreads) k_field_summary_serial(SumFields f, double* out_dev,
                                                                            double* out_host)
{
    extern __shared__ double terms[];   // [2 buffers][4 sums][kSumTile]
    const long n = f.n;
    const long ntiles = (n + kSumTile - 1) / kSumTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pt = (int)threadIdx.x - 128;   // producer thread id (< 0: a chain warp)

    auto produce = [&](long t) {
        double* dst = terms + (t & 1) * 4 * kSumTile;
        const long base = t * kSumTile;
        for (int m = pt; m < kSumTile; m += kSumProducers) {
            const long c = base + m;
            if (c >= n) break;
            double v[4];
            sum_terms(f, c, v);
            for (int q = 0; q < 4; ++q) dst[q * kSumTile + m] = v[q];
        }
    };

    double acc = 0.0;
    if (pt >= 0 && ntiles > 0) produce(0);
    __syncthreads();
    for (long t = 0; t < ntiles; ++t) {
        if (pt >= 0) {
            if (t + 1 < ntiles) produce(t + 1);
        } else if (lane == 0) {
            const double* src = terms + (t & 1) * 4 * kSumTile + warp * kSumTile;
            const int cnt = (int)min((long)kSumTile, n - t * kSumTile);
            if (cnt == kSumTile) {
#pragma unroll 16
                for (int m = 0; m < kSumTile; ++m) acc += src[m];
            } else {
                for (int m = 0; m < cnt; ++m) acc += src[m];
            }
        }
        __syncthreads();
    }
    if (pt < 0 && lane == 0) {
        out_dev[warp] = acc;
        if (out_host) out_host[warp] = acc;
    }
}

// The summary's launches, each through `launch(name, kernel call)`.
template <typename Launch>
inline void field_summary_ordered(cudaStream_t st, const SumFields& f, const SumScratch& s, double* out_dev,
                                  double* out_host, Launch launch)
{
    if (f.n <= kSumDirect) {
        // (raised on each call, so that every device a process uses is covered)
        cudaFuncSetAttribute(k_field_summary_serial, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem);
        launch("k_field_summary_serial",
               [&] { k_field_summary_serial<<<1, kSumThreads, kSumSmem, st>>>(f, out_dev, out_host); });
        return;
    }
    const int supers = (int)sum_supers(f.n);
    launch("k_summary_sums", [&] { k_summary_sums<<<supers, kSuperThreads, 0, st>>>(f, s, supers); });
    launch("k_summary_pairs", [&] { k_summary_pairs<<<supers, kSuperThreads, 0, st>>>(f, s); });
    launch("k_field_summary_ordered",
           [&] { k_field_summary_ordered<<<1, 128, 0, st>>>(f, s, supers, out_dev, out_host); });
}

}  // namespace tl
