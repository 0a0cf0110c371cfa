// gridsum.cuh -- exchange between the blocks of a persistent cooperative
// kernel by tagged words: grid-wide sums and the cells a block's neighbours
// read.
//
// Whatever one block hands to others travels as a 16-byte word {value, tag}
// written and read in one access, so the value is known to be the right one
// by the tag it comes with: no fence and no counter stands between the writer
// and the reader, and a hand-over costs one store and one load through L2. (A
// counter barrier followed by a read of the data is three dependent round
// trips and two fences of about 1000 cycles each: 3900-4500 cycles against
// 2200-2600 for 148 blocks.) The words of a block lie together, at least a
// 32-byte sector of them: where blocks share a sector their stores to it hold
// each other up (6200 cycles). A word is reused with the
// next tag; the callers see to it that it is rewritten only after all its
// readers have taken the old value. Waits are bounded: a word that has not
// come after kWordPolls polls raises the error word, which the other waits
// look at every kWordErrPoll polls.
#pragma once

#include "common.cuh"

namespace tl {

constexpr int kWordPolls = 1 << 22;    // each at least one L2 round trip: seconds
constexpr int kWordErrPoll = 1 << 10;

struct alignas(16) TagWord {
    double value;
    unsigned long long tag;
};

__device__ __forceinline__ void word_store(TagWord* s, double v, unsigned long long tag)
{
    asm volatile(
        "{\n"
        ".reg .b128 q;\n"
        "mov.b128 q, {%1, %2};\n"
        "st.relaxed.gpu.global.b128 [%0], q;\n"
        "}\n" ::"l"(s), "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}

__device__ __forceinline__ bool word_load(const TagWord* s, unsigned long long tag, double& v)
{
    unsigned long long lo, hi;
    asm volatile(
        "{\n"
        ".reg .b128 q;\n"
        "ld.relaxed.gpu.global.b128 q, [%2];\n"
        "mov.b128 {%0, %1}, q;\n"
        "}\n"
        : "=l"(lo), "=l"(hi)
        : "l"(s)
        : "memory");
    v = __longlong_as_double((long long)lo);
    return hi == tag;
}

// Waits for the word; sets *bad when the wait gave up (err raised).
static __device__ __noinline__ double word_wait(const TagWord* s, unsigned long long tag, int* err, int* bad)
{
    double v = 0.0;
    for (int n = 0; n < kWordPolls; ++n) {
        if (word_load(s, tag, v)) return v;
        if ((n & (kWordErrPoll - 1)) == kWordErrPoll - 1 && *(volatile int*)err) break;
    }
    *(volatile int*)err = 1;
    *bad = 1;
    return v;
}

// Shared memory of strip_sum for up to NV sums at once; `bad` starts at 0.
constexpr int kStripMax = 1280;   // strips of a mesh: 10 per thread of the final pass
template <int NV>
struct StripSumSmem {
    double vals[NV][kStripMax];
    short strip_of[3 * 512];   // the strip whose sums each word holds (negative: none)
    double warp[NV][2][16];    // warp sums of this block's strips
    double fin[NV][4];         // warp sums of the final pass
    double out[NV + 1];
    int bad;
};

// NV sums over the whole grid of the strips' values. A group of 128 threads
// (one of up to four in the block) holds values v[.][h] per thread for each
// of two strips and hands their sums over in words 2 pair and 2 pair + 1 of
// the `words` words of each sum (pair negative: the group has none);
// sm.strip_of says which strip each word belongs to, of at most three words
// per thread of a block. The same tree as tl::grid_sum<NV, 128> over blocks of
// 128 threads, bit for bit: warp shuffles, the four warps as (0 + 2) + (1 +
// 3), then thread t < 128 adds the sums of strips t, t + 128, ... in turn and
// the 128 results go through the same tree. `between` runs after the block's
// words are stored, before the wait. `scalar(totals)` runs in four warps;
// every thread gets the totals and its value. False when a wait gave up.
template <int NV, int NS, typename Between, typename Scalar_>
__device__ __forceinline__ bool strip_sum(double (&v)[NV][2], int pair, int strips, int words, StripSumSmem<NS>& sm,
                                          TagWord* slots, unsigned long long tag, int* err, Between between,
                                          Scalar_ scalar, double (&total)[NV], double& derived)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            v[n][0] += __shfl_down_sync(0xffffffffu, v[n][0], o);
            v[n][1] += __shfl_down_sync(0xffffffffu, v[n][1], o);
        }
    if (lane == 0)
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            sm.warp[n][0][warp] = v[n][0];
            sm.warp[n][1][warp] = v[n][1];
        }
    __syncthreads();
    if ((tid & 127) < 2 * NV && pair >= 0) {   // the first threads of each group publish its strips
        const int h = tid & 1, n = (tid & 127) >> 1;
        const double* q = sm.warp[n][h] + (tid >> 7) * 4;
        word_store(slots + n * words + 2 * pair + h, (q[0] + q[2]) + (q[1] + q[3]), tag);
    }
    between();
    {   // every word of the grid into shared memory: a first look at all of this thread's, then one by one
        double x[3 * NV];
        int strip_of[3];
        bool got[3 * NV];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            strip_of[m] = sm.strip_of[tid + m * T];
#pragma unroll
            for (int n = 0; n < NV; ++n)
                got[m * NV + n] = strip_of[m] < 0 || word_load(slots + n * words + tid + m * T, tag, x[m * NV + n]);
        }
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int n = 0; n < NV; ++n)
                if (strip_of[m] >= 0) {
                    if (!got[m * NV + n]) x[m * NV + n] = word_wait(slots + n * words + tid + m * T, tag, err, &sm.bad);
                    sm.vals[n][strip_of[m]] = x[m * NV + n];
                }
    }
    __syncthreads();
    if (tid < 128) {
        double t[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            double q[kStripMax / 128];
            t[n] = 0.0;
#pragma unroll
            for (int m = 0; m < kStripMax / 128; ++m) q[m] = tid + m * 128 < strips ? sm.vals[n][tid + m * 128] : 0.0;
#pragma unroll
            for (int m = 0; m < kStripMax / 128; ++m)
                if (tid + m * 128 < strips) t[n] += q[m];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int n = 0; n < NV; ++n) t[n] += __shfl_down_sync(0xffffffffu, t[n], o);
        if (lane == 0)
#pragma unroll
            for (int n = 0; n < NV; ++n) sm.fin[n][warp] = t[n];
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
        for (int n = 0; n < NV; ++n) t[n] = (sm.fin[n][0] + sm.fin[n][2]) + (sm.fin[n][1] + sm.fin[n][3]);
        const double d = scalar(t);
        if (tid == 0) {
#pragma unroll
            for (int n = 0; n < NV; ++n) sm.out[n] = t[n];
            sm.out[NV] = d;
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NV; ++n) total[n] = sm.out[n];
    derived = sm.out[NV];
    return sm.bad == 0;
}

}  // namespace tl
