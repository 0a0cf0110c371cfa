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
// come after a number of polls raises the error word, which the other waits
// look at every kWordErrPoll polls. A block in which a wait gave up leaves the
// loop as one, at the end of the sum it is in (StripSumSmem::ok): its threads
// meet at barriers, so none may leave before the others.
#pragma once

#include "common.cuh"

namespace tl {

constexpr int kWordPolls = 1 << 22;    // default limit: each at least one L2 round trip, so seconds
constexpr int kWordErrPoll = 1 << 10;  // (a power of two)

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

// What the waits of a block share. They look at it, and at the error word, after
// every kWordErrPoll polls only (a shorter limit starts the count late): a limit
// looked at after every poll, here or as an argument of the call, took 3 to 5 %
// of the preconditioned loop at 1013 x 777 (23.1 to 24.0 ms a timestep).
struct WordWaits {
    int* err;    // device word raised by the waits that give up
    int polls;   // limit of a wait
    int skip;    // polls the count starts at: kWordErrPoll - polls, 0 for a longer limit
    int bad;     // a wait of this block gave up
};

// Waits for the word; sets waits->bad when the wait gave up (*waits->err raised).
static __device__ __noinline__ double word_wait(const TagWord* s, unsigned long long tag, WordWaits* waits)
{
    double v = 0.0;
    int n = waits->skip;
    do {
        if (word_load(s, tag, v)) return v;
        if ((n & (kWordErrPoll - 1)) == kWordErrPoll - 1 && (*(volatile int*)waits->err || n >= waits->polls)) break;
    } while (++n < kWordPolls);
    *(volatile int*)waits->err = 1;
    waits->bad = 1;
    return v;
}

// Shared memory of strip_sum for up to NV sums of up to NH strips at once.
constexpr int kStripMax = 1280;   // strips of a mesh
// Words a group of NH strips has per sum: whole sectors.
constexpr int strip_words(int nh) { return (nh + 1) / 2 * 2; }
template <int NH, int NV>
struct StripSumSmem {
    double vals[NV][kStripMax];
    short strip_of[3 * 512];   // the strip whose sums each word holds (negative: none)
    double warp[NV][NH][16];   // warp sums of this block's strips
    double fin[NV][8];         // warp sums of the final pass
    double out[NV + 1];
    WordWaits waits;           // set before the first wait
    int ok;                    // as the last sum found it: the same for every thread
};

// The values of NT / 32 warps in the order of tl::block_sum's second stage.
template <int NT>
__device__ __forceinline__ double warps_sum(const double* q)
{
    static_assert(NT == 128 || NT == 256, "four or eight warps");
    if (NT == 128) return (q[0] + q[2]) + (q[1] + q[3]);
    return ((q[0] + q[4]) + (q[2] + q[6])) + ((q[1] + q[5]) + (q[3] + q[7]));
}

// NV sums over the whole grid of the strips' values. A group of NT threads
// (blocks have up to 512) holds values v[.][h] per thread for each of NH
// strips and hands their sums over in the first of words strip_words(NH) unit
// .. of the `words` words of each sum (unit, the group's number in the grid;
// negative: it has no strips); sm.strip_of says which strip each word belongs to, of at
// most three words per thread of a block. The same tree as tl::grid_sum<NV,
// NT> over blocks of NT threads, bit for bit: warp shuffles, the block's warps,
// then thread t < NT adds the sums of strips t, t + NT, ... in turn and the NT
// results go through the same tree. `between` runs after the block's words
// are stored, before the wait. `scalar(totals)` runs in NT threads; every
// thread gets the totals and its value. False, in every thread of the block, when a
// wait of the block gave up in this sum or before it.
template <int NT, int NH, int NV, int NS, typename Between, typename Scalar_>
__device__ __forceinline__ bool strip_sum(double (&v)[NV][NH], int unit, int strips, int words,
                                          StripSumSmem<NH, NS>& sm, TagWord* slots, unsigned long long tag,
                                          Between between, Scalar_ scalar, double (&total)[NV], double& derived)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, T = blockDim.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
            for (int h = 0; h < NH; ++h) v[n][h] += __shfl_down_sync(0xffffffffu, v[n][h], o);
    if (lane == 0)
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
            for (int h = 0; h < NH; ++h) sm.warp[n][h][warp] = v[n][h];
    __syncthreads();
    if ((tid & (NT - 1)) < NH * NV && unit >= 0) {   // the first threads of each group publish its strips
        const int h = (tid & (NT - 1)) % NH, n = (tid & (NT - 1)) / NH;
        word_store(slots + n * words + strip_words(NH) * unit + h, warps_sum<NT>(sm.warp[n][h] + tid / NT * (NT / 32)), tag);
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
                    if (!got[m * NV + n])
                        x[m * NV + n] = word_wait(slots + n * words + tid + m * T, tag, &sm.waits);
                    sm.vals[n][strip_of[m]] = x[m * NV + n];
                }
    }
    __syncthreads();
    if (tid < NT) {
        constexpr int per = kStripMax / NT;
        double t[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            double q[per];
            t[n] = 0.0;
#pragma unroll
            for (int m = 0; m < per; ++m) q[m] = tid + m * NT < strips ? sm.vals[n][tid + m * NT] : 0.0;
#pragma unroll
            for (int m = 0; m < per; ++m)
                if (tid + m * NT < strips) t[n] += q[m];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int n = 0; n < NV; ++n) t[n] += __shfl_down_sync(0xffffffffu, t[n], o);
        if (lane == 0)
#pragma unroll
            for (int n = 0; n < NV; ++n) sm.fin[n][warp] = t[n];
        asm volatile("bar.sync 1, %0;\n" ::"n"(NT) : "memory");
#pragma unroll
        for (int n = 0; n < NV; ++n) t[n] = warps_sum<NT>(sm.fin[n]);
        const double d = scalar(t);
        if (tid == 0) {
#pragma unroll
            for (int n = 0; n < NV; ++n) sm.out[n] = t[n];
            sm.out[NV] = d;
            sm.ok = sm.waits.bad == 0;
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NV; ++n) total[n] = sm.out[n];
    derived = sm.out[NV];
    return sm.ok != 0;   // (not waits.bad, which a thread already past this sum may set)
}

}  // namespace tl
