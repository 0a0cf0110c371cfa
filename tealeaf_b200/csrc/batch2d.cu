// batch2d.cu -- many independent 2D timesteps in one persistent launch.
//
// A batch holds `count` initialised chunks of different sizes (each with its
// own tea.in settings). One batched timestep runs, for every problem, the
// reference's solve() (2d/diffuse.c:22-80) with the CG solve replaced by the
// refinement CG of refine2d.cuh (FP32 vectors and coefficients, FP32
// arithmetic in the sweeps, FP64 dot products, scalars and solution, FP64
// residual replacement) stopped
// when the FP64 residual satisfies the problem's own r.r < eps:
//
//   per problem: energy/density halos, cg_init, u0 = u, T-layout setup
//   ONE persistent cooperative kernel: the CG iterations of all problems
//   per problem: energy = u / density, energy halo
//
// captured once into a CUDA graph and replayed for every timestep.
//
// The persistent kernel starts every problem with its own group of blocks,
// sized by the problem's estimated work (cells x (nx + ny), CG's iteration
// count growing with the grid's side) and at least one block. Each problem
// walks its phases -- w = A p, then the u/r update, then (when the problem
// asked for one) the FP64 fold and residual -- with its tiles handed out by
// an atomic counter per problem; a block whose problem has no tile left in
// its open phase takes one from the problem with the most tiles left, so no
// block idles at a problem's phase boundary while other problems have work,
// and the largest problems get the whole grid once the small ones have
// converged. A block holds at most one tile and never waits while holding
// it; only a block that finds no tile anywhere polls, bounded by a clock
// limit (a timeout sets an error word and the blocks return). Taking a tile
// costs two L2 round trips: one load that brings every schedule and its
// scalar, one atomic that hands out the tile and says of which phase (a poll,
// a draw, a fence and three loads were 5500 cycles; closing a phase 7700,
// 5500 with the scalars fetched beside the partials). Per-problem
// dot products are reduced deterministically: each tile writes its block
// sum, and the block finishing the problem's last tile of the phase sums
// the problem's tile partials in tile order and runs the CG scalar update
// (alpha, beta, replacement and stop decisions) for it, then opens the
// problem's next phase.
//
// tile_rows (and the persistent grid size the groups share) come from the
// autotuner (tl2d_batch_tune): it times a few iterations of the real batch
// with each candidate and keeps the fastest.
#include "refine2d.cuh"
#include "suite2d_impl.hpp"

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

using namespace tl2d;
using namespace tl2d::rf;

namespace {

// Arithmetic of the batch's FP32 sweeps (dot products and scalars are FP64
// either way): FP32 (TL2D_BATCH_MATH_F32 1; with plain loads 785 against 846 ms for the
// 64-problem step, the same iterations) or FP64 on the FP32 values (0).
#ifndef TL2D_BATCH_MATH_F32
#define TL2D_BATCH_MATH_F32 1
#endif
using BatchM = std::conditional_t<TL2D_BATCH_MATH_F32 != 0, float, double>;

// The persistent kernel's two forms. A batch whose FP32 arrays fit L2 is bound
// by the latency of a phase -- a tile's rows, its dot product, the next phase's
// opening, twice an iteration -- and runs best with few blocks per SM, each with
// many registers and rows in flight; one that streams from HBM wants as many
// rows in flight per SM as shared memory holds. One step, 4 x 8 against 6 x 6
// (blocks per SM x rows): 24 problems of sides 64-768 (66 MB of arrays) 25.5
// against 28.3 ms, 64-1100 (90 MB) 39.3 / 42.2; 128-1400 (190 MB) 90.8 / 87.8,
// 200 of 64-400 (180 MB) 40.3 / 36.5, the 64 of 128-2048 (900 MB) 620 / 579;
// 8 x 6, with 64 registers a thread: 30.0, 49.8, 97.8, 36.1, 582.
struct Resident { static constexpr int MINB = 4, STAGES = 8; };
struct Streaming { static constexpr int MINB = 6, STAGES = 6; };
constexpr int kGroupsPerSm = 8;                  // blocks per SM that the problems' groups are cut for
constexpr long long kWaitLimit = 4000000000LL;   // default: SM clocks a phase wait may take (~2 s)

enum { BF_KX = 0, BF_KY, BF_P0, BF_P1, BF_W, BF_R, BF_XS, BF_COUNT };

struct BProb {
    Lay L;
    int tx, ty;      // tiles per row / column
    int tile0;       // first global tile of this problem
    int gx, hd;      // FP64 chunk arrays: row length, halo depth
    float* f[BF_COUNT];
    double* u;
    const double* u0;
    const double* kx;
    const double* ky;
};

struct BCtl {
    int err;          // a block found no tile to work on for longer than the limit
    int iters;        // most iterations any problem ran
    long long limit;  // SM clocks a block may go without a tile before it gives up (kept across steps)
};

// Per-problem schedule of the persistent kernel: the open phase (iteration and
// kind, high half of `word`), the tiles left to hand out in it (low half, above
// kNone) and the phase's scalar. A block takes a tile with one atomic
// subtraction and holds tile (left - 1) of that phase exactly when `left` was
// above kNone; what the phase is comes back with it. The block completing the
// phase's last tile runs the phase's scalar update, writes the next phase's
// scalar and opens it by swapping in its word; a finished problem has kind
// PH_DONE and no tiles. A block never waits while it holds a tile: when its
// problem has no tile left in the open phase it takes one from the problem with
// the most tiles left, and only when no problem has one does it poll (bounded by
// the clock limit). A schedule has a 128-byte line to itself: polls of one and
// draws from another would serialise on a shared line.
enum { PH_W = 0, PH_UR = 1, PH_FOLD = 2, PH_RESID = 3, PH_DONE = 4 };
constexpr unsigned kNone = 0x40000000u;   // failed draws take the low half below it
struct alignas(128) PCtl {
    double coef;               // beta (PH_W) or alpha (PH_UR) of the open phase
    unsigned long long word;   // (iteration << 3 | kind) << 32 | kNone + tiles left
};
__device__ __forceinline__ unsigned long long phase_word(int it, int kind, int tiles)
{
    return (unsigned long long)((unsigned)it << 3 | (unsigned)kind) << 32 | (kNone + (unsigned)(kind == PH_DONE ? 0 : tiles));
}
__device__ __forceinline__ int tiles_left(unsigned long long word) { return (int)((unsigned)word - kNone); }
__device__ __forceinline__ unsigned phase_of(unsigned long long word) { return (unsigned)(word >> 32); }

// The scalar and the word of a schedule in one 16-byte load. A draw that then
// finds the same phase open may use the scalar: the next phase's is written
// only once every tile of this one has been handed out and completed.
__device__ __forceinline__ unsigned long long sched_load(const PCtl* s, double& coef)
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
    coef = __longlong_as_double((long long)lo);
    return hi;
}
// What the phase's opener published is visible after the draw.
__device__ __forceinline__ unsigned long long sched_draw(PCtl* s)
{
    unsigned long long old;
    asm volatile("atom.add.acquire.gpu.global.u64 %0, [%1], %2;" : "=l"(old) : "l"(&s->word), "l"(~0ull) : "memory");
    return old;
}
__device__ __forceinline__ void sched_open(PCtl* s, double coef, unsigned long long word)
{
    unsigned long long old;
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(&s->coef), "d"(coef) : "memory");
    asm volatile("atom.exch.release.gpu.global.b64 %0, [%1], %2;" : "=l"(old) : "l"(&s->word), "l"(word) : "memory");
}

// Rows of a tile on their way from L2 to shared memory: every thread holds two
// cells of up to four arrays a row; of a pair of lanes the even one copies the
// pair's 16 bytes of the first two arrays, the odd one those of the other two,
// so a warp waits for its own copies only. Plain loads waited for L2 row by row
// (16-row tiles: 18200 cycles for the w sweep, 10500 for the u/r update) because
// a row's stores, which might alias, hold back the next row's loads; the copies
// need no registers and are issued STAGES rows ahead (7200 and 4000 cycles on a
// quiet SM).
struct alignas(128) RingRow {
    float2 cell[4][BX];         // [array][thread]
    float4 edge[3][BX / 16];    // [array][2 * warp + side]: the columns beside a warp's
};

__device__ __forceinline__ unsigned ring_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ring_copy(unsigned to, const float* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to), "l"(from) : "memory");
}
__device__ __forceinline__ Cells<float> ring_read(unsigned at)
{
    Cells<float> c;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(c.e[0]), "=f"(c.e[1]) : "r"(at) : "memory");
    return c;
}
__device__ __forceinline__ float ring_read1(unsigned at)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
// Rows are waited for two at a time; each pair commits one group, an empty one
// past the tile's end, so that a pair has arrived once at most ST / 2 - 1 groups
// are pending.
__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int ST>
__device__ __forceinline__ void ring_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(ST / 2 - 1) : "memory");
    __syncwarp();
}
constexpr unsigned kRow = sizeof(RingRow), kArr = sizeof(float2) * BX, kEdgeArr = sizeof(float4) * (BX / 16);
template <int ST>
__device__ __forceinline__ unsigned ring_after(unsigned slot)   // slot: byte offset of a pair of rows
{
    return slot == (ST - 2) * kRow ? 0u : slot + 2 * kRow;
}

// CG sweep 1 over tile (tx, ty): [p = bt p + r], w = A p; returns this thread's
// share of sum(w p). The arithmetic and its order are rf_w_tile's.
template <int ST, bool FUSE_P>
__device__ __forceinline__ double batch_w_tile(RingRow* R, const Lay& L, int tx, int ty, double bt_,
                                               const float* __restrict__ p_in, float* __restrict__ p_out,
                                               const float* __restrict__ r, float* __restrict__ w,
                                               const float* __restrict__ kx, const float* __restrict__ ky)
{
    using M = BatchM;
    constexpr int N = Pack<float>::N;
    const Span<N> s(L, tx, ty);
    const M bt = (M)bt_;
    const unsigned xp = (unsigned)L.xp;
    const int rows = s.j1 - s.j0;
    const bool first = s.lane == 0, final = s.lane == 31, odd = s.lane & 1, end = first || final;
    const bool in0 = s.c0 < L.nx, in1 = s.c0 + 1 < L.nx;
    const int c4 = min(s.c0 & ~3, L.xp - 4);   // the pair's four columns
    const int pair = threadIdx.x & ~1;
    const unsigned to = ring_addr(&R[0].cell[odd ? 2 : 0][pair]);
    const unsigned me = ring_addr(&R[0].cell[0][pair + ((s.cc - c4) >> 1)]);
    const unsigned ed = ring_addr(&R[0].edge[0][2 * (threadIdx.x >> 5) + (final ? 1 : 0)]);
    const unsigned near = ed + (final ? 0u : 12u);   // of the edge's four columns, the neighbour
    // row k of rows + 2: p, r (and ky from the tile's own first row on) of row
    // j0 - 1 + k, kx of the row before it, which is the one the operator is at
    const float* const one = (odd ? ky : p_in) + c4;
    const float* const two = (odd ? kx : r) + c4;
    const float* const pe_in = p_in + c4 + (final ? 4 : -4);
    const float* const re_in = r + c4 + (final ? 4 : -4);
    const float* const ke_in = kx + c4 + 4;
    unsigned g = (unsigned)s.j0 * xp;   // of the next row to fill
    int k = 0;
    auto fill = [&](unsigned at) {
        if (k < rows + 2) {
            if (!odd || k > 0) ring_copy(to + at, one + g);
            if (odd) {
                if (k > 1) ring_copy(to + at + kArr, two + (g - xp));
            } else if (FUSE_P) {
                ring_copy(to + at + kArr, two + g);
            }
            if (end) {
                if (k > 0 && k <= rows) {   // the tile's own rows only
                    ring_copy(ed + at, pe_in + g);
                    if (FUSE_P) ring_copy(ed + at + kEdgeArr, re_in + g);
                }
                if (final && k > 1) ring_copy(ed + at + 2 * kEdgeArr, ke_in + (g - xp));
            }
        }
        ++k;
        g += xp;
    };
    auto fill2 = [&](unsigned at) {
        fill(at);
        fill(at + kRow);
        ring_commit();
    };
    struct Row {
        Cells<float> p, q, ky, kx;
        float pe, qe, ke;
    };
    auto read = [&](unsigned at, Row& v) {
        v.p = ring_read(me + at);
        if (FUSE_P) v.q = ring_read(me + at + kArr);
        v.ky = ring_read(me + at + 2 * kArr);
        v.kx = ring_read(me + at + 3 * kArr);
        v.pe = v.qe = v.ke = 0.f;
        if (end) {
            v.pe = ring_read1(near + at);
            if (FUSE_P) v.qe = ring_read1(near + at + kEdgeArr);
            v.ke = ring_read1(near + at + 2 * kEdgeArr);
        }
    };
    auto fold = [&](Row& v) {
        if (FUSE_P) {
#pragma unroll
            for (int m = 0; m < N; ++m) v.p.e[m] = (float)(bt * (M)v.p.e[m] + (M)v.q.e[m]);
            v.pe = (float)(bt * (M)v.pe + (M)v.qe);
        }
    };
    unsigned slot = 0;
#pragma unroll
    for (int c = 0; c < ST; c += 2) fill2(c * kRow);
    double acc = 0.0;
    Cells<float> pd{}, pc{}, kyc{};
    float pe = 0.f;
    unsigned i = ((unsigned)s.j0 + 1) * xp + s.cc;
    auto step = [&](const Row& v) {   // the operator at (pc, kyc, pe), v the row above
        float pl = __shfl_up_sync(kFull, pc.e[N - 1], 1);
        float pr = __shfl_down_sync(kFull, pc.e[0], 1);
        float kxr = __shfl_down_sync(kFull, v.kx.e[0], 1);
        if (first) pl = pe;
        if (final) {
            pr = pe;
            kxr = v.ke;
        }
        Cells<float> wv;
#pragma unroll
        for (int m = 0; m < N; ++m) {
            const M c = (M)pc.e[m];
            const M l = m == 0 ? (M)pl : (M)pc.e[m - 1];
            const M rr = m == N - 1 ? (M)pr : (M)pc.e[m + 1];
            const M kr = m == N - 1 ? (M)kxr : (M)v.kx.e[m + 1];
            wv.e[m] = (float)smvp_m<M>((M)v.kx.e[m], kr, (M)kyc.e[m], (M)v.ky.e[m], c, l, rr, (M)pd.e[m],
                                       (M)v.p.e[m]);
        }
        if (s.any) {
            st8(w + i, wv);
            if (FUSE_P) st8(p_out + i, pc);
        }
        if (in0) acc += (double)wv.e[0] * (double)pc.e[0];
        if (in1) acc += (double)wv.e[1] * (double)pc.e[1];
        pd = pc;
        pc = v.p;
        kyc = v.ky;
        pe = v.pe;
        i += xp;
    };
    Row a, b;
    auto take2 = [&]() {
        ring_wait<ST>();
        read(slot, a);
        read(slot + kRow, b);
        __syncwarp();
        fill2(slot);
        slot = ring_after<ST>(slot);
        fold(a);
        fold(b);
    };
    take2();
    pd = a.p;
    pc = b.p;
    kyc = b.ky;
    pe = b.pe;
    for (int j = 0; j < rows; j += 2) {
        take2();
        step(a);
        if (j + 1 < rows) step(b);
    }
    return acc;
}

// CG sweep 2 over tile (tx, ty): xs += a p, r -= a w; returns this thread's
// share of sum(r r). The arithmetic and its order are rf_ur_tile's.
template <int ST>
__device__ __forceinline__ double batch_ur_tile(RingRow* R, const Lay& L, int tx, int ty, double a_,
                                                float* __restrict__ xs, const float* __restrict__ p,
                                                float* __restrict__ r, const float* __restrict__ w)
{
    using M = BatchM;
    constexpr int N = Pack<float>::N;
    const Span<N> s(L, tx, ty);
    if (!__any_sync(kFull, s.any)) return 0.0;
    const M al = (M)a_;
    const unsigned xp = (unsigned)L.xp;
    const int rows = s.j1 - s.j0;
    const bool odd = s.lane & 1, in0 = s.c0 < L.nx, in1 = s.c0 + 1 < L.nx;
    const int pair = threadIdx.x & ~1;
    const int c4 = min(s.c0 & ~3, L.xp - 4);
    const unsigned to = ring_addr(&R[0].cell[odd ? 2 : 0][pair]);
    const unsigned me = ring_addr(&R[0].cell[0][pair + ((s.cc - c4) >> 1)]);
    const float* const one = (odd ? p : xs) + c4;
    const float* const two = (odd ? w : r) + c4;
    unsigned g = ((unsigned)s.j0 + 1) * xp, i = g + s.cc;
    int k = 0;
    auto fill2 = [&](unsigned at) {
#pragma unroll
        for (int q = 0; q < 2; ++q, ++k, g += xp)
            if (k < rows) {
                ring_copy(to + at + q * kRow, one + g);
                ring_copy(to + at + q * kRow + kArr, two + g);
            }
        ring_commit();
    };
#pragma unroll
    for (int c = 0; c < ST; c += 2) fill2(c * kRow);
    double acc = 0.0;
    unsigned slot = 0;
    struct Row {
        Cells<float> xs, r, p, w;
    };
    auto read = [&](unsigned at, Row& v) {
        v.xs = ring_read(me + at);
        v.r = ring_read(me + at + kArr);
        v.p = ring_read(me + at + 2 * kArr);
        v.w = ring_read(me + at + 3 * kArr);
    };
    auto step = [&](Row& v) {
#pragma unroll
        for (int m = 0; m < N; ++m) {
            v.xs.e[m] = (float)((M)v.xs.e[m] + al * (M)v.p.e[m]);
            v.r.e[m] = (float)((M)v.r.e[m] - al * (M)v.w.e[m]);
        }
        if (s.any) {
            st8(xs + i, v.xs);
            st8(r + i, v.r);
        }
        if (in0) acc += (double)v.r.e[0] * (double)v.r.e[0];
        if (in1) acc += (double)v.r.e[1] * (double)v.r.e[1];
        i += xp;
    };
    for (int j = 0; j < rows; j += 2) {
        Row a, b;
        ring_wait<ST>();
        read(slot, a);
        read(slot + kRow, b);
        __syncwarp();
        fill2(slot);
        slot = ring_after<ST>(slot);
        step(a);
        if (j + 1 < rows) step(b);
    }
    return acc;
}

// Block sum of this thread's values; returns true in every thread of the
// block that completed the problem's last tile of the phase, with the
// problem's totals (fixed-order sum of its tile partials) in tot (thread 0)
// and its scalars in cp, fetched beside the partials.
template <int N>
__device__ bool tile_done(double (&v)[N], int t, const BProb& P, unsigned* ticket, double* partials,
                          const MxState* st, MxState& cp, double (&tot)[N])
{
    constexpr int kWords = sizeof(MxState) / sizeof(double);
    static_assert(sizeof(MxState) % sizeof(double) == 0 && kWords <= BX, "one word per thread");
    __shared__ double smem[N][BX / tl::kWarp];
    __shared__ bool last;
    const int nt = P.tx * P.ty;
    __syncthreads();
    tl::block_sum<N, BX>(v, smem);
    if (threadIdx.x == 0) {
        unsigned before;
#pragma unroll
        for (int r = 0; r < N; ++r) partials[(long)t * 2 + r] = v[r];
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(ticket) : "memory");
        last = before == (unsigned)(nt - 1);
    }
    __syncthreads();
    if (!last) return false;
    if (threadIdx.x < kWords) ((double*)&cp)[threadIdx.x] = __ldcg((const double*)st + threadIdx.x);
    double s[N];
#pragma unroll
    for (int r = 0; r < N; ++r) s[r] = 0.0;
    // partials k = tid, tid + BX, ... added in that order; four loads in flight
    for (int k0 = threadIdx.x; k0 < nt; k0 += 4 * BX) {
        double q[4][N];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int r = 0; r < N; ++r)
                q[u][r] = k0 + u * BX < nt ? __ldcg(&partials[(long)(P.tile0 + k0 + u * BX) * 2 + r]) : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + u * BX < nt)
#pragma unroll
                for (int r = 0; r < N; ++r) s[r] += q[u][r];
    }
    __syncthreads();
    tl::block_sum<N, BX>(s, smem);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int r = 0; r < N; ++r) tot[r] = s[r];
        *ticket = 0u;
    }
    return true;
}

// Warp 0: draws a tile of problem b, or, when it has none left in its open
// phase, of the problem with the most tiles left. 1 with b, t, phase and coef
// set; 0 when no problem has a tile right now; -1 when every problem has
// finished. The first 32 problems looked at, b among them, cost one round trip.
__device__ __forceinline__ int find_tile(PCtl* pc, int np, int& b, int& t, unsigned& phase, double& coef)
{
    constexpr int kOwn = 0x3fffffff;
    const int lane = threadIdx.x & 31;
    int best = 0, who = -1;
    unsigned seen = 0;
    double c = 0.0;
    bool live = false;
    for (int k0 = 0; k0 < np; k0 += 32) {
        const int k = k0 + lane, q = b + k < np ? b + k : b + k - np;
        if (k < np) {
            double cq;
            const unsigned long long word = sched_load(&pc[q], cq);
            live |= (phase_of(word) & 7u) != PH_DONE;
            int left = tiles_left(word);
            if (left > 0 && k == 0) left = kOwn;   // its own problem first
            if (left > best) {
                best = left;
                who = q;
                seen = phase_of(word);
                c = cq;
            }
        }
        if (__any_sync(0xffffffffu, best == kOwn)) break;
    }
    if (!__any_sync(0xffffffffu, live)) return -1;
    const int most = __reduce_max_sync(0xffffffffu, best);
    if (most <= 0) return 0;
    const int from = __ffs(__ballot_sync(0xffffffffu, best == most)) - 1;
    int got = 0;
    if (lane == from) {
        const unsigned long long word = sched_draw(&pc[who]);
        t = tiles_left(word) - 1;
        phase = phase_of(word);
        got = t >= 0;
        coef = c;
        if (got && phase != seen) sched_load(&pc[who], coef);
    }
    got = __shfl_sync(0xffffffffu, got, from);
    if (got) {
        b = __shfl_sync(0xffffffffu, who, from);
        t = __shfl_sync(0xffffffffu, t, from);
        phase = __shfl_sync(0xffffffffu, phase, from);
        coef = __shfl_sync(0xffffffffu, coef, from);
    }
    return got;
}

// K: Resident or Streaming.
template <typename K>
__global__ void __launch_bounds__(BX, K::MINB) k_batch_cg(const BProb* __restrict__ P, int np,
                                                          const int* __restrict__ block_prob, MxState* st,
                                                          unsigned* tickets, double* partials, PCtl* pc,
                                                          BCtl* ctl, int max_iters)
{
    // 128-byte lines: the copies of a warp take a third longer across them
    extern __shared__ __align__(128) unsigned char ring_bytes[];
    RingRow* const ring = reinterpret_cast<RingRow*>(ring_bytes);
    __shared__ int sh_go, sh_b, sh_t;
    __shared__ unsigned sh_phase;
    __shared__ double sh_coef;
    __shared__ BProb Q;       // the problem of the block's tile
    __shared__ MxState cp;
    int b = block_prob[blockIdx.x], have = -1;
    const long long limit = ctl->limit;
    long long idle0 = clock64();
    for (;;) {
        if (threadIdx.x < 32) {
            int t = 0;
            unsigned phase = 0;
            double coef = 0.0;
            const int err = vol_read(&ctl->err);   // under way beside the schedules
            int go = find_tile(pc, np, b, t, phase, coef);
            if (go == 1) {
                idle0 = clock64();
            } else if (go == 0) {
                if (err) {
                    go = -1;
                } else if (clock64() - idle0 > limit) {
                    if (threadIdx.x == 0) atomicExch(&ctl->err, 1);
                    go = -1;
                } else {
                    __nanosleep(64);
                }
                go = __shfl_sync(0xffffffffu, go, 0);
            }
            if (threadIdx.x == 0) {
                sh_go = go;
                sh_b = b;
                sh_t = t;
                sh_phase = phase;
                sh_coef = coef;
            }
        }
        __syncthreads();
        const int go = sh_go, lt = sh_t, kind = sh_phase & 7u, it = sh_phase >> 3;
        const double coef = sh_coef;
        b = sh_b;
        if (go == 1 && b != have) {
            static_assert(sizeof(BProb) % sizeof(int) == 0 && sizeof(BProb) / sizeof(int) <= BX, "one word per thread");
            if (threadIdx.x < sizeof(BProb) / sizeof(int)) ((int*)&Q)[threadIdx.x] = ((const int*)&P[b])[threadIdx.x];
            have = b;
        }
        __syncthreads();   // sh_* are rewritten by the next pass
        if (go < 0) return;
        if (go == 0) continue;
        const int tx = lt % Q.tx, ty = lt / Q.tx;
        double v[2] = {0.0, 0.0};
        if (kind == PH_W) {
            float* pin = Q.f[it == 0 ? BF_P0 : (((it - 1) & 1) ? BF_P1 : BF_P0)];
            float* pout = Q.f[(it & 1) ? BF_P1 : BF_P0];
            v[0] = it == 0 ? batch_w_tile<K::STAGES, false>(ring, Q.L, tx, ty, 0.0, pin, pin, Q.f[BF_R], Q.f[BF_W],
                                                  Q.f[BF_KX], Q.f[BF_KY])
                           : batch_w_tile<K::STAGES, true>(ring, Q.L, tx, ty, coef, pin, pout, Q.f[BF_R], Q.f[BF_W],
                                                 Q.f[BF_KX], Q.f[BF_KY]);
        } else if (kind == PH_UR) {
            v[0] = batch_ur_tile<K::STAGES>(ring, Q.L, tx, ty, coef, Q.f[BF_XS], Q.f[(it & 1) ? BF_P1 : BF_P0], Q.f[BF_R],
                                 Q.f[BF_W]);
        } else if (kind == PH_FOLD) {
            rf_fold_tile<float>(Q.L, tx, ty, Q.gx, Q.hd, Q.u, Q.f[BF_XS]);
        } else {
            rf_resid_tile<float>(Q.L, tx, ty, Q.gx, Q.hd, Q.u, Q.u0, Q.kx, Q.ky, Q.f[BF_R], v);
        }
        double tot[2];
        if (tile_done<2>(v, Q.tile0 + lt, Q, &tickets[b], partials, &st[b], cp, tot) && threadIdx.x == 0) {
            // the phase is complete: its scalar update, then open the next phase
            int next = PH_W, nit = it;
            if (kind == PH_W) {
                FinMxW{&cp}(tot);
                next = PH_UR;
            } else if (kind == PH_UR) {
                FinMxUr{&cp}(tot);
                if (cp.upd) next = PH_FOLD;
                else nit = it + 1;
            } else if (kind == PH_FOLD) {
                next = PH_RESID;
            } else {
                FinMxRes{&cp, nullptr}(tot);
                nit = it + 1;
                if (cp.done) next = PH_DONE;
            }
            if (next == PH_W && nit >= max_iters) next = PH_DONE;
            if (next == PH_DONE) atomicMax(&ctl->iters, nit);
            st[b] = cp;
            sched_open(&pc[b], next == PH_W ? cp.beta : cp.alpha, phase_word(nit, next, Q.tx * Q.ty));
        }
    }
}

// Clears the per-problem tile tickets and schedules (a step that gave up may
// have left them mid-phase) and the step's control words; the clock limit is
// kept. A problem the setup already converged starts closed.
__global__ void k_batch_reset(const BProb* __restrict__ P, const MxState* st, int np, BCtl* ctl, unsigned* tickets,
                              PCtl* pc)
{
    for (int b = threadIdx.x; b < np; b += blockDim.x) {
        const bool done = st[b].done != 0;
        tickets[b] = 0u;
        pc[b].coef = 0.0;
        pc[b].word = phase_word(0, done ? PH_DONE : PH_W, P[b].tx * P[b].ty);
    }
    if (threadIdx.x == 0) {
        ctl->err = 0;
        ctl->iters = 0;
    }
}

}  // namespace

// ------------------------------------------------------------------ batch --

struct TlBatch {
    int count = 0;
    int device = 0;
    int sm_count = 148;
    cudaStream_t stream = nullptr;
    std::vector<Chunk*> chunks;
    std::vector<Settings*> settings;
    std::vector<TlSuite2D*> suites;
    std::vector<Lay> lay;
    void* slab = nullptr;            // FP32 arrays of every problem
    size_t slab_bytes = 0;
    std::vector<size_t> field_off;   // per problem: offset of its first FP32 array
    std::vector<size_t> field_bytes; // per problem: bytes of one FP32 array
    BProb* d_prob = nullptr;
    int* d_block_prob = nullptr;     // problem of every block of the persistent grid
    PCtl* d_pctl = nullptr;          // per-problem schedules
    MxState* d_st = nullptr;
    unsigned* d_tickets = nullptr;
    double* d_partials = nullptr;
    BCtl* d_ctl = nullptr;
    tl::ReduceSlots rs{};
    long rs_capacity = 0;
    DevState* d_scratch_state = nullptr;
    int max_tiles = 0;               // capacity of the tile tables
    int ntiles = 0;
    int tile_rows = 0;
    int grid_blocks = 0;             // blocks the groups share
    int launch_blocks = 0;           // blocks launched: the sum of the group sizes, the co-resident limit at most
    int max_grid = 0;                // most blocks the groups may share
    int resident = 0;                // co-resident blocks of the persistent kernel
    const void* kernel = nullptr;    // its form
    size_t smem = 0;                 // bytes of its row ring
    int max_iters = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bool graph_ok = false;
};

namespace {

void batch_free(TlBatch* B)
{
    if (B->exec) cudaGraphExecDestroy(B->exec);
    if (B->graph) cudaGraphDestroy(B->graph);
    void* ptrs[] = {B->slab, B->d_prob, B->d_block_prob, B->d_pctl, B->d_st, B->d_tickets, B->d_partials, B->d_ctl,
                    B->rs.partials, B->rs.ticket, B->rs.out_dev, B->d_scratch_state};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (B->stream) cudaStreamDestroy(B->stream);
    delete B;
}

// Splits the grid_blocks blocks into one group per problem, in proportion
// to the estimated work cells x (nx + ny) (CG's iteration count grows with
// the grid's side), at least one block and at most one per tile of the
// problem's finest tiling; lays out the tiles for tile_rows and uploads the
// problem and block tables. tile_rows > 0: that height for every problem;
// kAdaptiveRows: per problem the height that gives its group about one tile
// per block per phase (between 2 and 64 rows).
constexpr int kAdaptiveRows = -1;

bool batch_layout(TlBatch* B, int tile_rows)
{
    const int n = B->count;
    std::vector<double> work(n);
    std::vector<long> cap(n);
    double total = 0.0;
    for (int b = 0; b < n; ++b) {
        Lay L = B->lay[b];
        work[b] = (double)L.nx * L.ny * (double)(L.nx + L.ny);
        total += work[b];
        L.rows = tile_rows > 0 ? tile_rows : 2;
        const dim3 t = lay_tiles<float>(L);
        cap[b] = (long)t.x * t.y;
    }
    if (B->grid_blocks < n) {
        tl::fail(62, "batch: %d problems need at least %d blocks, the grid has %d", n, n, B->grid_blocks);
        return false;
    }
    std::vector<int> size(n);
    long used = 0;
    for (int b = 0; b < n; ++b) {
        size[b] = (int)std::min<long>(cap[b], std::max<long>(1, (long)(B->grid_blocks * work[b] / total)));
        used += size[b];
    }
    while (used > B->grid_blocks) {   // the one-block minimum overshot: trim the largest groups
        int k = (int)(std::max_element(size.begin(), size.end()) - size.begin());
        --size[k];
        --used;
    }
    while (used < B->grid_blocks) {   // hand the rest to the most loaded groups per block
        int k = -1;
        double best = 0.0;
        for (int b = 0; b < n; ++b)
            if (size[b] < cap[b] && work[b] / size[b] > best) {
                best = work[b] / size[b];
                k = b;
            }
        if (k < 0) break;
        ++size[k];
        ++used;
    }
    std::vector<BProb> P(n);
    std::vector<int> bp;
    int tiles = 0;
    for (int b = 0; b < n; ++b) {
        Lay L = B->lay[b];
        if (tile_rows == kAdaptiveRows) {
            L.rows = 64;
            const long tx = lay_tiles<float>(L).x;
            L.rows = (int)std::min<long>(64, std::max<long>(2, (L.ny * tx + size[b] - 1) / size[b]));
        } else {
            L.rows = tile_rows;
        }
        B->lay[b] = L;
        const dim3 t = lay_tiles<float>(L);
        BProb& Q = P[b];
        Q.L = L;
        Q.tx = (int)t.x;
        Q.ty = (int)t.y;
        Q.tile0 = tiles;
        tiles += Q.tx * Q.ty;
        bp.insert(bp.end(), std::min(size[b], Q.tx * Q.ty), b);
        Q.gx = B->suites[b]->g.x;
        Q.hd = B->suites[b]->g.hd;
        char* base = (char*)B->slab + B->field_off[b];
        for (int k = 0; k < BF_COUNT; ++k) Q.f[k] = (float*)(base + B->field_bytes[b] * k);
        Chunk* c = B->chunks[b];
        Q.u = c->u;
        Q.u0 = c->u0;
        Q.kx = c->kx;
        Q.ky = c->ky;
    }
    if (tiles > B->max_tiles) {
        tl::fail(62, "batch: %d tiles exceed the table capacity %d", tiles, B->max_tiles);
        return false;
    }
    B->ntiles = tiles;
    B->tile_rows = tile_rows;
    // more group blocks than fit the chip at once: an even selection of them is
    // launched (a problem left without a block of its own is served by those of
    // the others, which take work wherever most is left)
    const size_t want = bp.size();
    if (want > (size_t)B->resident) {
        for (size_t k = 0; k < (size_t)B->resident; ++k) bp[k] = bp[k * want / B->resident];
        bp.resize(B->resident);
    }
    B->launch_blocks = (int)bp.size();
    if (!TL_CUDA(cudaMemcpyAsync(B->d_prob, P.data(), sizeof(BProb) * P.size(), cudaMemcpyHostToDevice, B->stream)))
        return false;
    if (!TL_CUDA(cudaMemcpyAsync(B->d_block_prob, bp.data(), sizeof(int) * bp.size(), cudaMemcpyHostToDevice,
                                 B->stream)))
        return false;
    return TL_CUDA(cudaStreamSynchronize(B->stream));
}

void launch_halos(TlBatch* B, int b, int depth, std::initializer_list<double*> fields)
{
    TlSuite2D* s = B->suites[b];
    Chunk* c = B->chunks[b];
    HaloArgs a{};
    for (double* f : fields) a.f[a.nf++] = f;
    for (int f = 0; f < 4; ++f) a.ext[f] = c->neighbours[f] == TL_EXTERNAL_FACE;
    const long per = (long)depth * (2L * (s->g.y - 2 * s->g.hd) + 2L * (s->g.x - 2 * s->g.hd));
    k_local_halos<<<dim3(tl::ceil_div(per, 256), a.nf), 256, 0, B->stream>>>(s->g, depth, a);
}

// Everything of one batched timestep, issued on B->stream (capturable).
// iter_cap limits the iterations of the persistent kernel; finish = run the
// per-problem finalise (a full timestep) or stop after the solve (tuning).
void issue_step(TlBatch* B, int iter_cap, bool finish)
{
    for (int b = 0; b < B->count; ++b) {
        TlSuite2D* s = B->suites[b];
        Chunk* c = B->chunks[b];
        Settings* st = B->settings[b];
        const double dt = c->dt_init < st->dt_init ? c->dt_init : st->dt_init;
        const double rx = dt / (st->dx * st->dx), ry = dt / (st->dy * st->dy);
        launch_halos(B, b, 2, {c->density, c->energy});
        k_cg_init<<<full_grid(s->g), FB, 0, B->stream>>>(s->g, st->coefficient, rx, ry, c->density, c->energy, c->u,
                                                          c->p, nullptr, nullptr, c->r, c->w, c->kx, c->ky, B->rs,
                                                          FinCgInit{B->d_scratch_state, nullptr});
        k_copy_u<<<interior_grid(s->g), BX, 0, B->stream>>>(s->g, c->u0, c->u);
        char* base = (char*)B->slab + B->field_off[b];
        float* f[BF_COUNT];
        for (int k = 0; k < BF_COUNT; ++k) f[k] = (float*)(base + B->field_bytes[b] * k);
        k_rf_init<float><<<B->sm_count, 256, 0, B->stream>>>(
            s->g.x, s->g.hd, B->lay[b], c->r, c->u0, c->kx, c->ky, f[BF_KX], f[BF_KY], f[BF_R], f[BF_P0], f[BF_P1],
            f[BF_W], f[BF_XS], B->rs, FinMxInit{&B->d_st[b], 0.0, st->eps, st->max_iters, nullptr});
    }
    k_batch_reset<<<1, 128, 0, B->stream>>>(B->d_prob, B->d_st, B->count, B->d_ctl, B->d_tickets, B->d_pctl);
    void* args[] = {&B->d_prob, &B->count, &B->d_block_prob, &B->d_st, &B->d_tickets, &B->d_partials, &B->d_pctl,
                    &B->d_ctl, &iter_cap};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(B->launch_blocks);
    cfg.blockDim = dim3(BX);
    cfg.dynamicSmemBytes = B->smem;
    cfg.stream = B->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelExC(&cfg, B->kernel, args);
    if (!finish) return;
    for (int b = 0; b < B->count; ++b) {
        TlSuite2D* s = B->suites[b];
        Chunk* c = B->chunks[b];
        k_finalise<<<interior_grid(s->g), BX, 0, B->stream>>>(s->g, c->energy, c->density, c->u);
        launch_halos(B, b, 1, {c->energy});
    }
}

bool check_ctl(TlBatch* B, BCtl* out)
{
    BCtl h{};
    if (!TL_CUDA(cudaMemcpyAsync(&h, B->d_ctl, sizeof(BCtl), cudaMemcpyDeviceToHost, B->stream))) return false;
    if (!TL_CUDA(cudaStreamSynchronize(B->stream))) return false;
    if (h.err) {
        tl::fail(63, "batch: a phase wait of the persistent kernel timed out");
        return false;
    }
    if (out) *out = h;
    return true;
}

void drop_graph(TlBatch* B)
{
    if (B->exec) cudaGraphExecDestroy(B->exec);
    if (B->graph) cudaGraphDestroy(B->graph);
    B->exec = nullptr;
    B->graph = nullptr;
    B->graph_ok = false;
}

}  // namespace

extern "C" {

TlBatch* tl2d_batch_create(Chunk** chunks, Settings** settings, int count, int tile_rows, int grid_blocks)
{
    if (tl::failed()) return nullptr;
    if (!chunks || !settings || count < 1) {
        tl::fail(60, "tl2d_batch_create: need count >= 1 chunks and settings");
        return nullptr;
    }
    TlBatch* B = new TlBatch();
    B->count = count;
    TL_CUDA(cudaGetDevice(&B->device));
    TL_CUDA(cudaDeviceGetAttribute(&B->sm_count, cudaDevAttrMultiProcessorCount, B->device));
    if (!TL_CUDA(cudaStreamCreateWithFlags(&B->stream, cudaStreamNonBlocking))) {
        batch_free(B);
        return nullptr;
    }
    long max_full = 1;
    size_t total = 0;
    for (int b = 0; b < count; ++b) {
        TlSuite2D* s = suite_of(chunks[b]);
        if (!s) {
            batch_free(B);
            return nullptr;
        }
        const Faces fc = faces_of(chunks[b]);
        if (settings[b]->num_chunks_per_rank != 1 || !(fc.l && fc.r && fc.b && fc.t) ||
            (settings[b]->coefficient != TL_CONDUCTIVITY && settings[b]->coefficient != TL_RECIP_CONDUCTIVITY)) {
            tl::fail(61, "tl2d_batch_create: problem %d needs one chunk, four external faces, a valid coefficient", b);
            batch_free(B);
            return nullptr;
        }
        TL_CUDA(cudaStreamSynchronize(s->stream));
        B->chunks.push_back(chunks[b]);
        B->settings.push_back(settings[b]);
        B->suites.push_back(s);
        const int nx = s->g.x - 2 * s->g.hd, ny = s->g.y - 2 * s->g.hd;
        B->lay.push_back(make_lay<float>(nx, ny, 2));
        const size_t fbytes = ((size_t)B->lay.back().cells() * sizeof(float) + 255) & ~(size_t)255;
        B->field_off.push_back(total);
        B->field_bytes.push_back(fbytes);
        total += fbytes * BF_COUNT;
        const dim3 gf = full_grid(s->g);
        max_full = std::max<long>(max_full, (long)gf.x * gf.y);
        B->max_iters = std::max(B->max_iters, settings[b]->max_iters);
    }
    // tile tables sized for the shortest tiles (2 rows)
    long tiles = 0;
    for (int b = 0; b < count; ++b) {
        const dim3 t = lay_tiles<float>(B->lay[b]);
        tiles += (long)t.x * t.y;
    }
    B->max_tiles = (int)tiles;
    B->rs_capacity = std::max<long>(max_full, B->sm_count) * tl::kMaxSums;
    bool ok = TL_CUDA(cudaMalloc(&B->slab, total)) && TL_CUDA(cudaMalloc(&B->d_prob, sizeof(BProb) * count)) &&
              TL_CUDA(cudaMalloc(&B->d_pctl, sizeof(PCtl) * count)) &&
              TL_CUDA(cudaMalloc(&B->d_st, sizeof(MxState) * count)) &&
              TL_CUDA(cudaMalloc(&B->d_tickets, sizeof(unsigned) * count)) &&
              TL_CUDA(cudaMalloc(&B->d_partials, sizeof(double) * 2 * tiles)) &&
              TL_CUDA(cudaMalloc(&B->d_ctl, sizeof(BCtl))) &&
              TL_CUDA(cudaMalloc(&B->rs.partials, sizeof(double) * B->rs_capacity)) &&
              TL_CUDA(cudaMalloc(&B->rs.ticket, 256)) && TL_CUDA(cudaMalloc(&B->rs.out_dev, 256)) &&
              TL_CUDA(cudaMalloc(&B->d_scratch_state, sizeof(DevState)));
    if (!ok) {
        batch_free(B);
        return nullptr;
    }
    B->slab_bytes = total;
    B->rs.out_host = nullptr;
    TL_CUDA(cudaMemsetAsync(B->rs.ticket, 0, 256, B->stream));
    TL_CUDA(cudaMemsetAsync(B->d_tickets, 0, sizeof(unsigned) * count, B->stream));
    TL_CUDA(cudaMemsetAsync(B->d_ctl, 0, sizeof(BCtl), B->stream));
    static const long long default_limit = kWaitLimit;
    TL_CUDA(cudaMemcpyAsync(&B->d_ctl->limit, &default_limit, sizeof(long long), cudaMemcpyHostToDevice, B->stream));
    // Resident when the FP32 arrays fit L2 (see Resident)
    int l2 = 0;
    TL_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, B->device));
    const bool resident = total <= (size_t)l2;
    B->kernel = resident ? (const void*)k_batch_cg<Resident> : (const void*)k_batch_cg<Streaming>;
    B->smem = (resident ? Resident::STAGES : Streaming::STAGES) * sizeof(RingRow);
    int per_sm = 0;
    TL_CUDA(cudaFuncSetAttribute(B->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)B->smem));
    TL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, B->kernel, BX, B->smem));
    B->resident = std::max(1, per_sm) * B->sm_count;
    B->max_grid = kGroupsPerSm * B->sm_count;
    B->grid_blocks = grid_blocks > 0 ? std::min(grid_blocks, B->max_grid) : B->max_grid;
    if (!TL_CUDA(cudaMalloc(&B->d_block_prob, sizeof(int) * B->max_grid))) {
        batch_free(B);
        return nullptr;
    }
    if (!batch_layout(B, tile_rows != 0 ? tile_rows : 16)) {
        batch_free(B);
        return nullptr;
    }
    return B;
}

void tl2d_batch_destroy(TlBatch* B)
{
    if (!B) return;
    cudaStreamSynchronize(B->stream);
    batch_free(B);
}

// Autotuner: times `trial_iters` iterations of the batch's own CG (setup
// included, energy untouched; 0: the whole solve) for each tile height in
// {adaptive (-1), 4, 8, 16, 32, 64}
// and each number of {2, 4, 6, 8} blocks per SM that the problems' groups are
// cut for (of which as many as fit at once are launched, 4 or 6 per SM), and
// keeps the fastest. Returns 0 or an error code;
// the choice is readable with tl2d_batch_config.
int tl2d_batch_tune(TlBatch* B, int trial_iters, double* best_ms)
{
    if (tl::failed()) return tl::error_state().code;
    if (!B || trial_iters < 0) {
        tl::fail(64, "tl2d_batch_tune: batch and trial_iters >= 0 are required");
        return 64;
    }
    const int iters = trial_iters > 0 ? trial_iters : B->max_iters;   // 0: the whole solve
    drop_graph(B);
    const int rows_c[] = {kAdaptiveRows, 4, 8, 16, 32, 64};
    const int per_sm_c[] = {2, 4, 6, 8};
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    double best = 1e300;
    int best_rows = B->tile_rows, best_grid = B->grid_blocks;
    for (int k : per_sm_c) {
        const int grid = std::min(B->max_grid, k * B->sm_count);
        B->grid_blocks = grid;
        for (int rows : rows_c) {
            if (!batch_layout(B, rows)) break;   // the adaptive heights depend on the grid
            for (int rep = 0; rep < 2; ++rep) {   // first run warms up
                cudaEventRecord(e0, B->stream);
                issue_step(B, iters, false);
                cudaEventRecord(e1, B->stream);
                if (!check_ctl(B, nullptr)) break;
            }
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                best_rows = rows;
                best_grid = grid;
            }
        }
        if (tl::failed() || grid == B->max_grid) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (tl::failed()) return tl::error_state().code;
    B->grid_blocks = best_grid;
    batch_layout(B, best_rows);
    if (best_ms) *best_ms = best;
    return tl::failed() ? tl::error_state().code : 0;
}

void tl2d_batch_config(TlBatch* B, int* tile_rows, int* grid_blocks)
{
    if (!B) return;
    if (tile_rows) *tile_rows = B->tile_rows;
    if (grid_blocks) *grid_blocks = B->grid_blocks;
}

// One timestep of every problem of the batch (a CUDA graph replay after the
// first call). Per-problem outcomes through tl2d_batch_results.
int tl2d_batch_step(TlBatch* B, TlBatchStats* stats)
{
    if (tl::failed()) return tl::error_state().code;
    if (!B) {
        tl::fail(64, "tl2d_batch_step: null batch");
        return 64;
    }
    TlBatchStats local{};
    TlBatchStats* out = stats ? stats : &local;
    *out = TlBatchStats{};
    for (TlSuite2D* s : B->suites) TL_CUDA(cudaStreamSynchronize(s->stream));
    if (!B->exec && !B->graph_ok) {
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(B->stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            issue_step(B, B->max_iters, true);
            e = cudaStreamEndCapture(B->stream, &g);
        }
        if (e == cudaSuccess && g) e = cudaGraphInstantiate(&B->exec, g, 0);
        if (e == cudaSuccess) {
            B->graph = g;
            B->graph_ok = true;
        } else {
            cudaGetLastError();   // capture unsupported here: the same launches run directly
            if (g) cudaGraphDestroy(g);
            B->exec = nullptr;
        }
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, B->stream);
    if (B->exec) TL_CUDA(cudaGraphLaunch(B->exec, B->stream));
    else issue_step(B, B->max_iters, true);
    cudaEventRecord(e1, B->stream);
    TL_CUDA(cudaGetLastError());
    BCtl ctl{};
    const bool ok = check_ctl(B, &ctl);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (!ok) return tl::error_state().code;
    std::vector<MxState> st(B->count);
    TL_CUDA(cudaMemcpy(st.data(), B->d_st, sizeof(MxState) * B->count, cudaMemcpyDeviceToHost));
    out->problems = B->count;
    for (const MxState& m : st) {
        out->converged += m.reason == 1 ? 1 : 0;
        out->max_iterations = std::max(out->max_iterations, m.trip);
        out->total_iterations += m.trip;
    }
    out->kernel_iterations = ctl.iters;
    out->tile_rows = B->tile_rows;
    out->grid_blocks = B->grid_blocks;
    out->graph = B->exec ? 1 : 0;
    out->device_ms = ms;
    return tl::failed() ? tl::error_state().code : 0;
}

// How long (SM clocks) a phase wait of the persistent kernel may take
// before it gives up; cycles <= 0 restores the default (about 2 s). The
// limit lives in device memory, so captured graphs pick it up.
int tl2d_batch_set_wait_limit(TlBatch* B, long long cycles)
{
    if (!B) {
        tl::fail(64, "tl2d_batch_set_wait_limit: null batch");
        return 64;
    }
    const long long v = cycles > 0 ? cycles : kWaitLimit;
    if (!TL_CUDA(cudaMemcpyAsync(&B->d_ctl->limit, &v, sizeof(long long), cudaMemcpyHostToDevice, B->stream)) ||
        !TL_CUDA(cudaStreamSynchronize(B->stream)))
        return tl::error_state().code;
    return 0;
}

// Per-problem CG iterations and final FP64 residual r.r of the last step.
int tl2d_batch_results(TlBatch* B, int* iterations, double* rr, int* converged)
{
    if (!B) return 64;
    std::vector<MxState> st(B->count);
    if (!TL_CUDA(cudaMemcpy(st.data(), B->d_st, sizeof(MxState) * B->count, cudaMemcpyDeviceToHost)))
        return tl::error_state().code;
    for (int b = 0; b < B->count; ++b) {
        if (iterations) iterations[b] = st[b].trip;
        if (rr) rr[b] = st[b].rtrue;
        if (converged) converged[b] = st[b].reason == 1 ? 1 : 0;
    }
    return 0;
}

}  // extern "C"
