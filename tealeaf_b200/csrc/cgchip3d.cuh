// cgchip3d.cuh -- the CG loop of a mesh that fits on chip as one persistent
// cooperative kernel (3D, FP64, six external faces); the 3D twin of
// cgchip2d.cuh, which has the reasons.
//
// A unit is an x-y tile of 32 x 8 columns and up to kChipPlanes3 planes: T of
// the one-step sweeps' z-pencils (ZR planes each) on top of one another, so
// that their sums are those sweeps' sums. One thread holds one column: p, r
// and w in registers, u in registers (up to 8 planes) or shared memory (up to
// 12), the face coefficients in shared memory except kz of units of more than
// 8 planes, which is read through L2. One unit of 256 threads per block, or
// two. x-neighbours come by shuffle, y-neighbours through a shared plane, one
// barrier per plane; beyond the unit's six faces a unit carries the ghost
// cells of p itself and updates them from the edge cells of r that their
// owners hand over.
//
// What bounds it: the sums' hand-overs and, of the unit's 128 registers a thread
// (48 to 808 bytes of spill stores), one barrier per plane in the w sweep. 48^3
// captured: 13 % of the issue slots, the largest stalls the polls and the barriers.
// Measured, us per trip of a whole timestep, against the two launches per trip
// it replaces: 32^3 6.7 / 23.0, 48^3 8.8 / 21.9, 64^3 9.2 / 23.8, 80^3 11.2 /
// 30.2, 100 x 90 x 80 20.9 / 39.5.
#pragma once

#include "gridsum.cuh"
#include "suite3d_impl.hpp"

namespace tl3d {

struct Chip3Args {
    double *p, *r, *u, *w;
    const double *kx, *ky, *kz;
    tl::TagWord* words;        // chip3_words per unit: all sums p.w, all r.r, side columns, edge rows, end planes
    unsigned long long tag0;   // tags tag0 + 1 .. tag0 + max_iters are new to the words
    int gx, gy, tiles_z;       // z-pencils of the mesh
    int groups;                // units per block
    DevState* st;
    double *alphas, *betas;
    DevParams prm;
    int* host_mirror;
    int* err;                  // device word: a wait gave up
    int* err_host;             // its mapped copy for the host
    int polls;                 // polls of a wait before it gives up
};

template <int ZR, int T>
struct Chip3Place {
    static constexpr int R = ZR * T;             // planes of a unit
    static constexpr bool kRegU = R <= 8;        // u in registers
    static constexpr bool kSmemU = !kRegU && R <= 12;   // or shared memory, else in memory
    static constexpr bool kSmemKz = R <= 8;
    static constexpr int kx = 0;                               // [R][8][33]
    static constexpr int ky = kx + R * BY * 33;                // [R][9][32]
    static constexpr int kz = ky + R * 9 * 32;                 // [R + 1][8][32]
    static constexpr int u = kz + (kSmemKz ? (R + 1) * NT : 0);   // [R][8][32]
    static constexpr int yg = u + (kSmemU ? R * NT : 0);       // [2][R][32] ghost rows of p
    static constexpr int pl = yg + 2 * R * 32;                 // [2][8][32] p of the plane at hand
    static constexpr int side = pl + 2 * NT;                   // [8][32] per warp: planes 0 .. left, 16 .. right
    static constexpr int total = side + BY * 32;               // of one unit
    static constexpr int bytes = (int)sizeof(double) * total;
};

template <int ZR, int T>
static __global__ void __launch_bounds__(2 * NT, 1) k3_cg_chip(Geo g, Chip3Args a)
{
    extern __shared__ double chip3_raw[];
    __shared__ tl::StripSumSmem<T, 1> sums;
    using P = Chip3Place<ZR, T>;
    constexpr int R = P::R, TW = tl::strip_words(T);   // words of a unit per sum
    static_assert(R <= kChipPlanes3, "side columns: one lane per plane and side");
    static_assert(2 * P::bytes + sizeof(sums) <= 227 * 1024, "shared memory of a block");

    const int tid = threadIdx.x, lane = tid & 31, group = tid / NT, ty = (tid % NT) >> 5;
    double* const S = chip3_raw + group * P::total;
    const int unit = blockIdx.x * a.groups + group;
    const int bx = unit % a.gx, by = unit / a.gx % a.gy, cz = unit / (a.gx * a.gy);
    const int ncz = (a.tiles_z + T - 1) / T, units = a.gx * a.gy * ncz, strips = a.gx * a.gy * a.tiles_z;
    const bool has = cz < ncz;
    for (int n = tid; n < 3 * (int)blockDim.x; n += blockDim.x) {
        const int un = n / TW, h = n % TW, bz = un / (a.gx * a.gy) * T + h;
        sums.strip_of[n] = (short)(h < T && bz < a.tiles_z ? un % (a.gx * a.gy) + a.gx * a.gy * bz : -1);
    }
    if (tid == 0) sums.waits = {a.err, a.polls, max(0, tl::kWordErrPoll - a.polls), 0};
    const int hd = g.hd, x = g.x, xy = g.x * g.y;   // a mesh that fits on chip has 32-bit indices
    const int k = hd + bx * BX + lane, j = hd + by * BY + ty;
    const int i0 = has ? hd + cz * R : hd, i1 = min(i0 + R, g.z - hd);
    const int nr = has ? i1 - i0 : 1;
    const bool rowok = has && j < g.y - hd, active = rowok && k < g.x - hd;
    const int kk = min(k, g.x - hd - 1), jj = min(j, g.y - hd - 1);   // cells past the interior load its last ones
    const bool at_l = k == hd, at_r = k == g.x - hd - 1, at_b = j == hd, at_t = j == g.y - hd - 1;
    const bool refl_k = i0 == hd || !active, refl_f = i1 == g.z - hd || !active;
    const int c0 = kk + jj * x + i0 * xy;
    // side columns: lane q has plane q of the column left of the row, lane 16 + q of the one right of it
    const int gq = lane & 15, gk = lane < 16 ? k - lane - 1 : k - lane + 32;
    const bool ghost = rowok && gq < nr && gk >= hd && gk < g.x - hd;
    const bool edge = rowok && gq < nr && k - lane + (lane < 16 ? 0 : 31) < g.x - hd;
    // words
    const int w0 = 2 * TW * units;
    const int side_w = w0 + (unit * BY + ty) * 32 + lane;
    const int side_r = lane < 16 ? side_w - BY * 32 + 16 : side_w + BY * 32 - 16;
    const int y0 = w0 + 256 * units, rows_w = y0 + unit * 2 * R * 32;   // [bottom, top][R][32]
    const int z0 = y0 + 64 * R * units, ends_w = z0 + unit * 2 * NT + tid % NT;   // [back, front][8][32]
    const int back_r = ends_w - (2 * a.gx * a.gy - 1) * NT, front_r = ends_w + 2 * a.gx * a.gy * NT;
    // ghost rows below (side 0) and above (1) the tile: this warp's share of their 2 R planes
    const bool below = has && by > 0 && lane + bx * BX < g.x - 2 * hd;
    const bool above = has && by + 1 < a.gy && lane + bx * BX < g.x - 2 * hd;
    double* const mine = S + P::side + ty * 32;
    double* const KX = S + P::kx + ty * 33 + lane;
    double* const KY = S + P::ky + ty * 32 + lane;
    double* const KZ = S + P::kz + tid % NT;
    double* const U = S + P::u + tid % NT;
    double* const YG = S + P::yg + lane;
    double* const PL = S + P::pl + tid % NT;
    const int bar = 2 + group;   // the unit's barrier

    double p[R], r[R], w[R], u[P::kRegU ? R : 1];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int i = c0 + (q < nr ? q : 0) * xy;
        p[q] = a.p[i];
        r[q] = a.r[i];
        w[q] = 0.0;
        if (P::kRegU) u[P::kRegU ? q : 0] = a.u[i];
        if (P::kSmemU) U[q * NT] = a.u[i];
        KX[q * BY * 33] = a.kx[i + (k > kk ? 1 : 0)];   // (past the interior: its right and upper faces)
        if (lane == 31) KX[q * BY * 33 + 1] = a.kx[i + 1];
        KY[q * 9 * 32] = a.ky[i + (j > jj ? x : 0)];
        if (ty == BY - 1) KY[q * 9 * 32 + 32] = a.ky[i + x];
        if (P::kSmemKz) KZ[q * NT] = a.kz[i];
    }
    if (P::kSmemKz) KZ[nr * NT] = a.kz[c0 + nr * xy];
    double p_k = refl_k ? 0.0 : a.p[c0 - xy];
    double p_f = refl_f ? 0.0 : a.p[c0 + nr * xy];
    double p_s = ghost ? a.p[gk + j * x + (i0 + gq) * xy] : 0.0;
    for (int n = ty; n < 2 * R; n += BY) {
        const int q = n % R, side = n / R;
        if (q < nr && (side ? above : below))
            YG[n * 32] = a.p[k + (hd + by * BY + (side ? BY : -1)) * x + (i0 + q) * xy];
    }
    double rro = a.st->rro, pw[1] = {0.0}, rrn[1] = {0.0}, alpha = 0.0, beta = 0.0;
    int trip = 0, reason = 0;
    bool ok = true;
    __syncthreads();

    // w = A p and p.w over the unit's planes; FULL: all R of them
    auto sweep_w = [&](auto full, auto& acc) {
        constexpr bool FULL = decltype(full)::value;
        double bk = refl_k ? p[0] : p_k;
        double kzc = P::kSmemKz ? KZ[0] : __ldg(a.kz + c0);
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (!FULL && q >= nr) break;
            const double c = p[q];
            double* const pl = PL + (q & 1) * NT;
            *pl = c;
            asm volatile("bar.sync %0, %1;\n" ::"r"(bar), "n"(NT) : "memory");
            const bool top = FULL ? q == R - 1 : q == nr - 1;
            const double fr = top ? (refl_f ? c : p_f) : p[q + 1 < R ? q + 1 : q];
            double l = __shfl_up_sync(kFull3, c, 1);
            double rt = __shfl_down_sync(kFull3, c, 1);
            if (lane == 0) l = mine[q];
            if (lane == 31) rt = mine[16 + q];
            if (at_l) l = c;
            if (at_r) rt = c;
            double d = ty > 0 ? pl[-32] : YG[q * 32];
            double up = ty < BY - 1 ? pl[32] : YG[(R + q) * 32];
            if (at_b) d = c;
            if (at_t) up = c;
            const double kzf = P::kSmemKz ? KZ[(q + 1) * NT] : __ldg(a.kz + c0 + (q + 1) * xy);
            const double v = smvp(KX[q * BY * 33], KX[q * BY * 33 + 1], KY[q * 9 * 32], KY[q * 9 * 32 + 32], kzc, kzf,
                                  c, l, rt, d, up, bk, fr);
            w[q] = v;
            acc[q / ZR] += v * c;
            bk = c;
            kzc = kzf;
        }
    };
    // r -= alpha w and r.r, planes in the order of k3_cg_ur; its edge columns into `mine`
    auto sweep_r = [&](auto full, auto& acc) {
        constexpr bool FULL = decltype(full)::value;
#pragma unroll
        for (int n = 0; n < R; ++n) {
            const int q = TL3D_UR_REVERSE ? R - 1 - n : n;
            if (!FULL && q >= nr) continue;
            const double rn = r[q] - alpha * w[q];
            r[q] = rn;
            acc[q / ZR] += rn * rn;
            if (lane == 0 || lane == 31) mine[(lane & 16) + q] = rn;
        }
    };
    const bool full = nr == R;

    while (reason == 0) {
        const unsigned long long tag = a.tag0 + 1 + (unsigned long long)trip;
        if (trip > 0) {   // p = beta p + r, the ghosts with their owners' r
            double r_k = 0.0, r_f = 0.0, r_s = 0.0;
            const bool gb = refl_k || word_load(a.words + back_r, tag - 1, r_k);
            const bool gf = refl_f || word_load(a.words + front_r, tag - 1, r_f);
            const bool gs = !ghost || word_load(a.words + side_r, tag - 1, r_s);
            double r_y[(2 * R + BY - 1) / BY];
            bool gy[(2 * R + BY - 1) / BY];
#pragma unroll
            for (int m = 0; m < (2 * R + BY - 1) / BY; ++m) {
                const int n = ty + m * BY, q = n % R, side = n / R;
                r_y[m] = 0.0;
                // the tile below's top row, the tile above's bottom row
                gy[m] = n >= 2 * R || q >= nr || !(side ? above : below) ||
                        word_load(a.words + rows_w + (side ? a.gx * 2 * R * 32 + q * 32 : (R + q - 2 * a.gx * R) * 32) + lane,
                                  tag - 1, r_y[m]);
            }
#pragma unroll
            for (int q = 0; q < R; ++q) p[q] = beta * p[q] + r[q];
            if (!gb) r_k = tl::word_wait(a.words + back_r, tag - 1, &sums.waits);
            if (!gf) r_f = tl::word_wait(a.words + front_r, tag - 1, &sums.waits);
            if (!gs) r_s = tl::word_wait(a.words + side_r, tag - 1, &sums.waits);
            p_s = beta * p_s + r_s;
            p_k = beta * p_k + r_k;
            p_f = beta * p_f + r_f;
#pragma unroll
            for (int m = 0; m < (2 * R + BY - 1) / BY; ++m) {
                const int n = ty + m * BY, q = n % R, side = n / R;
                if (!gy[m])
                    r_y[m] = tl::word_wait(a.words + rows_w +
                                               (side ? a.gx * 2 * R * 32 + q * 32 : (R + q - 2 * a.gx * R) * 32) + lane,
                                           tag - 1, &sums.waits);
                if (n < 2 * R && q < nr && (side ? above : below)) YG[n * 32] = beta * YG[n * 32] + r_y[m];
            }
        }
        __syncwarp();
        mine[lane] = p_s;
        __syncwarp();
        double acc[1][T] = {};
        if (full) sweep_w(std::true_type(), acc[0]);
        else sweep_w(std::false_type(), acc[0]);
        if (!active)
#pragma unroll
            for (int h = 0; h < T; ++h) acc[0][h] = 0.0;
        // nothing to publish: every ghost was read before its reader's partial was formed
        ok = tl::strip_sum<NT, T, 1>(acc, has ? unit : -1, strips, TW * units, sums, a.words, tag, [] {},
                                     [&](const double* t) { return rro / t[0]; }, pw, alpha);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < T; ++h) acc[0][h] = 0.0;
        if (full) sweep_r(std::true_type(), acc[0]);
        else sweep_r(std::false_type(), acc[0]);
        if (!active)
#pragma unroll
            for (int h = 0; h < T; ++h) acc[0][h] = 0.0;
        __syncwarp();
        if (edge) tl::word_store(a.words + side_w, mine[lane], tag);
        if (active && (ty == 0 || ty == BY - 1)) {
#pragma unroll
            for (int q = 0; q < R; ++q)
                if (q < nr) tl::word_store(a.words + rows_w + ((ty ? R : 0) + q) * 32 + lane, r[q], tag);
        }
        if (active) {
            tl::word_store(a.words + ends_w, r[0], tag);
            double top = r[R - 1];
            if (!full) {
                top = r[0];
#pragma unroll
                for (int q = 1; q < R; ++q) top = q < nr ? r[q] : top;
            }
            tl::word_store(a.words + ends_w + NT, top, tag);
        }
        ok = tl::strip_sum<NT, T, 1>(acc, has ? unit : -1, strips, TW * units, sums, a.words + TW * units, tag,
                                     [&] {
#pragma unroll
                                         for (int q = 0; q < R; ++q) {
                                             if (P::kRegU) u[P::kRegU ? q : 0] += alpha * p[q];
                                             else if (P::kSmemU) U[q * NT] += alpha * p[q];
                                             else if (active && q < nr) a.u[c0 + q * xy] += alpha * p[q];
                                         }
                                     },
                                     [&](const double* t) { return t[0] / rro; }, rrn, beta);
        if (!ok) break;
        if (blockIdx.x == 0 && tid == 0) {
            a.alphas[trip] = alpha;
            a.betas[trip] = beta;
        }
        rro = rrn[0];
        reason = tl::trip_reason(a.prm, a.prm.dims3 ? sqrt(rro) : rro, trip);
        ++trip;
    }

    if (active) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (q < nr) {
                const int i = c0 + q * xy;
                a.p[i] = p[q];
                a.r[i] = r[q];
                a.w[i] = w[q];
                if (P::kRegU) a.u[i] = u[P::kRegU ? q : 0];
                if (P::kSmemU) a.u[i] = U[q * NT];
            }
        }
    }
    if (!ok && tid == 0) *(volatile int*)a.err_host = 1;   // whichever block it is
    if (blockIdx.x == 0 && tid == 0) {
        DevState* st = a.st;
        st->pw = pw[0];
        st->rro = st->rrn = rro;
        st->error = a.prm.dims3 ? sqrt(rro) : rro;
        st->alpha = alpha;
        st->beta = beta;
        st->trip = trip;
        st->done = 1;
        st->reason = reason;
        a.host_mirror[0] = 1;
        a.host_mirror[1] = trip;
        a.host_mirror[2] = reason;
    }
}

template <int ZR, int T>
static bool launch_chip3(TlSuite3D* s, Chip3Args& a, int units)
{
    const int threads = a.groups * NT, smem = a.groups * Chip3Place<ZR, T>::bytes;
    // the limit of both group counts, so that a thread that launches the other one at the same time sets the same
    TL_CUDA(cudaFuncSetAttribute(k3_cg_chip<ZR, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 2 * Chip3Place<ZR, T>::bytes));
    void* args[] = {&s->g, &a};
    return tl::launch_persistent(s, "k3_cg_chip", (const void*)k3_cg_chip<ZR, T>, tl::ceil_div(units, a.groups), threads,
                                 args, smem);
}

// The whole CG loop in one launch, for a chunk with chip words: p, r, w of the
// chunk, the solution in `u`, stopped as `prm` says; the state is left as the
// two-launch loop leaves it, p in the buffer it was in. False (nothing done)
// where it does not run: the mesh does not fit, or not all its blocks do. The
// caller waits for the stream and calls check_chip.
static bool cg_chip3(TlSuite3D* s, Chunk* chunk, double* u, const DevParams& prm)
{
    if (!s->chip_words || !s->chip_loop || prm.max_iters <= 0) return false;
    const dim3 grid = interior_grid(s->g);
    const Chip3Cut c = chip3_cut(s->g, s->sm_count);
    const int units = (int)(grid.x * grid.y) * tl::ceil_div(grid.z, c.tiles);
    Chip3Args a{chunk->vec_p, chunk->vec_r, u, chunk->vec_w, chunk->vec_kx, chunk->vec_ky, chunk->vec_kz,
                s->chip_words, s->chip_tag, (int)grid.x, (int)grid.y, (int)grid.z,
                tl::ceil_div(units, s->sm_count), s->d_state, s->d_cg_alphas, s->d_cg_betas, prm, s->d_mirror,
                s->chip_err, s->d_mirror + kChipErrWord, s->chip_polls};
    s->chip_tag += (unsigned long long)prm.max_iters;
    switch (s->g.zr * 8 + c.tiles) {
        case 4 * 8 + 1: return launch_chip3<4, 1>(s, a, units);
        case 4 * 8 + 2: return launch_chip3<4, 2>(s, a, units);
        case 4 * 8 + 3: return launch_chip3<4, 3>(s, a, units);
        case 4 * 8 + 4: return launch_chip3<4, 4>(s, a, units);
        case 5 * 8 + 1: return launch_chip3<5, 1>(s, a, units);
        case 5 * 8 + 2: return launch_chip3<5, 2>(s, a, units);
        case 5 * 8 + 3: return launch_chip3<5, 3>(s, a, units);
        case 6 * 8 + 1: return launch_chip3<6, 1>(s, a, units);
        default: return launch_chip3<6, 2>(s, a, units);
    }
}

}  // namespace tl3d
