// cgchip2d.cuh -- the CG loop of a mesh that fits on chip as one persistent
// cooperative kernel (2D, FP64, four external faces).
//
// A mesh cut into strips of at most kChipRows rows, 8 strips per SM (about 1.2
// million cells on 148 SMs), keeps its CG state on the SMs for the whole loop.
// A thread holds one column of a pair of vertically adjacent strips (up to
// 16 rows): p, r and w in registers, the face coefficients in shared memory
// (in registers for strips of two rows), u in registers or shared memory. Two
// strips per thread rather than one leave 128 registers a thread, of which
// the temporaries take their share once, not twice. The strips, the row
// order in a strip and the reduction trees are those of k_cg_w_fused and
// k_cg_ur_fused, so p, r, u, w, the scalars and the trip count are theirs bit
// for bit.
//
// One trip is two grid-wide sums with the stencil between them. A pair needs p
// one cell beyond its edges: it carries those ghost cells itself and updates
// them as their owners do, p = beta p + r, from the edge cells of r that
// every warp hands over as tagged words (gridsum.cuh). An edge word is
// rewritten after the next p.w sum, to which each of its readers has
// contributed a partial formed with it; a slot of one sum after the other
// sum, to which every block contributes only when it has read all the slots.
//
// BS > 0: the preconditioned CG of pcg2d.cuh, BS rows to a block of M (1:
// jac_diag, 4: jac_block), in strips of whole blocks. z takes w's registers
// once r is updated, the edge cells handed over are z's (p = beta p + z),
// mi stays in shared memory (strips of 7 and 8 rows read it through L2) and the
// second sum is the pair r.r, r.z. w of the last trip is formed again at the
// end. The strips are rounded up to whole blocks, which the two-launch loop does
// for its u/r/z sweep only: with jac_block on a mesh whose strips are not a
// multiple of 4 rows, p.w is summed over another partition than there (3e-15
// relative); everywhere else the two loops agree bit for bit.
//
// What bounds it: two sums per trip, each one hand-over through L2, three block
// barriers and two shuffle trees (about 2 us of a trip); then the latency of the
// rows' own chains at 12 or 16 warps an SM. Captured: 512^2 and 1000^2 issue in 30
// and 32 % of the slots, the largest stalls the block barriers and the polls;
// at 14 rows a thread shared memory is 33 % busy, FP64 15 %. The kernel holds
// its SMs from the first trip to the last: another stream's solve waits for it.
// Measured, us per trip of a whole
// timestep: 64^2 5.7 against 20 for the two launches per trip it replaces,
// 512^2 6.5 against 27, 1000^2 10.2; 1080^2, just past the limit, still takes
// 37 with two launches.
#pragma once

#include "gridsum.cuh"
#include "suite2d_impl.hpp"

namespace tl2d {

struct ChipArgs {
    double *p, *r, *u, *w, *z;
    const double *kx, *ky, *mi;
    tl::TagWord* words;        // kChipWords per pair: all sums p.w, r.r, r.z, side cells, edge rows
    unsigned long long tag0;   // tags tag0 + 1 .. tag0 + max_iters are new to the words
    int gx, gy;                // strips of the mesh
    int groups;                // strip pairs per block
    DevState* st;
    double *alphas, *betas;
    DevParams prm;
    int* host_mirror;
    int* err;                  // device word: a wait gave up
    int* err_host;             // its mapped copy for the host
    int polls;                 // polls of a wait before it gives up
};

// Where a block keeps the arrays other than p, r and w: registers up to the rows
// given here, else shared memory, laid out for the largest block. No form fits
// its 128 registers a thread without spills: 56 bytes of stores at 3 rows and
// jac_diag to 616 at 8 rows and jac_block. The
// operator is held as the face coefficient left of each cell, the one below
// and, while there is room, the diagonal 1 + (kxr + kxc) + (kyu + kyc); kx is
// laid out 33 to a warp, the last being the one right of its columns.
constexpr int kChipT = BX * kChipPairs, kChipWarps = kChipT / 32;
template <int H, int BS>
struct ChipPlace {
    static constexpr int R = 2 * H;                        // rows of a pair
    static constexpr bool kRegK = H <= 2;                  // the operator in registers
    static constexpr bool kRegU = H <= 4;                  // u in registers
    static constexpr bool kSmemMi = BS && H <= 6;          // mi in shared memory, else read from L2
    static constexpr bool kDiag = H <= (BS == 0 ? 6 : 4);  // the diagonal kept
    static constexpr int KXW = kChipWarps * 33;
    static constexpr int kd = 0;                                          // [R][T]
    static constexpr int kx = kd + (kRegK || !kDiag ? 0 : R * kChipT);    // [R][warps][33]
    static constexpr int ky = kx + (kRegK ? 0 : R * KXW);                 // [R + 1][T]
    static constexpr int u = ky + (kRegK ? 0 : (R + 1) * kChipT);     // [R][T]
    static constexpr int mi = u + (kRegU ? 0 : R * kChipT);              // [R][T]
    static constexpr int bytes = (int)sizeof(double) * (mi + (kSmemMi ? R * kChipT : 0));
};

template <int H, int BS>
static __global__ void __launch_bounds__(kChipT, 1) k_cg_chip(Geo g, ChipArgs a)
{
    extern __shared__ double chip_smem_raw[];
    constexpr int NV = BS ? 2 : 1;   // sums of the second sweep
    __shared__ tl::StripSumSmem<2, NV> sums;
    __shared__ double side[kChipWarps][32];   // per warp: rows 0 .. left, 16 .. right of its columns
    using P = ChipPlace<H, BS>;
    constexpr int R = P::R;
    constexpr bool kRegK = P::kRegK, kRegU = P::kRegU, kDiag = P::kDiag;
    static_assert(BS == 0 || H % BS == 0, "a strip holds whole blocks of M");
    static_assert(P::bytes + sizeof(tl::StripSumSmem<2, NV>) + sizeof(double) * kChipWarps * 32 <= 227 * 1024,
                  "shared memory of a block");

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pair = blockIdx.x * a.groups + tid / BX;
    const int by = pair / a.gx * 2, bx = pair % a.gx;
    const bool has = by < a.gy;
    const int pairs = a.gx * ((a.gy + 1) / 2), strips = a.gx * a.gy;
    for (int n = tid; n < 3 * (int)blockDim.x; n += blockDim.x) {
        const int row = (n >> 1) / a.gx * 2 + (n & 1);
        sums.strip_of[n] = (short)(row < a.gy ? (n >> 1) % a.gx + row * a.gx : -1);
    }
    if (tid == 0) sums.waits = {a.err, a.polls, max(0, tl::kWordErrPoll - a.polls), 0};
    const int k = g.hd + bx * BX + tid % BX;
    const int j0 = has ? g.hd + by * g.rows : g.hd, j1 = min(j0 + 2 * g.rows, g.y - g.hd);
    const int nr = has ? j1 - j0 : 1;
    const bool active = has && k < g.x - g.hd;
    const int kk = min(k, g.x - g.hd - 1);   // lanes past the interior load its last column
    const bool at_l = k == g.hd, at_r = k == g.x - g.hd - 1;
    const bool refl_d = j0 == g.hd || !active, refl_u = j1 == g.y - g.hd || !active;
    const int x = g.x, i0 = kk + j0 * x;     // a mesh that fits on chip has 32-bit indices
    // side cells: lane q has row q of the column left of the warp's, lane 16 + q of the one right of them
    const int gq = lane & 15, gk = k - lane + (lane < 16 ? -1 : 32);
    const bool ghost = has && gq < nr && gk >= g.hd && gk < g.x - g.hd;
    const int gi = gk + (j0 + gq) * x;       // (valid when ghost)
    // and hands over row q of its own first (0 ..) or last (16 ..) column
    const bool edge = has && gq < nr && k - lane + (lane < 16 ? 0 : 31) < g.x - g.hd;
    // word indices: the warps of a row of pairs in column order; the rows of edge cells bottom, top
    const int side_w = 6 * pairs + (pair * 4 + (warp & 3)) * 32 + lane;
    const int side_r = lane < 16 ? side_w - 32 + 16 : side_w + 32 - 16;
    const int row_w = 134 * pairs + pair * 2 * BX + tid % BX;
    const int down_r = row_w - (2 * a.gx - 1) * BX, up_r = row_w + 2 * a.gx * BX;
    double* const mine = side[warp];
    const double* const mine_l = mine + (lane == 0 ? 0 : 16);   // the neighbour a lane at the warp's edge lacks
    const bool first = lane == 0, last = lane == 31 || at_r;
    const bool lone = first && at_r;         // a warp of one column: its right neighbour is itself
    const bool wl = k - lane == g.hd, wr = k - lane + 32 >= g.x - g.hd;   // warp at the domain's left / right

    double* const KD = chip_smem_raw + P::kd + tid;
    double* const KX = chip_smem_raw + P::kx + warp * 33 + lane;
    double* const KY = chip_smem_raw + P::ky + tid;
    double* const U = chip_smem_raw + P::u + tid;
    double* const MI = chip_smem_raw + P::mi + tid;
    double p[R], r[R], w[R], u[kRegU ? R : 1], kdv[kRegK ? R : 1], kxv[kRegK ? R : 1], kyv[kRegK ? R : 1];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int i = i0 + (q < nr ? q : 0) * x;
        p[q] = a.p[i];
        r[q] = a.r[i];
        w[q] = 0.0;
        if (kRegU) u[kRegU ? q : 0] = a.u[i];
        else U[q * kChipT] = a.u[i];
        if (P::kSmemMi) MI[q * kChipT] = a.mi[i];
        const double kxc = a.kx[i], kyc = a.ky[i];
        const double kd = 1.0 + (a.kx[i + 1] + kxc) + (a.ky[i + x] + kyc);
        if (kRegK) {
            kdv[kRegK ? q : 0] = kd;
            kxv[kRegK ? q : 0] = kxc;
            kyv[kRegK ? q : 0] = kyc;
        } else {
            if (kDiag) KD[q * kChipT] = kd;
            KX[q * P::KXW] = a.kx[i + (k > kk ? 1 : 0)];   // (past the interior: its right face)
            if (lane == 31) KX[q * P::KXW + 1] = a.kx[i + 1];
            KY[q * kChipT] = kyc;
        }
    }
    const double ky_top = a.ky[i0 + nr * x];   // the face above the pair
    if (!kRegK) KY[nr * kChipT] = ky_top;
    double p_d = refl_d ? 0.0 : a.p[i0 - x];
    double p_u = refl_u ? 0.0 : a.p[i0 + nr * x];
    double p_s = ghost ? a.p[gi] : 0.0;
    const double k_s = ghost && lane >= 16 ? a.kx[gi] : 1.0;   // right of the warp: the face's coefficient
    double rro = a.st->rro, pw[1] = {0.0}, rrn[NV] = {}, alpha = 0.0, beta = 0.0;   // (rro: r.z with BS)
    int trip = 0, reason = 0;
    bool ok = true;
    __syncthreads();

    // the cells beside the warp's columns for sweep_w: p left of them, kx p right
    auto fill_side = [&] {
        __syncwarp();
        mine[lane] = k_s * p_s;
        __syncwarp();
        if (wl || wr) {   // the reflective halo: the edge cell itself
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (at_l) mine[q] = p[q];
                if (at_r) mine[16 + q] = __ldg(a.kx + i0 + (q < nr ? q : 0) * x + 1) * p[q];
            }
            __syncwarp();
        }
    };
    // w = A p and p.w over the pair's rows; FULL: all R of them. The term of
    // the right neighbour, kxr r, is that cell's own kxc c, formed there.
    auto sweep_w = [&](auto full, auto& acc) {
        constexpr bool FULL = decltype(full)::value;
        double pd = refl_d ? p[0] : p_d;
        double kyc = kRegK ? kyv[0] : KY[0];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (!FULL && q >= nr) break;
            const double pc = p[q];
            const bool top = FULL ? q == R - 1 : q == nr - 1;
            const double pu = top ? (refl_u ? pc : p_u) : p[q + 1 < R ? q + 1 : q];
            const double kxc = kRegK ? kxv[kRegK ? q : 0] : KX[q * P::KXW];
            const double gh = mine_l[q];
            double pl = __shfl_up_sync(kFull, pc, 1);
            double xr = __shfl_down_sync(kFull, kxc * pc, 1);
            if (first) pl = gh;
            if (last) xr = gh;
            if (lone) {
                pl = mine[q];
                xr = mine[16 + q];
            }
            const double kyu = kRegK ? (top ? ky_top : kyv[kRegK && q + 1 < R ? q + 1 : 0]) : KY[(q + 1) * kChipT];
            double kd;
            if (kRegK) kd = kdv[kRegK ? q : 0];
            else if (kDiag) kd = KD[q * kChipT];
            else kd = 1.0 + (KX[q * P::KXW + 1] + kxc) + (kyu + kyc);
            const double v = kd * pc - (xr + kxc * pl) - (kyu * pu + kyc * pd);   // smvp
            w[q] = v;
            acc[q / H] += v * pc;
            pd = pc;
            kyc = kyu;
        }
    };
    // r -= alpha w and r.r, rows in the order of k_cg_ur_fused; its edge columns into `mine`
    auto sweep_r = [&](auto full, auto& acc) {
        constexpr bool FULL = decltype(full)::value;
#pragma unroll
        for (int n = 0; n < R; ++n) {
            const int q = TL2D_UR_REVERSE ? R - 1 - n : n;
            if (!FULL && q >= nr) continue;
            const double rn = r[q] - alpha * w[q];
            r[q] = rn;
            acc[0][q / H] += rn * rn;
            if (lane == 0 || lane == 31) mine[(lane & 16) + q] = rn;
        }
    };
    // BS > 0: r -= alpha w, z = M^-1 r (into w), r.r and r.z, in the order of k_pcg_ur
    auto sweep_z = [&](auto full, auto& acc) {
        constexpr bool FULL = decltype(full)::value;
        constexpr int B = BS ? BS : 1;
#pragma unroll
        for (int q0 = 0; q0 < R; q0 += B) {
            if (!FULL && q0 >= nr) break;
            double g[B], y[B], z[B];
#pragma unroll
            for (int m = 0; m < B; ++m) {
                const int q = q0 + m < R ? q0 + m : 0;
                if (!FULL && q >= nr) break;
                const double rn = r[q] - alpha * w[q];
                r[q] = rn;
                acc[0][q / H] += rn * rn;
                g[m] = P::kSmemMi ? MI[q * kChipT] : __ldg(a.mi + i0 + q * x);
                y[m] = BS > 1 ? (m == 0 ? rn * g[0] : (rn + KY[q * kChipT] * y[m > 0 ? m - 1 : 0]) * g[m]) : g[m] * rn;
            }
            double zn = 0.0;
#pragma unroll
            for (int m = B - 1; m >= 0; --m) {
                const int q = q0 + m < R ? q0 + m : 0;
                if (!FULL && q >= nr) continue;
                if (m == B - 1 || (!FULL && q == nr - 1)) {
                    zn = y[m];
                } else {
                    const double c = -KY[(q + 1) * kChipT] * g[m];
                    zn = y[m] - c * zn;
                }
                w[q] = zn;
                z[m] = zn;
                if (lane == 0 || lane == 31) mine[(lane & 16) + q] = zn;
            }
#pragma unroll
            for (int m = 0; m < B; ++m) {
                const int q = q0 + m < R ? q0 + m : 0;
                if (!FULL && q >= nr) break;
                acc[NV - 1][q / H] += r[q] * z[m];
            }
        }
    };
    const bool full = nr == R;
    // the field folded into p
    auto fold = [&](int q) { return BS ? w[q] : r[q]; };

    while (reason == 0) {
        const unsigned long long tag = a.tag0 + 1 + (unsigned long long)trip;
        if (trip > 0) {   // p = beta p + r (or z), the ghosts with their owners'
            double r_d = 0.0, r_u = 0.0, r_s = 0.0;
            const bool gd = refl_d || word_load(a.words + down_r, tag - 1, r_d);
            const bool gu = refl_u || word_load(a.words + up_r, tag - 1, r_u);
            const bool gs = !ghost || word_load(a.words + side_r, tag - 1, r_s);
#pragma unroll
            for (int q = 0; q < R; ++q) p[q] = beta * p[q] + fold(q);
            if (!gd) r_d = tl::word_wait(a.words + down_r, tag - 1, &sums.waits);
            if (!gu) r_u = tl::word_wait(a.words + up_r, tag - 1, &sums.waits);
            if (!gs) r_s = tl::word_wait(a.words + side_r, tag - 1, &sums.waits);
            p_s = beta * p_s + r_s;
            p_d = beta * p_d + r_d;
            p_u = beta * p_u + r_u;
        }
        fill_side();
        double aw[1][2] = {{0.0, 0.0}};
        if (full) sweep_w(std::true_type(), aw[0]);
        else sweep_w(std::false_type(), aw[0]);
        if (!active) aw[0][0] = aw[0][1] = 0.0;
        ok = tl::strip_sum<BX, 2, 1>(aw, has ? pair : -1, strips, 2 * pairs, sums, a.words, tag, [] {},
                              [&](const double* t) { return rro / t[0]; }, pw, alpha);
        if (!ok) break;
        double ar[NV][2] = {};
        if (BS) {
            if (full) sweep_z(std::true_type(), ar);
            else sweep_z(std::false_type(), ar);
        } else {
            if (full) sweep_r(std::true_type(), ar);
            else sweep_r(std::false_type(), ar);
        }
        if (!active)
#pragma unroll
            for (int n = 0; n < NV; ++n) ar[n][0] = ar[n][1] = 0.0;
        __syncwarp();
        if (edge) tl::word_store(a.words + side_w, mine[lane], tag);
        if (active) {
            tl::word_store(a.words + row_w, fold(0), tag);
            double top = fold(R - 1);
            if (!full) {
                top = fold(0);
#pragma unroll
                for (int q = 1; q < R; ++q) top = q < nr ? fold(q) : top;
            }
            tl::word_store(a.words + row_w + BX, top, tag);
        }
        ok = tl::strip_sum<BX, 2, NV>(ar, has ? pair : -1, strips, 2 * pairs, sums, a.words + 2 * pairs, tag,
                               [&] {
#pragma unroll
                                   for (int q = 0; q < R; ++q) {
                                       if (kRegU) u[kRegU ? q : 0] += alpha * p[q];
                                       else U[q * kChipT] += alpha * p[q];
                                   }
                               },
                               [&](const double* t) { return t[NV - 1] / rro; }, rrn, beta);
        if (!ok) break;
        if (blockIdx.x == 0 && tid == 0) {
            a.alphas[trip] = alpha;
            a.betas[trip] = beta;
        }
        rro = rrn[NV - 1];
        reason = tl::trip_reason(a.prm, rrn[0], trip);
        ++trip;
    }

    if (BS) {   // z, which holds w's registers; then w again
        if (active)
#pragma unroll
            for (int q = 0; q < R; ++q)
                if (q < nr) a.z[i0 + q * x] = w[q];
        double acc[2] = {0.0, 0.0};
        fill_side();
        sweep_w(std::false_type(), acc);
    }
    if (active) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (q < nr) {
                const int i = i0 + q * x;
                a.p[i] = p[q];
                a.r[i] = r[q];
                a.w[i] = w[q];
                a.u[i] = kRegU ? u[kRegU ? q : 0] : U[q * kChipT];
            }
        }
    }
    if (!ok && tid == 0) *(volatile int*)a.err_host = 1;   // whichever block it is
    if (blockIdx.x == 0 && tid == 0) {
        DevState* st = a.st;
        st->pw = pw[0];
        st->rro = rro;
        st->rrn = st->error = rrn[0];
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

}  // namespace tl2d
