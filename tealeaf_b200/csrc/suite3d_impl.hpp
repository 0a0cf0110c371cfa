// suite3d_impl.hpp -- host-side state of one 3D chunk, shared by the
// kernel-interface layer (suite3d.cu) and the device-resident driver
// (driver3d.cu). Same design as the 2D suite (suite2d_impl.hpp).
#pragma once

#include "blocked3d.cuh"
#include "gridsum.cuh"
#include "kernels3d.cuh"
#include "summary.cuh"
#include "tmacache.hpp"

#include <cuda_runtime.h>

#include <vector>

enum AltField3 { ALT3_P = 0, ALT3_U = 1, ALT3_R = 2, ALT3_SD = 3, ALT3_COUNT = 4 };

struct TlSuite3D {
    int device = 0;
    int sm_count = 148;
    cudaStream_t stream = nullptr;
    tl3d::Geo g{0, 0, 0, 0};
    void* slab = nullptr;
    size_t slab_bytes = 0;
    tl::ReduceSlots rs{};
    double* h_out = nullptr;
    long partial_capacity = 0;
    long sum_cells = 0;               // interior cells of the field summary
    void* sum_scratch = nullptr;      // its tile sums and pairs (summary.cuh)
    State* d_states = nullptr;
    int d_states_cap = 0;
    double* d_comm = nullptr;
    long d_comm_cap = 0;
    double* alt[ALT3_COUNT] = {nullptr, nullptr, nullptr, nullptr};
    tl::Profiler prof;
    struct {
        bool calc_p = false;
        double beta = 0.0;
        int halo[TL3_NUM_FIELDS] = {0, 0, 0, 0, 0, 0};
    } pend;
    tl::DevState* d_state = nullptr;
    int* h_mirror = nullptr;
    int* d_mirror = nullptr;
    double* d_cg_alphas = nullptr;
    double* d_cg_betas = nullptr;
    double* d_cheby_alphas = nullptr;
    double* d_cheby_betas = nullptr;
    int table_len = 0;
    // CG loop of a mesh that fits on chip (cgchip3d.cuh): the words its blocks
    // exchange (null for a larger mesh), the last tag used in them and the
    // word its bounded waits raise.
    tl::TagWord* chip_words = nullptr;
    unsigned long long chip_tag = 0;
    int* chip_err = nullptr;
    int chip_loop = tl::kChipOn;       // whether that loop is used (tl3d_set_chip_loop)
    int chip_polls = tl::kWordPolls;   // polls of a wait before it gives up (tl3d_set_chip_wait_limit)
    bool tma = true;   // feed the CG w sweep by TMA where the layout allows (tl3d_set_tma)
    bool temporal_blocking = true;   // Chebyshev / PPCG blocks (tl3d_set_temporal_blocking)
    // Chebyshev trips / PPCG inner steps of the run_* path deferred while the
    // reference drivers' call pattern holds, then run temporally blocked
    struct Queue {
        bool active = false;
        std::vector<double> a, b;
    };
    Queue cq, pq;
    tl::TmaCache<CUtensorMap, 40> tma_cache;   // tensor maps encoded once per array
};

// Index of the int, in the mapped mirror words, that the bounded TMA barrier
// waits set when one gives up.
constexpr int kTmaErrWord = 15;
// The same for the waits of the CG loop on chip.
constexpr int kChipErrWord = 14;

#define TL3_LAUNCH(s, name, ...)               \
    do {                                       \
        (s)->prof.begin((s)->stream, name);    \
        __VA_ARGS__;                           \
        (s)->prof.end((s)->stream);            \
        TL_LAUNCHED(name);                     \
    } while (0)

namespace tl3d {

TlSuite3D* suite_of(Chunk* chunk);

inline dim3 interior_grid(const Geo& g)
{
    return dim3(tl::ceil_div(g.x - 2 * g.hd, BX), tl::ceil_div(g.y - 2 * g.hd, BY), tl::ceil_div(g.z - 2 * g.hd, g.zr));
}
// z cells per thread of the interior sweeps: the grid should be whole waves
// both for the staged stencil sweeps (TL3D_MINB blocks per SM) and for the
// pointwise ones (8 per SM); longer pencils carry less prologue (one extra
// staged plane per pencil).
inline int choose_zr(int nx, int ny, int nz, int sm_count)
{
    const long bxy = (long)tl::ceil_div(nx, BX) * tl::ceil_div(ny, BY);
    int best = ZR;
    double best_score = -1.0;
    for (int zr = 4; zr <= 32; ++zr) {
        const long blocks = bxy * tl::ceil_div(nz, zr);
        auto eff = [&](long slots) {
            const long waves = (blocks + slots - 1) / slots;
            return (double)blocks / (double)(waves * slots);
        };
        const double score = eff((long)sm_count * TL3D_MINB) * eff((long)sm_count * 8) * zr / (zr + 1.0);
        if (score > best_score + 1e-12) {
            best_score = score;
            best = zr;
        }
    }
    return best;
}
// How a mesh is cut to be held on the SMs (cgchip3d.cuh): units of `tiles`
// z-pencils, at most kChipPlanes3 planes, two units per SM at most; tiles 0
// where it does not fit. choose_zr gives pencils of 4 to 6 planes to nearly
// every mesh small enough. The fewest pencils per unit that fit: more units,
// less work in each.
constexpr int kChipPlanes3 = 16;
struct Chip3Cut {
    int tiles, units;
};
inline Chip3Cut chip3_cut(const Geo& g, int sm_count)
{
    const dim3 d = interior_grid(g);
    if (g.zr >= 4 && g.zr <= 6)
        for (int t = 1; t * g.zr <= kChipPlanes3; ++t) {
            const long units = (long)d.x * d.y * tl::ceil_div(d.z, t);
            if (units <= 2L * sm_count) return {t, (int)units};
        }
    return {0, 0};
}
// Words of one unit: its sums, twice; 8 rows' 32 side cells; 2 edge rows of
// its planes; 2 end planes.
inline size_t chip3_words(int planes, int tiles) { return 2 * tl::strip_words(tiles) + 256 + 64 * (size_t)planes + 2 * NT; }

inline dim3 full_grid(const Geo& g) { return dim3(tl::ceil_div(g.x, FBX), tl::ceil_div(g.y, FBY), g.z); }
// Interior grid plus the halo-duty z-plane of the fused sweeps.
inline dim3 fused_grid(const Geo& g)
{
    dim3 d = interior_grid(g);
    d.z += 1;
    return d;
}
inline dim3 interior_block() { return dim3(BX, BY); }
inline dim3 full_block() { return dim3(FBX, FBY); }
bool fetch(TlSuite3D* s, int n, double* out);
void flush(TlSuite3D* s, Chunk* chunk);
Faces faces_of(const Chunk* chunk);
double** field_slot(Chunk* chunk, AltField3 f);
void swap_alt(TlSuite3D* s, Chunk* chunk, AltField3 f);


// Tensor map of a chunk array for walkt: kind 0 operand (box (BX+4) x (BY+2)),
// 1 kx (BX+2) x BY, 2 ky BX x (BY+1), 3 kz BX x BY; for k3_cg_ur_tma kind 4
// BX x BY x kPlanesU; for k3_blocked_tma kind 5 kRX x kRYT; encoded once per
// array.
inline const CUtensorMap* tma_map(TlSuite3D* s, const double* ptr, int kind)
{
    static const unsigned box[6][3] = {{BX + 4, BY + 2, 1}, {BX + 2, BY, 1}, {BX, BY + 1, 1}, {BX, BY, 1},
                                       {BX, BY, kPlanesU}, {kRX, kRYT, 1}};
    return s->tma_cache.lookup(ptr, kind, [&](CUtensorMap* m) {
        return tl::tma_encode_3d(m, ptr, s->g.x, s->g.y, s->g.z, box[kind][0], box[kind][1], box[kind][2]);
    });
}

// The TMA boxes start at x = hd - 2 + 32 bx: an even halo depth and an even
// row length keep every start and stride on a 16-byte boundary.
inline bool tma_usable(const TlSuite3D* s) { return s->tma && s->g.hd % 2 == 0 && s->g.x % 2 == 0; }

inline bool tma_failed(const TlSuite3D* s) { return s->h_mirror && s->h_mirror[kTmaErrWord] != 0; }

// After a CG loop on chip has run and the stream was waited for: reports a wait
// that gave up in it and clears its words, so that the chunk's next solve is on
// its own.
inline void check_chip(TlSuite3D* s)
{
    const int word = kChipErrWord;
    if (!s->h_mirror[word]) return;
    s->h_mirror[word] = 0;
    TL_CUDA(cudaMemsetAsync(s->chip_err, 0, sizeof(int), s->stream));
    tl::fail(38, "the CG loop on chip did not complete: a wait for another block's sums or edge cells gave up after "
                 "%d polls", s->chip_polls);
}

// One launch of the temporally blocked Chebyshev (MODE 0) / PPCG (MODE 1)
// steps: region planes by TMA where the boxes can start on 16-byte
// boundaries (even halo depth, margin and row length), else per-thread
// loads; the same results either way. Internal linkage, like the kernels.
template <int MODE, int HS>
static void launch_blocked3_tma(TlSuite3D* s, const char* name, Blocked3Args a, const Blocked3Maps& m,
                                double* A_out, double* B_out, double* u, double* w, double* r, const int* done)
{
    static unsigned set = 0;   // devices on which the shared-memory size was raised
    if (!(set & (1u << (s->device & 31)))) {
        TL_CUDA(cudaFuncSetAttribute(k3_blocked_tma<MODE, HS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kBlocked3TmaBytes));
        set |= 1u << (s->device & 31);
    }
    const dim3 grid = blocked3_grid(s->g, kTX3, kTYT3, s->sm_count, a.planes);
    TL3_LAUNCH(s, name, (k3_blocked_tma<MODE, HS><<<grid, dim3(kRX, kTYT), kBlocked3TmaBytes,
                                                    s->stream>>>(s->g, a, m, A_out, B_out, u, w, r, done,
                                                                 s->d_mirror + kTmaErrWord)));
}

template <int MODE>
static void launch_blocked3(TlSuite3D* s, Chunk* chunk, Blocked3Args a, const double* A_in,
                            const double* B_in, double* A_out, double* B_out, const double* u0, double* u, double* w,
                            double* r, const int* done)
{
    const char* name = MODE == 0 ? "k3_blocked<cheby>" : "k3_blocked<ppcg>";
    if (tma_usable(s) && kTB3 % 2 == 0 && a.steps >= 1 && a.steps <= 2) {
        const CUtensorMap* ma = tma_map(s, A_in, 5);
        const CUtensorMap* mb = tma_map(s, B_in, 5);
        const CUtensorMap* mc = tma_map(s, MODE == 0 ? u0 : u, 5);
        const CUtensorMap* mx = tma_map(s, chunk->vec_kx, 5);
        const CUtensorMap* my = tma_map(s, chunk->vec_ky, 5);
        const CUtensorMap* mz = tma_map(s, chunk->vec_kz, 5);
        if (ma && mb && mc && mx && my && mz) {
            const Blocked3Maps m{*ma, *mb, *mc, *mx, *my, *mz};
            if (a.steps == 1) launch_blocked3_tma<MODE, 1>(s, name, a, m, A_out, B_out, u, w, r, done);
            else launch_blocked3_tma<MODE, 2>(s, name, a, m, A_out, B_out, u, w, r, done);
            return;
        }
    }
    const dim3 grid = blocked3_grid(s->g, kTX3, kTY3, s->sm_count, a.planes);
    TL3_LAUNCH(s, name, (k3_blocked<MODE><<<grid, dim3(kRX, kRY), 0, s->stream>>>(
                            s->g, a, A_in, B_in, A_out, B_out, u0, u, w, r, chunk->vec_kx, chunk->vec_ky,
                            chunk->vec_kz, done)));
}

// Where the sums of a sweep go: a device-resident loop (done) keeps them on the
// device, a call of the kernel interface has the host read them. A kernel that
// writes to mapped host memory ends when the write has crossed the bus (1 us).
inline tl::ReduceSlots loop_slots(const TlSuite3D* s, const int* done)
{
    tl::ReduceSlots rs = s->rs;
    if (done) rs.out_host = nullptr;
    return rs;
}

// The fused CG w sweep (k3_cg_w semantics), by TMA where possible; U: with the
// u updates of the two trips before it. Internal linkage, like the kernels it launches: each translation unit has
// its own kernel copies, so each keeps its own record of the raised
// shared-memory limit.
template <bool F, bool R, bool U = false, typename Finish>
static void launch_cg_w3(TlSuite3D* s, Chunk* chunk, dim3 grid, const Faces& fc, Scalar beta, const double* p_in,
                  double* p_out, const double* r, double* w, double* u_halo, int uhd, const int* done, Finish fin,
                  const CgU& cu = CgU{})
{
    const char* name = U ? "k3_cg_wu" : "k3_cg_w";
    const dim3 bl = interior_block();
    if (tma_usable(s)) {
        const CUtensorMap* a = tma_map(s, p_in, 0);
        const CUtensorMap* b = F ? tma_map(s, r, 0) : a;
        const CUtensorMap* kx = tma_map(s, chunk->vec_kx, 1);
        const CUtensorMap* ky = tma_map(s, chunk->vec_ky, 2);
        const CUtensorMap* kz = tma_map(s, chunk->vec_kz, 3);
        if (a && b && kx && ky && kz) {
            const Tma3Maps m{*a, *b, *kx, *ky, *kz};
            static unsigned attr_set = 0;   // devices on which the shared-memory size was raised
            if (!(attr_set & (1u << (s->device & 31)))) {
                TL_CUDA(cudaFuncSetAttribute(k3_cg_w_tma<F, R, U, Finish>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kTmaRingBytes));
                attr_set |= 1u << (s->device & 31);
            }
            TL3_LAUNCH(s, name, (k3_cg_w_tma<F, R, U><<<grid, bl, kTmaRingBytes, s->stream>>>(
                                    s->g, fc, beta, cu, m, p_in, p_out, r, w, u_halo, uhd, loop_slots(s, done), done,
                                    fin,
                                    s->d_mirror + kTmaErrWord)));
            return;
        }
    }
    TL3_LAUNCH(s, name, (k3_cg_w<F, R, U><<<grid, bl, 0, s->stream>>>(s->g, fc, beta, cu, p_in, p_out, r, w,
                                                                      chunk->vec_kx, chunk->vec_ky, chunk->vec_kz,
                                                                      u_halo, uhd, loop_slots(s, done), done, fin)));
}

// The fused CG u/r update (k3_cg_ur semantics), by TMA where possible
// (internal linkage as launch_cg_w3).
template <typename Finish>
static void launch_cg_ur3(TlSuite3D* s, dim3 grid, Scalar alpha, double* u, const double* p, double* r,
                          const double* w, const int* done, Finish fin)
{
    const dim3 bl = interior_block();
    if (tma_usable(s)) {
        const CUtensorMap* mu = tma_map(s, u, 4);
        const CUtensorMap* mp = tma_map(s, p, 4);
        const CUtensorMap* mr = tma_map(s, r, 4);
        const CUtensorMap* mw = tma_map(s, w, 4);
        if (mu && mp && mr && mw) {
            const Tma3UrMaps m{*mu, *mp, *mr, *mw};
            static unsigned attr_set = 0;   // devices on which the shared-memory size was raised
            if (!(attr_set & (1u << (s->device & 31)))) {
                TL_CUDA(cudaFuncSetAttribute(k3_cg_ur_tma<Finish>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kTmaUr3Bytes));
                attr_set |= 1u << (s->device & 31);
            }
            TL3_LAUNCH(s, "k3_cg_ur", (k3_cg_ur_tma<<<grid, bl, kTmaUr3Bytes, s->stream>>>(
                                          s->g, alpha, m, u, r, loop_slots(s, done), done, fin,
                                          s->d_mirror + kTmaErrWord)));
            return;
        }
    }
    TL3_LAUNCH(s, "k3_cg_ur", (k3_cg_ur<<<grid, bl, 0, s->stream>>>(s->g, alpha, u, p, r, w,
                                                                           loop_slots(s, done), done, fin)));
}

// The fused CG r update (k3_cg_r semantics), by TMA where possible.
template <typename Finish>
static void launch_cg_r3(TlSuite3D* s, dim3 grid, Scalar alpha, double* r, const double* w, const int* done, Finish fin)
{
    const dim3 bl = interior_block();
    if (tma_usable(s)) {
        const CUtensorMap* mr = tma_map(s, r, 4);
        const CUtensorMap* mw = tma_map(s, w, 4);
        if (mr && mw) {
            const Tma3RMaps m{*mr, *mw};
            static unsigned attr_set = 0;   // devices on which the shared-memory size was raised
            if (!(attr_set & (1u << (s->device & 31)))) {
                TL_CUDA(cudaFuncSetAttribute(k3_cg_r_tma<Finish>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kTmaR3Bytes));
                attr_set |= 1u << (s->device & 31);
            }
            TL3_LAUNCH(s, "k3_cg_r", (k3_cg_r_tma<<<grid, bl, kTmaR3Bytes, s->stream>>>(
                                         s->g, alpha, m, r, loop_slots(s, done), done, fin, s->d_mirror + kTmaErrWord)));
            return;
        }
    }
    TL3_LAUNCH(s, "k3_cg_r", (k3_cg_r<<<grid, bl, 0, s->stream>>>(s->g, alpha, r, w, loop_slots(s, done), done, fin)));
}

// The CG loop of a mesh that does not fit on chip, its solution in u: the w
// sweep of every second trip applies the u updates of the two trips before it
// (CgU), so p goes round three buffers, the third the suite's second sd buffer
// (unused by CG; cg_init has cleared its halo as p's). loop(trip) launches the
// trips trip(0), ... and returns the state they end in.
template <typename Loop>
static DevState cg_deferred3(TlSuite3D* s, Chunk* chunk, double* u, const DevParams& prm, Loop loop)
{
    double* buf[3] = {chunk->vec_p, s->alt[ALT3_P], s->alt[ALT3_SD]};   // trip t's p is buf[t % 3]
    const Faces fc = faces_of(chunk);
    const dim3 gi = interior_grid(s->g), gh = fused_grid(s->g);
    const int* done = &s->d_state->done;
    const tl::FinCgW fin_w{s->d_state, s->d_cg_alphas};
    const tl::FinCgUr fin_ur{s->d_state, s->d_cg_betas, prm, s->d_mirror};
    const Scalar beta{0.0, &s->d_state->beta}, alpha{0.0, &s->d_state->alpha};
    const DevState st = loop([&](int t) {
        double* const p = buf[t % 3];
        const double* const p1 = buf[(t + 2) % 3];
        if (t == 0)
            launch_cg_w3<false, false>(s, chunk, gh, fc, beta, p, p, chunk->vec_r, chunk->vec_w, nullptr, 0, done,
                                       fin_w);
        else if (t % 2 == 0)
            launch_cg_w3<true, true, true>(s, chunk, gh, fc, beta, p1, p, chunk->vec_r, chunk->vec_w, nullptr, 0, done,
                                           fin_w, CgU{u, buf[(t + 1) % 3], s->d_cg_alphas, t});
        else
            launch_cg_w3<true, true>(s, chunk, gh, fc, beta, p1, p, chunk->vec_r, chunk->vec_w, nullptr, 0, done,
                                     fin_w);
        launch_cg_r3(s, gi, alpha, chunk->vec_r, chunk->vec_w, done, fin_ur);
    });
    const int t = st.trip;   // trips that ran: t - 1 is the last
    if (t > 0) {
        TL3_LAUNCH(s, "k3_cg_u_close", (k3_cg_u_close<<<gi, interior_block(), 0, s->stream>>>(
                                           s->g, u, buf[(t + 1) % 3], buf[(t + 2) % 3], s->d_cg_alphas, t,
                                           t % 2 == 0 ? 1 : 0)));
        chunk->vec_p = buf[(t + 2) % 3];
        s->alt[ALT3_P] = buf[t % 3];
        s->alt[ALT3_SD] = buf[(t + 1) % 3];
    }
    return st;
}

// Tensor maps of a stencil sweep over operands a (and b) with the chunk's
// coefficients; false when the layout or an encoding rules TMA out.
static bool sweep_maps(TlSuite3D* s, Chunk* chunk, const double* a, const double* b, Tma3Maps* m)
{
    if (!tma_usable(s)) return false;
    const CUtensorMap* ma = tma_map(s, a, 0);
    const CUtensorMap* mb = b ? tma_map(s, b, 0) : ma;
    const CUtensorMap* kx = tma_map(s, chunk->vec_kx, 1);
    const CUtensorMap* ky = tma_map(s, chunk->vec_ky, 2);
    const CUtensorMap* kz = tma_map(s, chunk->vec_kz, 3);
    if (!(ma && mb && kx && ky && kz)) return false;
    *m = Tma3Maps{*ma, *mb, *kx, *ky, *kz};
    return true;
}

// Raises a TMA-fed kernel's dynamic shared-memory limit once per device
// (`set`: the caller's record of devices done).
template <typename Kernel>
static void raise_ring_smem(TlSuite3D* s, Kernel kernel, unsigned& set)
{
    if (set & (1u << (s->device & 31))) return;
    TL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTmaRingBytes));
    set |= 1u << (s->device & 31);
}
}  // namespace tl3d
