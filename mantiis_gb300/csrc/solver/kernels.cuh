// Kernels of the lattice Boltzmann step (sm_103a): the fused AA-pattern
// collide-and-stream, the output/residual pass, the coarse/fine interface
// exchange and the equilibrium initialisation.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "tma.cuh"

namespace mantiis
{
namespace dev
{
constexpr int kMaxLevels = 4;

struct AllLevels
{
    LevelView lv[kMaxLevels];
    int parity[kMaxLevels]; // parity of the next step of each level
    int direct[kMaxLevels]; // level holds f itself (no step since initialisation)
};

// Sum of two doubles over the block, then one atomic per block.
__device__ __forceinline__ void block_add2(double a, double b, double *dst)
{
    __shared__ double sa[32], sb[32];
    for (int o = 16; o > 0; o >>= 1)
    {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
    {
        sa[wid] = a;
        sb[wid] = b;
    }
    __syncthreads();
    if (wid == 0)
    {
        const int nw = blockDim.x >> 5;
        a = lane < nw ? sa[lane] : 0.0;
        b = lane < nw ? sb[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1)
        {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
        }
        if (lane == 0)
        {
            if (a != 0.0) atomicAdd(dst, a);
            if (b != 0.0) atomicAdd(dst + 1, b);
        }
    }
    __syncthreads();
}

// Loads the populations of a cell of level view L for a step (or a read) at
// parity P.  Returns 1/tau_s and, for special cells, a copy of the record.
template <int P>
__device__ __forceinline__ float load_cell(const LevelView &L, const Common &C, int x, int y, int direct, int first_sub,
                                           float df[9], bool &special, SpecialRec &rec)
{
    const int64_t s = site_of(L, x, y);
    float om = L.omega[s];
    special = om < 0.0f;
    if (!special)
    {
        if (direct) load_raw<0>(L, x, y, df);
        else load_raw<P>(L, x, y, df);
        return om;
    }
    rec = C.specials[L.spec[s]];
    const uint32_t flags = (rec.m1 >> 17) & 0xFu;
    if ((flags & SF_BUFFER) && (first_sub || direct))
    {
#pragma unroll
        for (int q = 0; q < 9; q++) df[q] = C.ibuf[(size_t)q * C.n_buf + rec.buf];
    }
    else if (direct)
        load_raw<0>(L, x, y, df);
    else
        load_special<P>(L, C, rec, x, y, df);
    return -om;
}

// The coarse-step-start moments (drho, u_x, u_y) of site s.  In a launch that
// uses them nothing writes them (phase 0 stored them), so the step kernels may
// take the read-only path (NC); the persistent step, where phase 0 ran earlier
// in the same launch, takes ordinary loads.
template <bool NC> __device__ __forceinline__ void load_snap(const LevelView &L, int64_t s, float sn[3])
{
    sn[0] = ldf<NC>(&L.snap[s]);
    sn[1] = ldf<NC>(&L.snap[L.plane + s]);
    sn[2] = ldf<NC>(&L.snap[2 * L.plane + s]);
}

// Collision of one cell with the populations df: equilibrium of the moments
// edrho, erho, eux, euy (the cell's own, or those of the coarse step's start),
// regularized MRT / MRT / BGK, the wall values of special cells
// (include/coreLB.hpp:420-430, 646-792, 834-977).  fs: the populations to stream.
__device__ __forceinline__ void collide_cell(const LevelView &L, const Common &C, int collision, int wall_mode, int parity,
                                             int64_t s, const float df[9], float edrho, float erho, float eux, float euy,
                                             float omega, bool special, const SpecialRec &rec, float fs[9])
{
    float feq[9];
    equilibrium(edrho, erho, eux, euy, feq);
    if (collision == COLL_RMRT) collide_rmrt(df, feq, edrho, erho, eux, euy, omega, fs);
    else if (collision == COLL_MRT) collide_mrt(df, feq, mrt_rates(1.0f / omega, L.tau2 ? L.tau2[s] : 1.0f), fs);
    else
    {
        const float inv_tau = 1.0f; // 1 / tau_SRT, tau_SRT = 1 (include/globalParameters.hpp:140)
#pragma unroll
        for (int q = 0; q < 9; q++) fs[q] = df[q] - inv_tau * (df[q] - feq[q]);
    }
    if (special)
    {
        const uint32_t wall = (rec.m0 >> 18) & 0x1FFu, quirk = rec.m1 & 0x1FFu;
        if (wall && wall_mode == WALL_MDBB)
        {
            // include/coreLB.hpp:936-967: reflected value
            //   r f*_q + (1 - r) (sum_{c.n<0} f / sum_{c.n>0} f_eq) f_eq,opp(q)
            // in deviation form; both sums share the weight total A.
            const uint32_t bnd = (rec.m1 >> 9) & 0xFFu;
            const uint32_t pos = bnd == 0xFFu ? 0u : c_npos[bnd], neg = bnd == 0xFFu ? 0u : c_nneg[bnd];
            float a = 0.f, ap = 0.f, A = 0.f;
#pragma unroll
            for (int q = 0; q < 9; q++)
            {
                if ((neg >> q) & 1u) a += df[q];
                if ((pos >> q) & 1u)
                {
                    ap += feq[q];
                    A += wq(q) * C.rho0;
                }
            }
            const float g = (A + ap) != 0.f ? (a - ap) / (A + ap) : 0.f;
            const float r = rec.r;
#pragma unroll
            for (int q = 0; q < 9; q++)
                if ((wall >> q) & 1u)
                {
                    const int po = d2q9::opp(q);
                    fs[q] = r * fs[q] + (1.0f - r) * (feq[po] + (wq(po) * C.rho0 + feq[po]) * g);
                }
        }
        if (quirk)
        {
            float *side_now = C.side + (size_t)parity * C.n_quirk;
            int qi = 0;
#pragma unroll
            for (int q = 0; q < 9; q++)
                if ((quirk >> q) & 1u) side_now[rec.quirk_base + qi++] = fs[q];
        }
    }
}

// Collision and streaming of one cell whose populations df are loaded:
// macroscopic moments (and the residual / snapshot side outputs), equilibrium,
// regularized MRT / MRT / BGK collision, the wall values of special cells and
// the AA-pattern store (include/coreLB.hpp:420-430, 646-792, 834-977, 1018-1054).
template <int P>
__device__ __forceinline__ void step_cell(const LevelView &L, const Common &C, const StepOpt &o, int diff, int store_u,
                                          int x, int y, int64_t s, const float df[9], float omega, bool special,
                                          const SpecialRec &rec, double &r_diff, double &r_norm, bool interior = false,
                                          const float *unorm_prev = nullptr, const float *snap_prev = nullptr)
{
    float drho, rho, ux, uy;
    macro(df, C.rho0, L.fshift, 0.0f, drho, rho, ux, uy);
    if (diff | store_u)
    {
        const float un = sqrtf(ux * ux + uy * uy);
        if (diff)
        {
            r_diff = (double)fabsf(un - (unorm_prev ? *unorm_prev : L.unorm[s]));
            r_norm = (double)un;
        }
        if (store_u) L.unorm[s] = un;
    }
    if (o.snap_store)
    {
        L.snap[s] = drho;
        L.snap[L.plane + s] = ux;
        L.snap[2 * L.plane + s] = uy;
    }
    float edrho = drho, erho = rho, eux = ux, euy = uy;
    if (o.snap_use)
    {
        // the coarse-step-start moments: loaded by the caller with the populations
        // where it can (a load here is one more dependent round trip per cell)
        edrho = snap_prev ? snap_prev[0] : L.snap[s];
        erho = C.rho0 + edrho;
        eux = snap_prev ? snap_prev[1] : L.snap[L.plane + s];
        euy = snap_prev ? snap_prev[2] : L.snap[2 * L.plane + s];
    }
    float fs[9];
    collide_cell(L, C, C.collision, C.wall, P, s, df, edrho, erho, eux, euy, omega, special, rec, fs);
    store_post<P>(L, x, y, fs, interior);
}

// Plain cells of one active tile (all nine populations stream in, no wall
// link): one thread per site of a 32x8 tile, the row masks of plain cells let
// the relaxation rate and the nine populations load together.  Each slot a
// thread reads is written by that thread alone in this launch (AA ownership),
// so the loads take the read-only path.  Special cells (walls, missing
// arrivals, buffers) go to their own kernel: in the same warps their longer
// path would hold the plain lanes.
template <int P>
__device__ __forceinline__ void plain_tile(const LevelView &L, const Common &C, const StepOpt &o, int t, int diff,
                                           int store_u, double &r_diff, double &r_norm)
{
    // the tile id and this row's plain-cell mask are independent loads
    const int tile = __ldg(&L.tiles[t]); // tx | ty << 16
    const uint32_t mask = __ldg(&L.tile_mask[t * 8 + (threadIdx.x >> 5)]);
    const int tx = tile & 0xFFFF, ty = tile >> 16;
    const int x = tx * 32 + (threadIdx.x & 31);
    const int y = ty * 8 + (threadIdx.x >> 5);
    // tiles off the border reach their neighbours without wrapping
    const bool interior = tx > 0 && tx + 1 < L.tiles_x && ty > 0 && ty + 1 < (L.H + 7) / 8;
    if ((mask >> (threadIdx.x & 31)) & 1u)
    {
        const int64_t s = site_of(L, x, y);
        // (a "direct" state is read like an even step: own slots)
        float df[9], sn[3] = {0.f, 0.f, 0.f};
        const float uprev = diff ? __ldg(&L.unorm[s]) : 0.0f; // with the populations, as in plain_tile8
        if (o.snap_use) load_snap<true>(L, s, sn);
        load_raw_ro<P>(L, x, y, df, interior);
        const float om = __ldg(&L.omega[s]);
        SpecialRec none;
        step_cell<P>(L, C, o, diff, store_u, x, y, s, df, om, false, none, r_diff, r_norm, interior, &uprev,
                     o.snap_use ? sn : nullptr);
    }
}

// Populations of a light cell (special only through missing arrivals and buffer
// status) from the slots it reads
__device__ __forceinline__ void light_rules(const Common &C, const SpecialRec &rec, float df[9])
{
    const uint32_t arrive = rec.m0 & 0x1FFu;
    const bool has_k = ((rec.m1 >> 17) & SF_HAS_K) != 0;
    const float *k = C.ktab + (size_t)(has_k ? rec.k_row : 0) * 9;
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        float v = ((arrive >> q) & 1u) ? df[q] : 0.0f;
        if (has_k) v += __ldg(&k[q]);
        df[q] = v;
    }
}

// Plain cells of one 8x4 tile, one warp per tile (lane = 8 * row + column):
// the same cell update as plain_tile; on sparse levels these tiles hold a
// larger share of active cells than 32x8 tiles, so fewer lanes idle and fewer
// sectors are fetched for inactive sites.  The tile's light cells (special only
// through missing arrivals and buffer status: most of the interface ring of a
// finer level) are stepped here too, with the reads of special_cell for such a
// record (interpolated values at the first substep, else the arrivals plus the
// constant row), so the special-cell kernel keeps only the cells with walls.
template <int P, bool NC = true>
__device__ __forceinline__ void plain_tile8(const LevelView &L, const Common &C, const StepOpt &o, int t, int diff,
                                            int store_u, double &r_diff, double &r_norm)
{
    const int lane = threadIdx.x & 31;
    const int tile = __ldg(&L.tiles8[t]); // tx | ty << 16, in 8- and 4-site units
    const uint32_t mask = __ldg(&L.tile8_mask[t]);
    if (!((mask >> lane) & 1u)) return;
    const bool light = (__ldg(&L.tile8_light[t]) >> lane) & 1u;
    const int tx = tile & 0xFFFF, ty = tile >> 16;
    const int x = tx * 8 + (lane & 7), y = ty * 4 + (lane >> 3);
    // tiles off the border reach their neighbours without wrapping
    const bool interior = tx > 0 && tx + 1 < (L.W + 7) / 8 && ty > 0 && ty + 1 < (L.H + 3) / 4;
    const int64_t s = site_of(L, x, y);
    float df[9];
    float om;
    // the |u| the residual compares with, loaded with the populations (the
    // cell's own site: this thread alone writes it, after reading it)
    const float uprev = diff ? ldf<NC>(&L.unorm[s]) : 0.0f;
    float sn[3] = {0.f, 0.f, 0.f};
    if (o.snap_use) load_snap<NC>(L, s, sn);
    if (!light)
    {
        load_raw_ro<P, NC>(L, x, y, df, interior);
        om = __ldg(&L.omega[s]);
    }
    else
    {
        const SpecialRec rec = C.specials[__ldg(&L.spec[s])];
        const uint32_t flags = (rec.m1 >> 17) & 0xFu;
        om = rec.omega;
        if ((flags & SF_BUFFER) && (o.first_sub || o.direct))
        {
#pragma unroll
            for (int q = 0; q < 9; q++) df[q] = C.ibuf[(size_t)q * C.n_buf + rec.buf];
        }
        else
        {
            // a direct state has parity 0: own slots, as load_raw<0>
            load_raw_ro<P, NC>(L, x, y, df, interior);
            if (!o.direct) light_rules(C, rec, df);
        }
    }
    SpecialRec none;
    step_cell<P>(L, C, o, diff, store_u, x, y, s, df, om, false, none, r_diff, r_norm, interior, &uprev,
                 o.snap_use ? sn : nullptr);
}

// One special cell (wall links, missing arrivals, interface buffer, inlet /
// outlet) from its record.
template <int P>
__device__ __forceinline__ void special_cell(const LevelView &L, const Common &C, const StepOpt &o, int64_t i, int diff,
                                             int store_u, double &r_diff, double &r_norm)
{
    const SpecialRec rec = C.specials[i];
    const int x = rec.xy & 0xFFFF, y = rec.xy >> 16;
    const int64_t s = site_of(L, x, y);
    // the |u| the residual compares with, in flight with the populations
    const float uprev = diff ? L.unorm[s] : 0.0f;
    float sn[3] = {0.f, 0.f, 0.f};
    if (o.snap_use) load_snap<false>(L, s, sn);
    float df[9];
    const uint32_t flags = (rec.m1 >> 17) & 0xFu;
    if ((flags & SF_BUFFER) && (o.first_sub || o.direct))
    {
#pragma unroll
        for (int q = 0; q < 9; q++) df[q] = C.ibuf[(size_t)q * C.n_buf + rec.buf];
    }
    else if (o.direct)
        load_raw<0>(L, x, y, df);
    else
        load_special<P>(L, C, rec, x, y, df);
    step_cell<P>(L, C, o, diff, store_u, x, y, s, df, rec.omega, true, rec, r_diff, r_norm, false, &uprev,
                 o.snap_use ? sn : nullptr);
}

// ---- phase kernels.  A coarse time step is a sequence of phases; a phase
// steps every (image, level) whose next substep falls on it.  All levels of an
// image are independent within a coarse step (they meet only in the interface
// exchange that closes it), so one launch covers them all.  The descriptors
// travel in the launch parameters: each owns a contiguous block range, so the
// descriptor index and its fields are block-uniform.

// One (image, level) in one phase: where its state is and how to step it.
struct StepDesc
{
    LevelView L;
    Common C;
    StepOpt o;
    int64_t spec_begin; // the level's special records
    int spec_count;
    int tile_base;      // first tile of the level's list this descriptor covers
};

// Per-launch residual switches: the residual terms (and the |u| store) apply
// to the first substep of each level, which falls on phase 0.
struct PhaseArgs
{
    int diff, store_u, red_slot;
};

constexpr int kMaxPhaseDescs = 24;

struct PhaseLaunch
{
    int ndesc;
    int start[kMaxPhaseDescs + 1]; // first block of each descriptor; start[ndesc] = blocks
    int grid;                      // blocks launched (k_phase_plain8: may be fewer; they loop)
    PhaseArgs a;
    StepDesc d[kMaxPhaseDescs];
};

// descriptor owning block b (block-uniform)
__device__ __forceinline__ int owner(const int *start, int n, int b)
{
    int j = 0;
#pragma unroll 1
    while (j + 1 < n && b >= start[j + 1]) j++;
    return j;
}

// plain cells with direct loads: blocks of a descriptor walk its tiles
__global__ void __launch_bounds__(256, 5) k_phase_plain(const __grid_constant__ PhaseLaunch P)
{
    const int j = owner(P.start, P.ndesc, (int)blockIdx.x);
    const StepDesc &d = P.d[j];
    const int t = d.tile_base + (int)blockIdx.x - P.start[j];
    const int diff = P.a.diff & d.o.first_sub, store_u = P.a.store_u & d.o.first_sub;
    double r_diff = 0.0, r_norm = 0.0;
    if (d.o.parity) plain_tile<1>(d.L, d.C, d.o, t, diff, store_u, r_diff, r_norm);
    else plain_tile<0>(d.L, d.C, d.o, t, diff, store_u, r_diff, r_norm);
    if (diff) block_add2(r_diff, r_norm, d.C.red + P.a.red_slot);
}

// plain cells in 8x4 tiles: 8 tiles (warps) per block-sized unit of work; a
// block walks units blockIdx.x, blockIdx.x + gridDim.x, ...  Alone the launch
// has a block per unit; when other images' kernels run beside it (batch
// streams) it has at most 4 blocks per SM, so they find room on every SM.
__global__ void __launch_bounds__(256, 5) k_phase_plain8(const __grid_constant__ PhaseLaunch P)
{
    const int units = P.start[P.ndesc];
    for (int u = (int)blockIdx.x; u < units; u += (int)gridDim.x)
    {
        const int j = owner(P.start, P.ndesc, u);
        const StepDesc &d = P.d[j];
        const int t = (u - P.start[j]) * 8 + (int)(threadIdx.x >> 5);
        const int diff = P.a.diff & d.o.first_sub, store_u = P.a.store_u & d.o.first_sub;
        double r_diff = 0.0, r_norm = 0.0;
        if (t < d.L.ntiles8)
        {
            if (d.o.parity) plain_tile8<1>(d.L, d.C, d.o, t, diff, store_u, r_diff, r_norm);
            else plain_tile8<0>(d.L, d.C, d.o, t, diff, store_u, r_diff, r_norm);
        }
        if (diff) block_add2(r_diff, r_norm, d.C.red + P.a.red_slot);
    }
}

// special cells: blocks of a descriptor walk its records, kSpecialBlock per block
// special records per block of k_phase_special (64 and 32 measured slower: config-2
// batch 338 / 343 / 353 us per coarse step for 128 / 64 / 32)
constexpr int kSpecialBlock = 128;

__global__ void __launch_bounds__(kSpecialBlock) k_phase_special(const __grid_constant__ PhaseLaunch P)
{
    const int j = owner(P.start, P.ndesc, (int)blockIdx.x);
    const StepDesc &d = P.d[j];
    const int i = ((int)blockIdx.x - P.start[j]) * kSpecialBlock + (int)threadIdx.x;
    const int diff = P.a.diff & d.o.first_sub, store_u = P.a.store_u & d.o.first_sub;
    double r_diff = 0.0, r_norm = 0.0;
    if (i < d.spec_count)
    {
        if (d.o.parity) special_cell<1>(d.L, d.C, d.o, d.spec_begin + i, diff, store_u, r_diff, r_norm);
        else special_cell<0>(d.L, d.C, d.o, d.spec_begin + i, diff, store_u, r_diff, r_norm);
    }
    if (diff) block_add2(r_diff, r_norm, d.C.red + P.a.red_slot);
}

// ---- plain cells through a TMA pipeline.  A persistent block walks the
// x-interior tiles of its descriptors; for each tile one bulk tensor copy
// brings the 9 planes with a halo of 4 columns and 1 row (a 40 x 10 x 9 box,
// x start 16-byte aligned), a second the tile's 32 x 8 relaxation rates and a
// bulk copy its 8 row masks into shared memory, two tiles ahead of the one
// being stepped.  Cells read their slots from shared memory (odd steps index
// the shifted neighbours there) and store as in plain_tile.
constexpr int kTmaW = 40, kTmaH = 10, kTmaStages = 2;
constexpr uint32_t kTmaFBytes = kTmaW * kTmaH * 9 * 4;
constexpr uint32_t kTmaOmOff = (kTmaFBytes + 127) / 128 * 128; // 128-byte aligned
constexpr uint32_t kTmaMaskOff = kTmaOmOff + 32 * 8 * 4;
constexpr uint32_t kTmaTxBytes = kTmaFBytes + 32 * 8 * 4 + 32;         // bytes the copies of one tile deliver
constexpr uint32_t kTmaStageBytes = (kTmaMaskOff + 32 + 127) / 128 * 128; // stage stride
constexpr int kMaxTmaDescs = 8;
constexpr uint32_t kWaitPolls = 1u << 26;

struct TmaLaunch
{
    CUtensorMap map[kMaxTmaDescs];    // per descriptor: its level's 9 planes as (x, y, q)
    CUtensorMap om_map[kMaxTmaDescs]; // per descriptor: its level's relaxation rates as (x, y)
    int grid;                         // persistent blocks of the launch (host side)
    int ndesc;
    int start[kMaxTmaDescs + 1];      // first tile (in launch order) of each descriptor
    PhaseArgs a;
    StepDesc d[kMaxTmaDescs];
};

template <int P>
__device__ __forceinline__ void plain_tile_smem(const LevelView &L, const Common &C, const StepOpt &o, int tile,
                                                const unsigned char *stage, int diff, int store_u, double &r_diff,
                                                double &r_norm)
{
    const float *sb = reinterpret_cast<const float *>(stage);
    const float *som = reinterpret_cast<const float *>(stage + kTmaOmOff);
    const uint32_t *smask = reinterpret_cast<const uint32_t *>(stage + kTmaMaskOff);
    const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
    if (!((smask[ly] >> lx) & 1u)) return;
    const int x = (tile & 0xFFFF) * 32 + lx, y = (tile >> 16) * 8 + ly;
    const int64_t s = site_of(L, x, y);
    const float om = som[ly * 32 + lx];
    const float uprev = diff ? L.unorm[s] : 0.0f;
    float sn[3] = {0.f, 0.f, 0.f};
    if (o.snap_use) load_snap<true>(L, s, sn);
    float df[9];
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        // even: own slot (x, q); odd: slot (x - c_q, opp q)
        const int pq = P == 0 ? q : d2q9::opp(q);
        const int sy = ly + 1 - (P == 0 ? 0 : d2q9::cy(q)), sx = lx + 4 - (P == 0 ? 0 : d2q9::cx(q));
        df[q] = sb[(pq * kTmaH + sy) * kTmaW + sx];
    }
    SpecialRec none;
    step_cell<P>(L, C, o, diff, store_u, x, y, s, df, om, false, none, r_diff, r_norm, true, &uprev,
                 o.snap_use ? sn : nullptr);
}

__global__ void __launch_bounds__(256, 4) k_phase_plain_tma(const __grid_constant__ TmaLaunch P)
{
    __shared__ __align__(128) unsigned char sbuf[kTmaStages][kTmaStageBytes];
    __shared__ __align__(8) uint64_t full[kTmaStages];
    __shared__ int s_tile[kTmaStages];
    __shared__ int s_fail;
    static_assert(kTmaStageBytes % 128 == 0 && kTmaOmOff % 128 == 0 && kTmaMaskOff % 16 == 0, "stage layout");
    const int total = P.start[P.ndesc];
    if (threadIdx.x == 0)
    {
        for (int st = 0; st < kTmaStages; st++) mbar_init(&full[st], 1);
        s_fail = 0;
        fence_barrier_init();
    }
    __syncthreads();
    auto issue = [&](int g, int st) {
        const int j = owner(P.start, P.ndesc, g);
        const int t = P.d[j].tile_base + g - P.start[j];
        const int tile = P.d[j].L.tiles[t];
        const int x0 = (tile & 0xFFFF) * 32, y0 = (tile >> 16) * 8;
        s_tile[st] = tile;
        mbar_arrive_expect_tx(&full[st], kTmaTxBytes);
        tma_load_3d(sbuf[st], &P.map[j], x0 - 4, y0 - 1, 0, &full[st]);
        tma_load_2d(sbuf[st] + kTmaOmOff, &P.om_map[j], x0, y0, &full[st]);
        bulk_load(sbuf[st] + kTmaMaskOff, P.d[j].L.tile_mask + (size_t)t * 8, 32, &full[st]);
    };
    if (threadIdx.x == 0)
        for (int st = 0; st < kTmaStages; st++)
        {
            const int g = (int)blockIdx.x + st * (int)gridDim.x;
            if (g < total) issue(g, st);
        }
    double r_diff = 0.0, r_norm = 0.0;
    int red_desc = -1;
    int it = 0;
    for (int g = (int)blockIdx.x; g < total; g += (int)gridDim.x, it++)
    {
        const int st = it % kTmaStages;
        const uint32_t parity = (uint32_t)(it / kTmaStages) & 1u;
        if (!mbar_wait_bounded(&full[st], parity, kWaitPolls)) atomicOr(&s_fail, 1);
        __syncthreads();
        if (s_fail) break;
        const int j = owner(P.start, P.ndesc, g);
        const StepDesc &d = P.d[j];
        const int diff = P.a.diff & d.o.first_sub, store_u = P.a.store_u & d.o.first_sub;
        if (diff) red_desc = j;
        const int tile = s_tile[st];
        double t_diff = 0.0, t_norm = 0.0; // this tile's terms
        if (d.o.parity) plain_tile_smem<1>(d.L, d.C, d.o, tile, sbuf[st], diff, store_u, t_diff, t_norm);
        else plain_tile_smem<0>(d.L, d.C, d.o, tile, sbuf[st], diff, store_u, t_diff, t_norm);
        r_diff += t_diff;
        r_norm += t_norm;
        // every thread is done with this stage before it is refilled
        __syncthreads();
        if (threadIdx.x == 0)
        {
            const int gn = g + kTmaStages * (int)gridDim.x;
            if (gn < total) issue(gn, st);
        }
    }
    if (s_fail)
    {
        if (threadIdx.x == 0)
        {
            atomicOr(P.d[0].C.err, kErrTmaTimeout);
            // let copies still in flight land before the block's shared memory goes
            for (int st = 0; st < kTmaStages; st++) mbar_wait_bounded(&full[st], 0u, 1024u);
        }
        return;
    }
    // residual terms: only single-image launches ask for them (one accumulator)
    if (P.a.diff)
    {
        const int rd = __syncthreads_or(red_desc >= 0) ? 0 : -1;
        if (rd == 0) block_add2(r_diff, r_norm, P.d[0].C.red + P.a.red_slot);
    }
}

// Maximum of a non-negative float over the block, then one atomic per block on
// the double it converts to: the conversion is exact and monotone, so this is
// the maximum of the converted values, with the shuffles on the FP32 pipe
// (non-negative doubles order like their bit patterns).
__device__ __forceinline__ void block_max(float v, double *dst)
{
    __shared__ float sm[32];
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sm[wid] = v;
    __syncthreads();
    if (wid == 0)
    {
        const int nw = blockDim.x >> 5;
        v = lane < nw ? sm[lane] : 0.0f;
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
        if (lane == 0 && v > 0.0f)
            atomicMax(reinterpret_cast<unsigned long long *>(dst), (unsigned long long)__double_as_longlong((double)v));
    }
    __syncthreads();
}

// Adsorption, first pass of a step (include/mantiisApp.hpp:248-252,
// include/coreLB.hpp:1056-1067, 515-531, 1269-1283): density of every cell from
// its streamed populations, its pseudopotential, and the relative density change
// since the previous step (maximum over the cells).
// density and pseudopotential of one cell (pass 1), the density change against
// the previous step's density for the residual
template <int P, bool SPEC>
__device__ __forceinline__ float ads_density(const LevelView &L, const Common &C, const StepOpt &o, int x, int y)
{
    const int64_t s = site_of(L, x, y);
    float df[9];
    if (SPEC)
    {
        bool special;
        SpecialRec rec;
        load_cell<P>(L, C, x, y, o.direct, o.first_sub, df, special, rec);
    }
    else if (o.direct)
        load_raw<0>(L, x, y, df);
    else
        load_raw<P>(L, x, y, df);
    float drho = 0.0f;
#pragma unroll
    for (int q = 0; q < 9; q++) drho += df[q];
    const float rho = C.rho0 + drho;
    L.psi[s] = pseudo_potential((float)C.psi_form, C.psi_rho0, C.eos_a, C.eos_b, C.eos_T, C.g_ff, rho);
    const float old = L.rho_prev[s];
    L.rho_prev[s] = rho;
    return fabsf(rho - old) / old;
}

// pass 1 over the plain cells of active 32x8 tile t (row masks): one block
template <int P> __device__ __forceinline__ float ads_psi_tile(const LevelView &L, const Common &C, const StepOpt &o, int t)
{
    const int tile = L.tiles[t]; // tx | ty << 16
    const uint32_t mask = L.tile_mask[t * 8 + (threadIdx.x >> 5)];
    const int x = (tile & 0xFFFF) * 32 + (threadIdx.x & 31);
    const int y = (tile >> 16) * 8 + (threadIdx.x >> 5);
    return ((mask >> (threadIdx.x & 31)) & 1u) ? ads_density<P, false>(L, C, o, x, y) : 0.0f;
}

// pass 1 of special record i of the level (i < spec_count)
template <int P>
__device__ __forceinline__ float ads_psi_record(const LevelView &L, const Common &C, const StepOpt &o, int64_t rec)
{
    const int32_t xy = C.specials[rec].xy;
    return ads_density<P, true>(L, C, o, xy & 0xFFFF, xy >> 16);
}

template <int P> __global__ void __launch_bounds__(256) k_ads_psi(LevelView L, Common C, StepOpt o)
{
    const float rmax = ads_psi_tile<P>(L, C, o, (int)blockIdx.x);
    if (o.diff) block_max(rmax, C.red + o.red_slot);
}

// pass 1 over the special cells, from their records (128 per block)
template <int P> __global__ void __launch_bounds__(128) k_ads_psi_special(LevelView L, Common C, StepOpt o,
                                                                          int64_t spec_begin, int spec_count)
{
    const int i = (int)blockIdx.x * 128 + (int)threadIdx.x;
    const float rmax = i < spec_count ? ads_psi_record<P>(L, C, o, spec_begin + i) : 0.0f;
    if (o.diff) block_max(rmax, C.red + o.red_slot);
}

// Adsorption, second pass: Shan-Chen force (include/coreLB.hpp:533-566),
// velocity with the half-force shift (:1069-1099), equilibrium, plain MRT
// (:694-742), Guo source term (:568-630), AA store.  Bounce-back walls, the
// x-periodic links and the inlet/outlet overwrite (:859-865, 969-1009) are
// applied when the populations are read in the next step.
// The coupling phase of the coupled run (include/mantiisApp.hpp:267-284) takes
// the same body with the regularized MRT, SRBB walls, no inlet / outlet and the
// velocity residual (C.collision, C.wall, C.inlet_outlet; o.diff accumulates
// sum |u| for both terms, as its |u| of the previous step is never stored).
// psi[r][c]: the pseudopotential at (x + c - 1, y + r - 1); df: the cell's
// populations, mr its relaxation rates (omega: 1/tau_s for the regularized
// MRT); special: its record applies.
template <int P>
__device__ __forceinline__ void ads_update(const LevelView &L, const Common &C, const StepOpt &o, int x, int y,
                                           const float df[9], float omega, const MrtRates &mr, bool special,
                                           const SpecialRec &rec, const float psi[3][3], double &r_diff, double &r_norm,
                                           bool interior = false)
{
    const int64_t s = site_of(L, x, y);
    const uint32_t out = special ? ((rec.m1 >> 21) & 0x1FFu) : 0x1FFu;
    const uint32_t wall = special ? ((rec.m0 >> 18) & 0x1FFu) : 0u;
    // sum over the streaming links of w_f psi(x + c) c, formed from psi differences
    const float psx = psi[1][1];
    float sx = 0.f, sy = 0.f, cwx = 0.f, cwy = 0.f, wwx = 0.f, wwy = 0.f;
#pragma unroll
    for (int q = 1; q < 9; q++)
    {
        const float w = (float)d2q9::wf(q);
        if ((out >> q) & 1u)
        {
            const float dpsi = psi[1 + d2q9::cy(q)][1 + d2q9::cx(q)] - psx;
            sx += w * dpsi * (float)d2q9::cx(q);
            sy += w * dpsi * (float)d2q9::cy(q);
            cwx += w * (float)d2q9::cx(q);
            cwy += w * (float)d2q9::cy(q);
        }
        if ((wall >> q) & 1u)
        {
            wwx += w * (float)d2q9::cx(q);
            wwy += w * (float)d2q9::cy(q);
        }
    }
    const float kff = -6.0f * C.g_ff * psx;
    const float Fx = kff * (sx + psx * cwx) - C.g_fs * psx * psx * wwx + C.fbody;
    const float Fy = kff * (sy + psx * cwy) - C.g_fs * psx * psx * wwy;
    float drho = 0.0f, jx = 0.0f, jy = 0.0f;
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        drho += df[q];
        jx += (float)d2q9::cx(q) * df[q];
        jy += (float)d2q9::cy(q) * df[q];
    }
    const float rho = C.rho0 + drho;
    const float ux = (jx + 0.5f * Fx) / rho, uy = (jy + 0.5f * Fy) / rho;
    if (o.snap_store)
    {
        L.snap[s] = drho;
        L.snap[L.plane + s] = ux;
        L.snap[2 * L.plane + s] = uy;
    }
    if (o.diff)
    {
        const float un = sqrtf(ux * ux + uy * uy);
        r_diff = (double)un;
        r_norm = (double)un;
    }
    float feq[9], fs[9];
    equilibrium(drho, rho, ux, uy, feq);
    if (C.collision == COLL_RMRT) collide_rmrt(df, feq, drho, rho, ux, uy, omega, fs);
    else collide_mrt(df, feq, mr, fs);
    add_source(fs, ux, uy, Fx, Fy, mr);
    if (special && (rec.m1 & 0x1FFu))
    {
        const uint32_t quirk = rec.m1 & 0x1FFu;
        float *side_now = C.side + (size_t)P * C.n_quirk;
        int qi = 0;
#pragma unroll
        for (int q = 0; q < 9; q++)
            if ((quirk >> q) & 1u) side_now[rec.quirk_base + qi++] = fs[q];
    }
    store_post<P>(L, x, y, fs, interior);
}

// The same of a cell whose populations are loaded here.  SPEC: the cell may be
// special, else it is a plain cell.
template <int P, bool SPEC>
__device__ __forceinline__ void ads_cell(const LevelView &L, const Common &C, const StepOpt &o, int x, int y,
                                         const float psi[3][3], double &r_diff, double &r_norm)
{
    const int64_t s = site_of(L, x, y);
    float df[9];
    bool special = false;
    SpecialRec rec;
    float omega;
    if (SPEC) omega = load_cell<P>(L, C, x, y, o.direct, o.first_sub, df, special, rec);
    else
    {
        if (o.direct) load_raw<0>(L, x, y, df);
        else load_raw<P>(L, x, y, df);
        omega = L.omega[s];
    }
    ads_update<P>(L, C, o, x, y, df, omega, mrt_rates(1.0f / omega, L.tau2[s]), special, rec, psi, r_diff, r_norm);
}

// Pass 2 over the plain cells of active 32x8 tile t: one block.  The
// neighbour pseudopotentials come by warp shuffles: a warp holds one row of
// the tile, each lane loads psi of its column in the rows y-1, y, y+1
// (coalesced), and takes the x-neighbours from the adjacent lanes; the lanes at
// the ends of the row (and the last image column) load their outer neighbours.
template <int P>
__device__ __forceinline__ void ads_step_tile(const LevelView &L, const Common &C, const StepOpt &o, int t, double &r_diff,
                                              double &r_norm)
{
    const int tile = L.tiles[t]; // tx | ty << 16
    const int lane = threadIdx.x & 31;
    const int x = (tile & 0xFFFF) * 32 + lane;
    const int y = (tile >> 16) * 8 + (threadIdx.x >> 5);
    const bool inside = x < L.W && y < L.H;
    float psi[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
    {
        const int yr = wrapx(y + r - 1, L.H);
        psi[r][1] = inside ? L.psi[site_of(L, x, yr)] : 0.0f;
        psi[r][0] = __shfl_up_sync(0xffffffffu, psi[r][1], 1);
        psi[r][2] = __shfl_down_sync(0xffffffffu, psi[r][1], 1);
        if (inside && lane == 0) psi[r][0] = L.psi[site_of(L, wrapx(x - 1, L.W), yr)];
        if (inside && (lane == 31 || x + 1 == L.W)) psi[r][2] = L.psi[site_of(L, wrapx(x + 1, L.W), yr)];
    }
    const uint32_t mask = L.tile_mask[t * 8 + (threadIdx.x >> 5)];
    if ((mask >> lane) & 1u) ads_cell<P, false>(L, C, o, x, y, psi, r_diff, r_norm);
}

// pass 2 of special record rec; the neighbour pseudopotentials are read directly
template <int P>
__device__ __forceinline__ void ads_step_record(const LevelView &L, const Common &C, const StepOpt &o, int64_t rec,
                                                double &r_diff, double &r_norm)
{
    const int32_t xy = C.specials[rec].xy;
    const int x = xy & 0xFFFF, y = xy >> 16;
    float psi[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++)
            psi[r][c] = L.psi[site_of(L, wrapx(x + c - 1, L.W), wrapx(y + r - 1, L.H))];
    ads_cell<P, true>(L, C, o, x, y, psi, r_diff, r_norm);
}

template <int P> __global__ void __launch_bounds__(256) k_ads_step(LevelView L, Common C, StepOpt o)
{
    double r_diff = 0.0, r_norm = 0.0;
    ads_step_tile<P>(L, C, o, (int)blockIdx.x, r_diff, r_norm);
    if (o.diff) block_add2(r_diff, r_norm, C.red + o.red_slot);
}

// pass 2 over the special cells, from their records (128 per block)
template <int P> __global__ void __launch_bounds__(128) k_ads_step_special(LevelView L, Common C, StepOpt o,
                                                                           int64_t spec_begin, int spec_count)
{
    const int i = (int)blockIdx.x * 128 + (int)threadIdx.x;
    double r_diff = 0.0, r_norm = 0.0;
    if (i < spec_count) ads_step_record<P>(L, C, o, spec_begin + i, r_diff, r_norm);
    if (o.diff) block_add2(r_diff, r_norm, C.red + o.red_slot);
}

// Reads the current state of every reference cell (no update): FP64 density,
// velocity and populations in reference cell order, plus the residual terms
// against the stored |u| and the pixel-area sums of u_x and rho.
__global__ void __launch_bounds__(256) k_cells(AllLevels A, Common C, const int32_t *cell_level, const int32_t *cell_site,
                                               const uint8_t *cell_buffer, int64_t n, double *rho_out, double *ux_out,
                                               double *uy_out, double *f_out, int diff, int store_u, int red_slot)
{
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double r_diff = 0.0, r_norm = 0.0, r_ux = 0.0, r_rho = 0.0;
    if (c < n)
    {
        const int l = cell_level[c] - 1;
        const LevelView &L = A.lv[l];
        const int s = cell_site[c];
        const int x = s % L.pitch, y = s / L.pitch;
        float df[9];
        bool special;
        SpecialRec rec;
        // after a coarse step every interface buffer holds its interpolated values
        if (A.parity[l] == 0) load_cell<0>(L, C, x, y, A.direct[l], 1, df, special, rec);
        else load_cell<1>(L, C, x, y, A.direct[l], 1, df, special, rec);
        float drho, rho, ux, uy;
        macro(df, C.rho0, L.fshift, 0.0f, drho, rho, ux, uy);
        if (diff | store_u)
        {
            const float un = sqrtf(ux * ux + uy * uy);
            if (diff)
            {
                r_diff = (double)fabsf(un - L.unorm[s]);
                r_norm = (double)un;
            }
            if (store_u) L.unorm[s] = un;
        }
        // FP64 outputs from the FP32 deviations
        double ddr = 0, jx = 0, jy = 0;
        for (int q = 0; q < 9; q++)
        {
            ddr += (double)df[q];
            jx += (double)d2q9::cx(q) * (double)df[q];
            jy += (double)d2q9::cy(q) * (double)df[q];
        }
        double r = (double)C.rho0 + ddr;
        double vx = (jx + (double)L.fshift) / r, vy = jy / r;
        if (C.adsorption)
        {
            // the reference reports the density and velocity computed at the
            // start of the last step (include/mantiisApp.hpp:248-265)
            r = (double)C.rho0 + (double)L.snap[s];
            vx = (double)L.snap[L.plane + s];
            vy = (double)L.snap[2 * L.plane + s];
        }
        if (rho_out) rho_out[c] = r;
        if (ux_out) ux_out[c] = vx;
        if (uy_out) uy_out[c] = vy;
        if (f_out)
            for (int q = 0; q < 9; q++) f_out[c * 9 + q] = d2q9::w(q) * (double)C.rho0 + (double)df[q];
        // interface buffer cells cover pixels of finer cells: left out of the
        // pixel-area sums (also those that step like plain cells)
        if (!cell_buffer[c])
        {
            const double area = (double)(1 << (2 * l));
            r_ux = vx * area;
            r_rho = r * area;
        }
    }
    if (red_slot >= 0)
    {
        block_add2(r_diff, r_norm, C.red + red_slot);
        block_add2(r_ux, r_rho, C.red + red_slot + 2);
    }
}

// Writes populations df of cell (x, y) into the slots its next step reads at
// parity P: its own slots (even) or the neighbours' opposite slots (odd).
// These slots belong to the cell (AA ownership), so nothing else touches them
// before that step.
__device__ __forceinline__ void store_for_load(const LevelView &L, int x, int y, const float df[9], int parity)
{
    if (parity == 0)
    {
        const int64_t s = site_of(L, x, y);
#pragma unroll
        for (int q = 0; q < 9; q++) L.f[q * L.plane + s] = df[q];
    }
    else
    {
#pragma unroll
        for (int q = 0; q < 9; q++)
        {
            const int xs = wrapx(x - d2q9::cx(q), L.W), ys = wrapx(y - d2q9::cy(q), L.H);
            L.f[d2q9::opp(q) * L.plane + site_of(L, xs, ys)] = df[q];
        }
    }
}

// The interface rows are handled by groups of 4 adjacent lanes (lane & 3 = k):
// each lane loads one child (coarse rows) or one or two spline nodes (fine
// rows), and the group exchanges the loaded populations with shuffles, so the
// loads of a row are in flight together and each is made once.  Sums run in
// the same order as one lane summing alone.

// populations of an interface source cell: its interpolation buffer, or the
// cell's own slots after streaming and its rules
// (`plain`: the row has no special source, which holds for all but a few rows;
// its cells' rates need not be looked up before their populations)
template <int P>
__device__ __forceinline__ void load_source(const LevelView &L, const Common &C, int site, int buf, bool plain, float z[9])
{
    if (buf >= 0)
    {
#pragma unroll
        for (int q = 0; q < 9; q++) z[q] = C.ibuf[(size_t)q * C.n_buf + buf];
    }
    else if (plain)
    {
        const int x = site % L.pitch, y = site / L.pitch;
        load_raw_ro<P, false>(L, x, y, z, x > 0 && x + 1 < L.W && y > 0 && y + 1 < L.H);
    }
    else
    {
        bool special;
        SpecialRec rec;
        load_cell<P>(L, C, site % L.pitch, site / L.pitch, 0, 0, z, special, rec);
    }
}

// Coarse buffer cells <- rescaled mean of their 4 children
// (include/coreLB.hpp:1104-1135): f_c = f_eq,c + 2 tau_c / mean(tau_f) (mean(f_f) - f_eq,c).
// Lane k of the group loads child k; lane 0 writes the result.
template <int PF>
__device__ __forceinline__ void coarse_row(const LevelView &Lf, const LevelView &Lc, const Common &C,
                                           const CoarseRowDev &row, int k, bool valid, int pc)
{
    const int lane = threadIdx.x & 31, base = lane & ~3;
    const bool has = valid && row.child[k] >= 0;
    float df[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (has) load_source<PF>(Lf, C, row.child[k], row.child_buf[k], !row.special, df);
    float mean[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
    {
        const bool present = __shfl_sync(0xffffffffu, has ? 1 : 0, base + kk) != 0;
#pragma unroll
        for (int q = 0; q < 9; q++)
        {
            const float v = __shfl_sync(0xffffffffu, df[q], base + kk);
            if (present) mean[q] += v;
        }
    }
    if (!valid || k != 0) return;
    const float drho = Lc.snap[row.site], ux = Lc.snap[Lc.plane + row.site], uy = Lc.snap[2 * Lc.plane + row.site];
    float feq[9];
    equilibrium(drho, C.rho0 + drho, ux, uy, feq);
    float v[9];
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        v[q] = feq[q] + row.ratio * (mean[q] * row.inv_nchild - feq[q]);
        C.ibuf[(size_t)q * C.n_buf + row.buf] = v[q];
    }
    if (row.plain_target) store_for_load(Lc, row.site % Lc.pitch, row.site / Lc.pitch, v, pc);
}

// Fine buffer cells <- bicubic spline of the parent neighbourhood
// (include/coreLB.hpp:1137-1230); the spline is linear in the node values, so
// each child holds 6 precomputed weights.  f = f_eq + tau_f / (2 tau_c) (f_spline - f_eq).
// Lane c of the group loads nodes c and c + 4 (c < 2) and computes child c.
template <int PC>
__device__ __forceinline__ void fine_child(const LevelView &Lf, const LevelView &Lc, const Common &C,
                                           const FineRowDev &row, int c, bool valid, int pf)
{
    const int lane = threadIdx.x & 31, base = lane & ~3;
    float za[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, zb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (valid)
    {
        load_source<PC>(Lc, C, row.node_site[c], row.node_buf[c], !row.special, za);
        if (c < 2) load_source<PC>(Lc, C, row.node_site[c + 4], row.node_buf[c + 4], !row.special, zb);
    }
    float acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 6; k++)
    {
        const float w = valid ? row.weight[c][k] : 0.0f;
#pragma unroll
        for (int q = 0; q < 9; q++)
        {
            const float z = __shfl_sync(0xffffffffu, k < 4 ? za[q] : zb[q], base + (k & 3));
            acc[q] += w * z;
        }
    }
    if (!valid) return;
    const int s = row.child_site[c];
    const float drho = Lf.snap[s], ux = Lf.snap[Lf.plane + s], uy = Lf.snap[2 * Lf.plane + s];
    float feq[9];
    equilibrium(drho, C.rho0 + drho, ux, uy, feq);
    const float rat = row.ratio[c];
    const int cb = row.child_buf[c];
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        acc[q] = feq[q] + rat * (acc[q] - feq[q]);
        C.ibuf[(size_t)q * C.n_buf + cb] = acc[q];
    }
    if ((row.plain_mask >> c) & 1) store_for_load(Lf, s % Lf.pitch, s / Lf.pitch, acc, pf);
}


// One level pair of one image in the interface exchange: the two levels'
// states (at their parities after the coarse step) and the pair's rows.
struct PairDesc
{
    LevelView Lf, Lc;
    Common C;
    const CoarseRowDev *coarse;
    const FineRowDev *fine;
    int pf, pc;  // parity of the next step of the fine / coarse level
    int kind;    // rows of this entry: 0 coarse, 1 fine
    int nrows;
};

constexpr int kMaxWaveDescs = 16;

struct WaveLaunch
{
    int ndesc;
    int start[kMaxWaveDescs + 1];
    PairDesc d[kMaxWaveDescs];
};

// Interface exchange wave: coarse rows of some pairs and fine rows of others
// (independent within a wave), 32 rows per block, 4 lanes per row.
__global__ void __launch_bounds__(128) k_wave(const __grid_constant__ WaveLaunch W)
{
    const int j = owner(W.start, W.ndesc, (int)blockIdx.x);
    const PairDesc &d = W.d[j];
    const int u = ((int)blockIdx.x - W.start[j]) * 128 + (int)threadIdx.x;
    const int r = u >> 2, k = u & 3;
    // lanes past the last row stay for the group shuffles
    const bool valid = r < d.nrows;
    const int rr = valid ? r : 0;
    if (d.kind == 0)
    {
        const CoarseRowDev &row = d.coarse[rr];
        if (d.pf) coarse_row<1>(d.Lf, d.Lc, d.C, row, k, valid, d.pc);
        else coarse_row<0>(d.Lf, d.Lc, d.C, row, k, valid, d.pc);
    }
    else
    {
        const FineRowDev &row = d.fine[rr];
        if (d.pc) fine_child<1>(d.Lf, d.Lc, d.C, row, k, valid, d.pf);
        else fine_child<0>(d.Lf, d.Lc, d.C, row, k, valid, d.pf);
    }
}

// ---- persistent step: one launch runs whole coarse steps of a group of
// images.  The work is a list of units (one block of 256 threads each) in claim
// order: 8 x tiles_per_warp tiles of 8x4 plain and light cells, 256 special
// records with walls, or 64 interface rows.  Units are grouped in segments,
// and the segments of one image form stages: the phases of its coarse step,
// then its interface waves.  A stage starts only when the image's previous
// stage is complete (the level substeps and the exchange that the phase engine
// orders by stream order), which a block learns from that stage's completion
// counter.  Blocks claim units with one atomic counter; every segment waits
// only on units earlier in claim order, so the unit with the lowest unfinished
// index can always run and the launch never deadlocks, whatever its grid size.
// Stages of different images interleave in the claim order, so while one image
// waits on its last units another image's work fills the GPU.
struct PersistSeg
{
    int kind;        // 0 plain8 tiles, 1 special records, 2 coarse rows, 3 fine rows
    int desc;        // StepDesc (kinds 0, 1) or PairDesc (2, 3) index
    int unit0;       // first unit of the segment in claim order
    int nunits;
    int wait_ctr;    // counter that must reach wait_target first (-1: none)
    unsigned wait_target;
    int done_ctr;    // counter each finished unit increments
    int pad;
};

constexpr int kPersistThreads = 256;
constexpr int kPersistRecords = kPersistThreads; // special records per unit
constexpr int kPersistRows = kPersistThreads / 4; // interface rows per unit (4 lanes each)
constexpr unsigned kErrDepTimeout = 2u;
// polls of a stage counter before a block gives up (an L2 round trip and a
// 64 ns sleep each: about a second); a normal wait takes microseconds
constexpr uint32_t kDepPolls = 1u << 22;

struct PersistLaunch
{
    const PersistSeg *segs;
    const StepDesc *sd;
    const PairDesc *pd;
    unsigned int *sync;   // [0] claim counter, [1 + c] stage counter c; zero at launch
    unsigned int *err;    // device error word
    int nseg, total_units;
    int tiles_per_warp;   // 8x4 tiles each warp of a plain-cell unit steps
};

__device__ __forceinline__ bool wait_counter(const unsigned int *c, unsigned int target)
{
    for (uint32_t i = 0; i < kDepPolls; i++)
    {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
        if (v >= target) return true;
        __nanosleep(64);
    }
    return false;
}

// Stage-counter update with release semantics: after the block barrier, every
// thread's stores of the unit are ordered before it (cumulativity).
__device__ __forceinline__ void add_release(unsigned int *c, unsigned int v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(c), "r"(v) : "memory");
}

// The descriptor of a segment, staged in shared memory once per segment (the
// array is read-only during the launch, so it takes the read-only path).
template <typename T> __device__ __forceinline__ void stage_desc(T *dst, const T *src)
{
    static_assert(sizeof(T) % 4 == 0, "descriptor size");
    const uint32_t *s = reinterpret_cast<const uint32_t *>(src);
    uint32_t *d = reinterpret_cast<uint32_t *>(dst);
    for (int i = (int)threadIdx.x; i < (int)(sizeof(T) / 4); i += (int)blockDim.x) d[i] = __ldg(&s[i]);
}

// MINB: blocks per SM the register budget is sized for (more blocks, fewer
// registers: the special-record and interface paths then spill a little; 5
// blocks of 48 registers measured best).
template <int MINB>
__global__ void __launch_bounds__(kPersistThreads, MINB) k_step_persistent(const __grid_constant__ PersistLaunch P)
{
    __shared__ union
    {
        StepDesc sd;
        PairDesc pd;
    } s_desc;
    __shared__ int s_unit, s_seg, s_next;
    int seg_cache = 0;        // thread 0: segment of the last claim (claims only grow)
    int ok_ctr = -1;          // thread 0: a counter already seen complete by this block
    unsigned ok_target = 0u;
    int staged = -1;          // segment whose descriptor is in shared memory
    if (threadIdx.x == 0) s_next = (int)atomicAdd(P.sync, 1u);
    for (;;)
    {
        if (threadIdx.x == 0)
        {
            const int u = s_next;
            int seg = -1;
            if (u < P.total_units)
            {
                while (seg_cache + 1 < P.nseg && __ldg(&P.segs[seg_cache + 1].unit0) <= u) seg_cache++;
                seg = seg_cache;
                const int wc = __ldg(&P.segs[seg].wait_ctr);
                const unsigned wt = __ldg(&P.segs[seg].wait_target);
                if (wc >= 0 && !(wc == ok_ctr && wt <= ok_target))
                {
                    if (wait_counter(P.sync + 1 + wc, wt))
                    {
                        ok_ctr = wc;
                        ok_target = wt;
                    }
                    else
                    {
                        // an earlier unit never finished: stop (its waiters stop too)
                        atomicOr(P.err, kErrDepTimeout);
                        seg = -1;
                    }
                }
                // the next claim is in flight while this unit runs
                if (seg >= 0) s_next = (int)atomicAdd(P.sync, 1u);
            }
            s_unit = u;
            s_seg = seg;
        }
        __syncthreads();
        const int u = s_unit, seg = s_seg;
        if (seg < 0) break;
        const int kind = __ldg(&P.segs[seg].kind), desc = __ldg(&P.segs[seg].desc);
        const int k = u - __ldg(&P.segs[seg].unit0);
        if (seg != staged)
        {
            if (kind < 2) stage_desc(&s_desc.sd, &P.sd[desc]);
            else stage_desc(&s_desc.pd, &P.pd[desc]);
            staged = seg;
            __syncthreads();
        }
        double r_diff = 0.0, r_norm = 0.0;
        if (kind == 0)
        {
            const StepDesc &d = s_desc.sd;
            const int t0 = (k * 8 + (int)(threadIdx.x >> 5)) * P.tiles_per_warp;
#pragma unroll 1
            for (int j = 0; j < P.tiles_per_warp; j++)
            {
                const int t = t0 + j;
                if (t < d.L.ntiles8)
                {
                    if (d.o.parity) plain_tile8<1, false>(d.L, d.C, d.o, t, 0, 0, r_diff, r_norm);
                    else plain_tile8<0, false>(d.L, d.C, d.o, t, 0, 0, r_diff, r_norm);
                }
            }
        }
        else if (kind == 1)
        {
            const StepDesc &d = s_desc.sd;
            const int i = k * kPersistRecords + (int)threadIdx.x;
            if (i < d.spec_count)
            {
                if (d.o.parity) special_cell<1>(d.L, d.C, d.o, d.spec_begin + i, 0, 0, r_diff, r_norm);
                else special_cell<0>(d.L, d.C, d.o, d.spec_begin + i, 0, 0, r_diff, r_norm);
            }
        }
        else
        {
            // 4 lanes per row, as k_wave
            const PairDesc &d = s_desc.pd;
            const int v = k * kPersistThreads + (int)threadIdx.x;
            const int r = v >> 2, c = v & 3;
            const bool valid = r < d.nrows;
            const int rr = valid ? r : 0;
            if (kind == 2)
            {
                const CoarseRowDev &row = d.coarse[rr];
                if (d.pf) coarse_row<1>(d.Lf, d.Lc, d.C, row, c, valid, d.pc);
                else coarse_row<0>(d.Lf, d.Lc, d.C, row, c, valid, d.pc);
            }
            else
            {
                const FineRowDev &row = d.fine[rr];
                if (d.pc) fine_child<1>(d.Lf, d.Lc, d.C, row, c, valid, d.pf);
                else fine_child<0>(d.Lf, d.Lc, d.C, row, c, valid, d.pf);
            }
        }
        // the unit's stores, then its count (release): a waiter's acquire load
        // of the counter then sees them
        __syncthreads();
        if (threadIdx.x == 0) add_release(P.sync + 1 + __ldg(&P.segs[seg].done_ctr), 1u);
    }
}

// ---- the adsorption step as one cooperative launch over many steps.  Each
// step is the two passes of k_ads_psi / k_ads_psi_special and k_ads_step /
// k_ads_step_special, each closed by a grid barrier; the per-cell arithmetic is
// the same code, so the states are bit-identical to the launch-per-pass engine.
//
// What bounds a step at these sizes (156 k cells: 1 k per SM) is latency: two
// grid barriers, a round trip to L2 for the populations and one for the
// neighbours' pseudopotentials, then the instructions of pass 2 (about 700 per
// warp of cells).  So one block per SM (fewest arrivals at a barrier) owns the
// same cells in every step, an equal share of the plain cells and of the special
// records, a warp at a time; it keeps what only it reads in shared memory:
// the populations between the two passes, the relaxation rates, the density of
// the previous step.  Populations are then read once a step, the density and
// the outputs leave for memory in the last step of the launch only.  Measured on
// a GB300, us per step: 512^2 image (156 k cells) 9.2, 190^2 6.9, 64^2 5.8 (a
// barrier alone is 1.3); with tiles dealt to 456 blocks that read the populations
// in both passes 24.4, 13.9 and 11.1.
struct AdsPersist
{
    LevelView L;
    Common C;
    const int32_t *plain_xy; // plain cells: x | y << 16
    int64_t spec_begin;
    int nplain, spec_count;
    int slots;              // cells' warps whose data fits a block's shared memory
    int rec_slots;          // of these, warps of special cells (their records come first)
    int nsteps, parity0, direct0;
    int slot0, ring;        // residual of step k in slot (slot0 + k) mod ring
    int psi_diff;           // accumulate the residual of pass 1 (density change)
    unsigned int *bar;      // arrivals at the grid barriers; zero at launch
    uint32_t polls;         // of a barrier's wait before the block gives up
};

// shared memory of one warp of cells: this many floats per lane
constexpr int kAdsFields = 15;
enum AdsField
{
    AF_F = 0,    // 9 populations, as the cell collides
    AF_RATE = 9, // relaxation rates 1/tau_d, 1/tau_q, 1/tau_s
    AF_PSI = 12, // the cell's pseudopotential
    AF_RHO = 13, // its density in the previous step
    AF_XY = 14,  // x | y << 16 of a plain cell, negative past the end
};
constexpr size_t kAdsSlotBytes = (size_t)kAdsFields * 32 * 4;
constexpr size_t kAdsRecBytes = (size_t)32 * sizeof(SpecialRec); // records of one warp of special cells
// Most threads of a block: blocks of one round of warps take the kernel of up to
// 512 threads (128 registers, nothing spilled), the others that of up to 640 (96)
constexpr int kAdsSmall = 512, kAdsLarge = 640;

// Sums of a and b over each warp, to sums[warp]; after a block barrier one warp
// adds the warps' sums to dst[0] and dst[1].
__device__ __forceinline__ void block_sums(double a, double b, double2 *sums)
{
    for (int o = 16; o > 0; o >>= 1)
    {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = make_double2(a, b);
}
__device__ __forceinline__ void add_block_sums(const double2 *sums, double *dst)
{
    const int lane = threadIdx.x & 31;
    double2 v = lane < (int)(blockDim.x >> 5) ? sums[lane] : make_double2(0.0, 0.0);
    for (int o = 16; o > 0; o >>= 1)
    {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0)
    {
        if (v.x != 0.0) atomicAdd(dst, v.x);
        if (v.y != 0.0) atomicAdd(dst + 1, v.y);
    }
}

// Grid barrier `target` = (barriers passed) x gridDim.x: every block adds one
// arrival with release semantics after its block barrier, then waits (bounded)
// for all of them, at most `polls` polls; where they run out (false) the caller
// notes it in the error word and the block stops.
// rmax: if not null, the block's maximum of the residual terms (non-negative
// floats by their bit patterns), which goes to dst and is cleared; clear: a
// counter in shared memory set to zero on the way; sums: if not null, the warps'
// pairs of sums in shared memory (block_sums), which warp 1 adds to sums_to while
// the block waits.
__device__ __forceinline__ bool grid_barrier(unsigned int *bar, unsigned int target, uint32_t polls,
                                             unsigned int *rmax, double *dst, unsigned int *clear = nullptr,
                                             const double2 *sums = nullptr, double *sums_to = nullptr)
{
    __shared__ int s_ok;
    __syncthreads();
    if (sums && threadIdx.x >= 32 && threadIdx.x < 64) add_block_sums(sums, sums_to);
    if (threadIdx.x == 0)
    {
        if (rmax && *rmax)
        {
            atomicMax(reinterpret_cast<unsigned long long *>(dst),
                      (unsigned long long)__double_as_longlong((double)__uint_as_float(*rmax)));
            *rmax = 0u;
        }
        if (clear) *clear = 0u;
        add_release(bar, 1u);
        bool ok = false;
        for (uint32_t i = polls; i != 0 && !ok; i--)
        {
            unsigned int v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            ok = v >= target;
        }
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// the neighbours' pseudopotentials around (x, y); the centre is the caller's
__device__ __forceinline__ void load_psi(const LevelView &L, int x, int y, bool interior, float psi[3][3])
{
    if (interior)
    {
        const float *p = L.psi + site_of(L, x, y);
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (r != 1 || c != 1) psi[r][c] = p[(r - 1) * (int64_t)L.pitch + c - 1];
    }
    else
    {
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                if (r != 1 || c != 1) psi[r][c] = L.psi[site_of(L, wrapx(x + c - 1, L.W), wrapx(y + r - 1, L.H))];
    }
}

// The block's cells: special records [s0, s1) in ws warps, plain cells [p0, p1)
// in wp warps.  Slot k of the shared memory belongs to warp-of-cells k.  The
// special ones go to the block's warps from the first on; a special cell takes
// about as long as two plain ones, so plain ones go to the warps after those
// where there are enough (first plain warp of this warp: pj0, then every pstep).
struct AdsShare
{
    int s0, s1, p0, p1, ws, wp, pj0, pstep;
    uint4 *recs; // special records of the first rec_slots warps, as [warp][half][lane]
};

// One warp of cells of the block as a lane sees it: the cell, and its data in
// shared memory (m; null where FITS is false and the slots ran out).
template <bool FITS> struct AdsCell
{
    const LevelView &L;
    float *m;
    int x, y;
    int64_t s;
    __device__ __forceinline__ AdsCell(const AdsPersist &A, float *sm, int u, int xy)
        : L(A.L), m(FITS || u < A.slots ? sm + (size_t)u * kAdsFields * 32 + (threadIdx.x & 31) : nullptr),
          x(xy & 0xFFFF), y(xy >> 16), s(site_of(A.L, x, y))
    {
    }
    __device__ __forceinline__ bool held() const { return FITS || m != nullptr; }
    __device__ __forceinline__ bool interior() const { return x > 0 && x + 1 < L.W && y > 0 && y + 1 < L.H; }
    __device__ __forceinline__ float old_density() const { return held() ? m[AF_RHO * 32] : L.rho_prev[s]; }
    __device__ __forceinline__ MrtRates rates(float omega) const
    {
        if (held()) return MrtRates{m[AF_RATE * 32], m[(AF_RATE + 1) * 32], m[(AF_RATE + 2) * 32]};
        return mrt_rates(1.0f / omega, L.tau2[s]);
    }
    // pass 1 with the populations df: pseudopotential, density change returned
    __device__ __forceinline__ float density(const Common &C, const float df[9], float old, bool last)
    {
        float drho = 0.0f;
#pragma unroll
        for (int q = 0; q < 9; q++) drho += df[q];
        const float rho = C.rho0 + drho;
        const float psi = pseudo_potential((float)C.psi_form, C.psi_rho0, C.eos_a, C.eos_b, C.eos_T, C.g_ff, rho);
        L.psi[s] = psi;
        if (!held() || last) L.rho_prev[s] = rho;
        if (held())
        {
#pragma unroll
            for (int q = 0; q < 9; q++) m[(AF_F + q) * 32] = df[q];
            m[AF_PSI * 32] = psi;
            m[AF_RHO * 32] = rho;
        }
        return fabsf(rho - old) / old;
    }
    __device__ __forceinline__ void populations(float df[9]) const
    {
#pragma unroll
        for (int q = 0; q < 9; q++) df[q] = m[(AF_F + q) * 32];
    }
};

// record of lane `lane` of special warp u (record i of the level)
__device__ __forceinline__ SpecialRec ads_record(const AdsPersist &A, const AdsShare &B, int u, int i, int lane)
{
    if (u >= A.rec_slots) return A.C.specials[A.spec_begin + i];
    union
    {
        SpecialRec rec;
        uint4 v[2];
    } t;
    static_assert(sizeof(SpecialRec) == 2 * sizeof(uint4), "record size");
    t.v[0] = B.recs[(u * 2) * 32 + lane];
    t.v[1] = B.recs[(u * 2 + 1) * 32 + lane];
    return t.rec;
}

// x | y << 16 of this lane's cell in plain warp j, negative past the share
template <bool FITS> __device__ __forceinline__ int ads_plain_xy(const AdsPersist &A, const AdsShare &B, const float *sm, int j)
{
    const int u = B.ws + j, lane = threadIdx.x & 31;
    if (FITS || u < A.slots) return __float_as_int(sm[((size_t)u * kAdsFields + AF_XY) * 32 + lane]);
    const int i = B.p0 + j * 32 + lane;
    return i < B.p1 ? __ldg(&A.plain_xy[i]) : -1;
}

// fills the block's shared memory: records, cells, relaxation rates and
// previous densities
__device__ __forceinline__ void ads_fill(const AdsPersist &A, const AdsShare &B, float *sm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int u = warp; u < B.ws + B.wp && u < A.slots; u += nw)
    {
        float *m = sm + (size_t)u * kAdsFields * 32 + lane;
        int xy = -1;
        float omega = 0.0f;
        if (u < B.ws)
        {
            const int i = B.s0 + u * 32 + lane;
            if (i < B.s1)
            {
                const uint4 *r = reinterpret_cast<const uint4 *>(A.C.specials + A.spec_begin + i);
                const uint4 r0 = r[0], r1 = r[1];
                if (u < A.rec_slots)
                {
                    B.recs[(u * 2) * 32 + lane] = r0;
                    B.recs[(u * 2 + 1) * 32 + lane] = r1;
                }
                xy = (int)r1.z;
                omega = __uint_as_float(r1.w);
            }
        }
        else
        {
            const int i = B.p0 + (u - B.ws) * 32 + lane;
            if (i < B.p1) xy = __ldg(&A.plain_xy[i]);
            if (xy >= 0) omega = A.L.omega[site_of(A.L, xy & 0xFFFF, xy >> 16)];
        }
        m[AF_XY * 32] = __int_as_float(xy);
        if (xy < 0) continue;
        const int64_t s = site_of(A.L, xy & 0xFFFF, xy >> 16);
        const MrtRates r = mrt_rates(1.0f / omega, A.L.tau2[s]);
        m[AF_RATE * 32] = r.d;
        m[(AF_RATE + 1) * 32] = r.q;
        m[(AF_RATE + 2) * 32] = r.s;
        m[AF_RHO * 32] = A.L.rho_prev[s];
    }
}

template <int P, bool FITS>
__device__ __forceinline__ float ads_pass1(const AdsPersist &A, const AdsShare &B, float *sm, bool direct, bool last)
{
    const LevelView &L = A.L;
    const Common &C = A.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float rmax = 0.0f;
#pragma unroll 1
    for (int u = warp; u < B.ws; u += nw)
    {
        const int i = B.s0 + u * 32 + lane;
        if (i >= B.s1) continue;
        const SpecialRec rec = ads_record(A, B, u, i, lane);
        AdsCell<FITS> c(A, sm, u, rec.xy);
        float df[9];
        const float old = c.old_density();
        if (direct) load_raw<0>(L, c.x, c.y, df);
        else load_special<P>(L, C, rec, c.x, c.y, df);
        rmax = fmaxf(rmax, c.density(C, df, old, last));
    }
    // plain cells, two warps of cells at a time: both populations in flight (a
    // direct state has parity 0: own slots)
#pragma unroll 1
    for (int j0 = B.pj0; j0 < B.wp; j0 += 2 * B.pstep)
    {
        float df[2][9];
        int xy[2];
#pragma unroll
        for (int k = 0; k < 2; k++)
        {
            xy[k] = j0 + k * B.pstep < B.wp ? ads_plain_xy<FITS>(A, B, sm, j0 + k * B.pstep) : -1;
            if (xy[k] < 0) continue;
            const AdsCell<FITS> c(A, sm, B.ws + j0 + k * B.pstep, xy[k]);
            load_raw_ro<P, false>(L, c.x, c.y, df[k], c.interior());
        }
#pragma unroll
        for (int k = 0; k < 2; k++)
        {
            if (xy[k] < 0) continue;
            AdsCell<FITS> c(A, sm, B.ws + j0 + k * B.pstep, xy[k]);
            rmax = fmaxf(rmax, c.density(C, df[k], c.old_density(), last));
        }
    }
    return rmax;
}

template <int P, bool FITS>
__device__ __forceinline__ void ads_pass2(const AdsPersist &A, const AdsShare &B, float *sm, const StepOpt &o, bool direct)
{
    const LevelView &L = A.L;
    const Common &C = A.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double none0 = 0.0, none1 = 0.0;
#pragma unroll 1
    for (int u = warp; u < B.ws; u += nw)
    {
        const int i = B.s0 + u * 32 + lane;
        if (i >= B.s1) continue;
        const SpecialRec rec = ads_record(A, B, u, i, lane);
        const AdsCell<FITS> c(A, sm, u, rec.xy);
        float psi[3][3], df[9];
        load_psi(L, c.x, c.y, c.interior(), psi);
        psi[1][1] = c.held() ? c.m[AF_PSI * 32] : L.psi[c.s];
        if (c.held()) c.populations(df);
        else if (direct) load_raw<0>(L, c.x, c.y, df);
        else load_special<P>(L, C, rec, c.x, c.y, df);
        ads_update<P>(L, C, o, c.x, c.y, df, rec.omega, c.rates(rec.omega), true, rec, psi, none0, none1);
    }
#pragma unroll 1
    for (int j = B.pj0; j < B.wp; j += B.pstep)
    {
        const int xy = ads_plain_xy<FITS>(A, B, sm, j);
        if (xy < 0) continue;
        const AdsCell<FITS> c(A, sm, B.ws + j, xy);
        float psi[3][3], df[9], omega = 0.0f;
        load_psi(L, c.x, c.y, c.interior(), psi);
        psi[1][1] = c.held() ? c.m[AF_PSI * 32] : L.psi[c.s];
        if (c.held()) c.populations(df);
        else
        {
            load_raw_ro<P, false>(L, c.x, c.y, df, c.interior());
            omega = L.omega[c.s];
        }
        const SpecialRec none{};
        ads_update<P>(L, C, o, c.x, c.y, df, omega, c.rates(omega), false, none, psi, none0, none1, c.interior());
    }
}

template <int THREADS, bool FITS>
__global__ void __launch_bounds__(THREADS, 1) k_ads_persistent(const __grid_constant__ AdsPersist A)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ unsigned int s_rmax;
    float *sm = reinterpret_cast<float *>(sm_raw + A.rec_slots * kAdsRecBytes);
    AdsShare B;
    const int64_t b = blockIdx.x, g = gridDim.x;
    B.s0 = (int)(b * A.spec_count / g);
    B.s1 = (int)((b + 1) * A.spec_count / g);
    B.p0 = (int)(b * A.nplain / g);
    B.p1 = (int)((b + 1) * A.nplain / g);
    B.ws = (B.s1 - B.s0 + 31) / 32;
    B.wp = (B.p1 - B.p0 + 31) / 32;
    const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (2 * B.ws <= nw)
    {
        B.pstep = nw - B.ws;
        B.pj0 = warp < B.ws ? B.wp : warp - B.ws;
    }
    else
    {
        B.pstep = nw;
        B.pj0 = (warp + nw - B.ws % nw) % nw;
    }
    B.recs = reinterpret_cast<uint4 *>(sm_raw);
    if (threadIdx.x == 0) s_rmax = 0u;
    ads_fill(A, B, sm);
    __syncthreads();
    unsigned int target = 0;
#pragma unroll 1
    for (int k = 0; k < A.nsteps; k++)
    {
        const int parity = (A.parity0 + k) & 1;
        const bool last = k + 1 == A.nsteps, direct = k == 0 && A.direct0;
        StepOpt o{};
        o.parity = parity;
        o.snap_store = last ? 1 : 0; // the outputs show the last step's
        const float rmax = parity ? ads_pass1<1, FITS>(A, B, sm, direct, last) : ads_pass1<0, FITS>(A, B, sm, direct, last);
        if (A.psi_diff)
        {
            // non-negative floats order like their bits; a NaN counts as no change
            const unsigned int v = __reduce_max_sync(0xffffffffu, rmax > 0.0f ? __float_as_uint(rmax) : 0u);
            if ((threadIdx.x & 31) == 0 && v) atomicMax(&s_rmax, v);
        }
        target += gridDim.x;
        if (!grid_barrier(A.bar, target, A.polls, A.psi_diff ? &s_rmax : nullptr,
                          A.C.red + (size_t)((A.slot0 + k) % A.ring) * 4))
        {
            if (threadIdx.x == 0) atomicOr(A.C.err, kErrDepTimeout);
            return;
        }
        if (parity) ads_pass2<1, FITS>(A, B, sm, o, direct);
        else ads_pass2<0, FITS>(A, B, sm, o, direct);
        target += gridDim.x;
        if (!last && !grid_barrier(A.bar, target, A.polls, nullptr, nullptr))
        {
            if (threadIdx.x == 0) atomicOr(A.C.err, kErrDepTimeout);
            return;
        }
    }
}

// ---- transport steps of a group of images as one cooperative launch over many
// coarse steps.  The stages of a coarse step are those of the phase engine (a
// phase steps every level whose next substep falls on it; the interface waves
// follow), each closed by a grid barrier, over all images of the group; the
// per-cell arithmetic is the same code, so the states are bit-identical.
//
// A stage of the phase engine costs a launch (2 us and more with its fork to the
// special cells' stream), blocks that fetch a descriptor, a tile and its masks
// before their first population, and 23 % idle lanes.  Here one block per SM
// owns the same warps of cells in every step (compacted lists of the cells of
// each kind and level, an equal share of each): what identifies a cell (position
// and relaxation rate, or its record), the |u| of the residual and the
// coarse-step-start moments that only the cell itself reads wait in shared
// memory.  A cell's populations are then the only round trip to memory.
//
// Measured on a GB300, us per coarse step without / with residuals: single block
// 64^2 3.6 / 4.4, 128^2 3.7 / 4.5, 512^2 5.3 / 7.1, 1024^2 11.7 / 15.7, two levels
// 256^2 16.1 / 17.6, 1024^2 34 / 37; the launches per phase 6.1 / 10.7, 6.2 / 10.4,
// 9.3 / 17.4, 16.4 / 34.7, 22.9 / 27.5, 42.8 / 55.9.  A grid barrier takes 0.85 us,
// a warp of special cells about 2.5: what small images wait for.  At 1024^2 the
// stages move 1.7 (single block) to 4 times (two levels: thin bands of fine cells)
// the cells' bytes, whole sectors, between L2 and the SMs.
constexpr int kMaxCoopDescs = 40, kMaxCoopPairs = 30;

enum CoopKind
{
    CK_HEAVY = 0, // special records with walls, periodic overrides, ...
    CK_LIGHT = 1, // special records with missing arrivals or buffer status only
    CK_EDGE = 2,  // plain buffer cells: the interface waves read their coarse-step-start moments
    CK_PLAIN = 3, // other plain cells
    CK_KINDS = 4,
};

struct CoopDesc // one level of one image
{
    LevelView L;
    Common C;
    const int32_t *xy[CK_KINDS]; // plain cells of the two kinds: x | y << 16
    int64_t spec_begin;      // the level's records: the heavy ones, then the light ones
    const int32_t *cut[CK_KINDS]; // block b steps cells [cut[b], cut[b + 1]) of each kind
    int nheavy;              // records before the light ones
    int lines[CK_KINDS];     // shared-memory lines per warp of cells
    int shift;               // steps in the phases that are multiples of 1 << shift
    int substeps, parity0, direct0, mb;
};

struct CoopPair // one level pair of one image
{
    const CoarseRowDev *coarse;
    const FineRowDev *fine;
    int ncoarse, nfine;
    int df, dc; // descriptors of its fine / coarse level
    int l1;     // 1 for levels (1, 2), ...
    int rot;
};

struct CoopLaunch
{
    int nd, np, nphase, nwave;
    int nsteps;
    // residual (one image): |u| stored by steps whose number is a multiple of
    // `every`, compared by the step after, into slot (number of the storing step) mod
    // ring; skip_first: not by the launch's first step, whose number mod `every` is
    // since0 and whose predecessor's slot is slot0
    int every, skip_first, ring, since0, slot0;
    unsigned int *bar; // grid-barrier arrivals, blocks that have left; both zero at launch and after it
    uint32_t polls;    // of a barrier's wait before the block gives up
    CoopDesc d[kMaxCoopDescs];
    CoopPair p[kMaxCoopPairs];
};

// W warps of interface rows dealt to G blocks: block b takes [cut(b), cut(b + 1));
// the rotation spreads the lists' remainders over the blocks.
__host__ __device__ inline int coop_cut(int W, int rot, int b, int G) { return (int)(((int64_t)W * b + rot) / G); }

// Shared memory in lines of 32 words (one per lane).  A plain warp of cells: the
// site (coop_site), 1/tau_s, |u|, and for CK_PLAIN on levels of several substeps
// the coarse-step-start moments; a special one: its records (two 16-byte halves),
// |u|.
constexpr int kCoopPlainLines = 3, kCoopSnapLines = 3, kCoopRecLines = 9;
constexpr uint32_t kCoopNone = 0xFFFFFFFFu; // a lane past the list

// site of cell (x, y) in the lower 28 bits, above it which of the level's borders
// the cell lies on: its neighbours there wrap around the torus
constexpr uint32_t kCoopSite = (1u << 28) - 1u, kCoopLeft = 1u << 28, kCoopRight = 1u << 29, kCoopLow = 1u << 30,
                   kCoopHigh = 1u << 31;
__device__ __forceinline__ uint32_t coop_site(const LevelView &L, int x, int y)
{
    return (uint32_t)site_of(L, x, y) | (x == 0 ? kCoopLeft : 0u) | (x + 1 == L.W ? kCoopRight : 0u) |
           (y == 0 ? kCoopLow : 0u) | (y + 1 == L.H ? kCoopHigh : 0u);
}

struct CoopRange // a block's cells of one kind and level, or rows (lo in warps, 32 "cells" to a warp)
{
    int lo, cells; // first cell, cells
    int n, line;   // warps of cells or rows, first line; coop_place: n of the ranges before
    __device__ __forceinline__ int warps() const { return (cells + 31) >> 5; }
};

// Slots of a cell.  A step reads and writes the same nine: on plane p its own
// site's (even step) or that of the site at +c_p (odd step); they hold the
// populations p / opp(p) before and opp(p) / p after the step.  The plane and row
// strides are read anew per cell (volatile): nine plane offsets kept in registers
// over the loops would cost the kernel a third of its warps.
struct CoopSlots
{
    float *f;
    uint32_t at[9];
    int par;
    __device__ __forceinline__ CoopSlots(const LevelView &L, const volatile uint2 *stride, uint32_t site, int parity)
        : f(L.f), par(parity)
    {
        const uint32_t plane = stride->x, s = site & kCoopSite;
        uint32_t up = stride->y, down = 0u - up, right = 1u, left = 0u - 1u;
        if (site & ~kCoopSite)
        {
            if (site & kCoopHigh) up -= (uint32_t)L.H * up;
            if (site & kCoopLow) down += (uint32_t)L.H * stride->y;
            if (site & kCoopRight) right -= (uint32_t)L.W;
            if (site & kCoopLeft) left += (uint32_t)L.W;
        }
        if (!par) up = down = right = left = 0u;
#pragma unroll
        for (int p = 0; p < 9; p++)
            at[p] = s + (d2q9::cy(p) > 0 ? up : d2q9::cy(p) < 0 ? down : 0u) +
                    (d2q9::cx(p) > 0 ? right : d2q9::cx(p) < 0 ? left : 0u) + p * plane;
    }
    __device__ __forceinline__ void read(float v[9]) const
    {
        float w[9];
#pragma unroll
        for (int p = 0; p < 9; p++) w[p] = f[at[p]];
#pragma unroll
        for (int q = 0; q < 9; q++) v[q] = par ? w[d2q9::opp(q)] : w[q];
    }
    __device__ __forceinline__ void write(const float v[9]) const
    {
#pragma unroll
        for (int p = 0; p < 9; p++) f[at[p]] = par ? v[p] : v[d2q9::opp(p)];
    }
    // values into the slots that a step of this parity reads
    __device__ __forceinline__ void fill(const float v[9]) const
    {
#pragma unroll
        for (int p = 0; p < 9; p++) f[at[p]] = par ? v[d2q9::opp(p)] : v[p];
    }
};

struct CoopStep // block-uniform state of one level in one phase
{
    StepOpt o;
    int diff, store_u;
    int collision, wall;
};

__device__ __forceinline__ SpecialRec coop_record(const float *line, int lane)
{
    union
    {
        SpecialRec rec;
        uint4 v[2];
    } t;
    static_assert(sizeof(SpecialRec) == 2 * sizeof(uint4), "record size");
    t.v[0] = reinterpret_cast<const uint4 *>(line)[lane];
    t.v[1] = reinterpret_cast<const uint4 *>(line)[32 + lane];
    return t.rec;
}

// Moments, residual and collision of a cell with the populations df.  snap: where
// its coarse-step-start moments are kept, three values `stride` apart; sn: these,
// loaded ahead (snap_use).
template <bool SPECIAL, bool RES>
__device__ __forceinline__ void coop_collide(const CoopDesc &D, const CoopStep &st, int64_t s, const float df[9], float *snap,
                                             int64_t stride, const float sn[3], float omega, const SpecialRec &rec,
                                             float *unorm, double2 *acc, float fs[9])
{
    float drho, rho, ux, uy;
    macro(df, D.C.rho0, D.L.fshift, 0.0f, drho, rho, ux, uy);
    if (RES && (st.diff | st.store_u))
    {
        const float un = sqrtf(ux * ux + uy * uy);
        if (st.diff)
        {
            double2 v = *acc;
            v.x += (double)fabsf(un - *unorm);
            v.y += (double)un;
            *acc = v;
        }
        if (st.store_u) *unorm = un;
    }
    if (st.o.snap_store && snap)
    {
        snap[0] = drho;
        snap[stride] = ux;
        snap[2 * stride] = uy;
    }
    float edrho = drho, erho = rho, eux = ux, euy = uy;
    if (st.o.snap_use)
    {
        edrho = sn[0];
        erho = D.C.rho0 + edrho;
        eux = sn[1];
        euy = sn[2];
    }
    collide_cell(D.L, D.C, st.collision, st.wall, st.o.parity, s, df, edrho, erho, eux, euy, omega, SPECIAL, rec, fs);
}

// One special cell from its record.
template <bool HEAVY, bool RES>
__device__ __forceinline__ void coop_special(const CoopDesc &D, const CoopStep &st, const volatile uint2 *stride,
                                             const SpecialRec &rec, float *unorm, double2 *acc)
{
    const LevelView &L = D.L;
    const int x = rec.xy & 0xFFFF, y = rec.xy >> 16;
    const int64_t s = site_of(L, x, y);
    const int par = st.o.parity;
    const uint32_t site = coop_site(L, x, y);
    float sn[3] = {0.f, 0.f, 0.f}, df[9], fs[9];
    if (st.o.snap_use) load_snap<false>(L, s, sn);
    if (((rec.m1 >> 17) & SF_BUFFER) && (st.o.first_sub || st.o.direct))
    {
#pragma unroll
        for (int q = 0; q < 9; q++) df[q] = D.C.ibuf[(size_t)q * D.C.n_buf + rec.buf];
    }
    else
    {
        // (a direct state has parity 0: own slots)
        float raw[9];
        CoopSlots(L, stride, site, par).read(raw);
        if (st.o.direct || !HEAVY)
        {
#pragma unroll
            for (int q = 0; q < 9; q++) df[q] = raw[q];
            if (!st.o.direct) light_rules(D.C, rec, df);
        }
        else
        {
            // a wall link's value lies where the previous step stored it
            const CoopSlots before(L, stride, site, par ^ 1);
            special_rules(D.C, rec, par, st.wall, raw,
                          [&](int q) { return &L.f[par ? before.at[d2q9::opp(q)] : before.at[q]]; }, df);
        }
    }
    coop_collide<HEAVY, RES>(D, st, s, df, L.snap ? L.snap + s : nullptr, L.plane, sn, rec.omega, rec, unorm, acc, fs);
    CoopSlots(L, stride, site, par).write(fs);
}

// The index, hidden from the compiler: descriptor fields are then read where they
// are used (from the parameter bank) and not held in registers over the loops.
__device__ __forceinline__ int coop_opaque(int d)
{
    asm volatile("" : "+r"(d));
    return d;
}

// The warps of a block claim its warps of cells (or rows) of a stage in order from
// a counter in shared memory, the long ones first: special cells take two to
// three times as long as plain ones, and a stage ends with its last warp.
struct CoopClaim
{
    unsigned int *next;
    int base, mine; // items before the current list, this warp's claim
    __device__ __forceinline__ explicit CoopClaim(unsigned int *counter) : next(counter), base(0) { claim(); }
    __device__ __forceinline__ void claim()
    {
        unsigned int v = 0;
        if ((threadIdx.x & 31) == 0) v = atomicAdd(next, 1u);
        mine = (int)__shfl_sync(0xffffffffu, v, 0);
    }
};

// One phase of one level over this block's cells.
template <bool RES>
__device__ __forceinline__ void coop_level(const CoopLaunch &A, int d, const CoopStep &st, const CoopRange *rng,
                                           const volatile uint2 *stride, float *sm, CoopClaim &claim, double2 *acc)
{
    const int lane = threadIdx.x & 31;
    {
        const CoopRange r = rng[CK_HEAVY];
#pragma unroll 1
        for (int i; (i = claim.mine - claim.base) < r.n; claim.claim())
        {
            const CoopDesc &D = A.d[coop_opaque(d)];
            const LevelView &L = D.L;
            if (i * 32 + lane >= r.cells) continue;
            float *m = sm + (size_t)(r.line + i * kCoopRecLines) * 32;
            coop_special<true, RES>(D, st, stride, coop_record(m, lane), m + 8 * 32 + lane, acc);
        }
        claim.base += r.n;
    }
    {
        const CoopRange r = rng[CK_LIGHT];
#pragma unroll 1
        for (int i; (i = claim.mine - claim.base) < r.n; claim.claim())
        {
            const CoopDesc &D = A.d[coop_opaque(d)];
            const LevelView &L = D.L;
            if (i * 32 + lane >= r.cells) continue;
            float *m = sm + (size_t)(r.line + i * kCoopRecLines) * 32;
            coop_special<false, RES>(D, st, stride, coop_record(m, lane), m + 8 * 32 + lane, acc);
        }
        claim.base += r.n;
    }
    const SpecialRec none{};
#pragma unroll 1
    for (int kind = CK_EDGE; kind <= CK_PLAIN; kind++)
    {
        // CK_PLAIN keeps its coarse-step-start moments in shared memory (where a
        // later substep uses them), CK_EDGE in the planes the waves read
        const CoopRange r = rng[kind];
        const int lines = A.d[d].lines[kind];
        const bool own = kind == CK_PLAIN;
#pragma unroll 1
        for (int i; (i = claim.mine - claim.base) < r.n; claim.claim())
        {
            const CoopDesc &D = A.d[coop_opaque(d)];
            const LevelView &L = D.L;
            float *m = sm + (size_t)(r.line + i * lines) * 32 + lane;
            const uint32_t site = __float_as_uint(m[0]), s = site & kCoopSite;
            if (site == kCoopNone) continue;
            float df[9], fs[9], sn[3] = {0.f, 0.f, 0.f};
            CoopSlots(L, stride, site, st.o.parity).read(df);
            float *snap = !own ? L.snap + s : lines > kCoopPlainLines ? m + kCoopPlainLines * 32 : nullptr;
            const int64_t step = own ? 32 : L.plane;
            if (st.o.snap_use)
            {
                sn[0] = snap[0];
                sn[1] = snap[step];
                sn[2] = snap[2 * step];
            }
            coop_collide<false, RES>(D, st, s, df, snap, step, sn, m[32], none, m + 64, acc, fs);
            CoopSlots(L, stride, site, st.o.parity).write(fs);
        }
        claim.base += r.n;
    }
}

// ---- interface waves of the cooperative steps.  The rows' tables wait in shared
// memory lane by lane (8 rows of 4 lanes to a warp), so the populations and
// the coarse-step-start moments of a row are one round trip to memory; the
// arithmetic is that of coarse_row / fine_child, which step the few rows that
// touch a special source or the level's border.
constexpr int kCoopCoarseLines = 3, kCoopFineLines = 12;
constexpr uint32_t kCoopAbsent = 0xFFFFFFFFu, kCoopBuf = 0x80000000u;

// a source or target of a row off the border is known by its site
__device__ __forceinline__ bool coop_inner_site(const LevelView &L, int site)
{
    const int x = site % L.pitch, y = site / L.pitch;
    return x > 0 && x + 1 < L.W && y > 0 && y + 1 < L.H;
}
__device__ __forceinline__ uint32_t coop_source(const LevelView &L, int site, int buf, bool &slow)
{
    if (site < 0) return kCoopAbsent;
    if (buf >= 0) return kCoopBuf | (uint32_t)buf;
    slow |= !coop_inner_site(L, site);
    return (uint32_t)site;
}
__device__ __forceinline__ void coop_read_source(const LevelView &L, const volatile uint2 *stride, int par, const Common &C,
                                                 uint32_t src, float z[9])
{
    if (src & kCoopBuf)
    {
#pragma unroll
        for (int q = 0; q < 9; q++) z[q] = C.ibuf[(size_t)q * C.n_buf + (src & ~kCoopBuf)];
    }
    else CoopSlots(L, stride, src, par).read(z);
}

// fills the lines of one warp of rows (r: this lane's row, k: its place in the row)
__device__ __forceinline__ void coop_fill_coarse(const CoopPair &Q, const LevelView &Lf, const LevelView &Lc, int r, int k,
                                                 float *m)
{
    const int lane = threadIdx.x & 31;
    bool slow = false;
    uint32_t src = kCoopAbsent, word = 0;
    if (r < Q.ncoarse)
    {
        const CoarseRowDev &row = Q.coarse[r];
        src = coop_source(Lf, row.child[k], row.child_buf[k], slow);
        slow |= row.special || (row.plain_target && !coop_inner_site(Lc, row.site));
        word = k == 0   ? (uint32_t)row.site
               : k == 1 ? (uint32_t)row.buf | (row.plain_target ? kCoopBuf : 0u)
               : k == 2 ? __float_as_uint(row.ratio)
                        : __float_as_uint(row.inv_nchild);
    }
    m[lane] = __uint_as_float(src);
    m[32 + lane] = __uint_as_float(word);
    m[64 + lane] = __int_as_float(slow);
}
__device__ __forceinline__ void coop_fill_fine(const CoopPair &Q, const LevelView &Lf, const LevelView &Lc, int r, int c, float *m)
{
    const int lane = threadIdx.x & 31;
    bool slow = false;
    uint32_t a = kCoopAbsent, b = kCoopAbsent, at = 0, buf = 0;
    float w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, ratio = 0.f;
    if (r < Q.nfine)
    {
        const FineRowDev &row = Q.fine[r];
        a = coop_source(Lc, row.node_site[c], row.node_buf[c], slow);
        if (c < 2) b = coop_source(Lc, row.node_site[c + 4], row.node_buf[c + 4], slow);
#pragma unroll
        for (int j = 0; j < 6; j++) w[j] = row.weight[c][j];
        ratio = row.ratio[c];
        at = (uint32_t)row.child_site[c];
        const bool plain = (row.plain_mask >> c) & 1;
        buf = (uint32_t)row.child_buf[c] | (plain ? kCoopBuf : 0u);
        slow |= row.special || (plain && !coop_inner_site(Lf, row.child_site[c]));
    }
    m[lane] = __uint_as_float(a);
    m[32 + lane] = __uint_as_float(b);
#pragma unroll
    for (int j = 0; j < 6; j++) m[(2 + j) * 32 + lane] = w[j];
    m[8 * 32 + lane] = ratio;
    m[9 * 32 + lane] = __uint_as_float(at);
    m[10 * 32 + lane] = __uint_as_float(buf);
    m[11 * 32 + lane] = __int_as_float(slow);
}

// One level as the waves see it: its view, strides and the parity of its next step
struct CoopSide
{
    const LevelView &L;
    const volatile uint2 *stride;
    int par;
};

// coarse_row for 8 rows of a warp
__device__ __forceinline__ void coop_coarse(const CoopSide &F, const CoopSide &Cd, const Common &C, const float *m, bool valid)
{
    const int lane = threadIdx.x & 31, base = lane & ~3;
    const uint32_t src = __float_as_uint(m[lane]);
    const uint4 t = reinterpret_cast<const uint4 *>(m + 32)[lane >> 2];
    const bool has = src != kCoopAbsent, out = valid && (lane & 3) == 0;
    float df[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (has) coop_read_source(F.L, F.stride, F.par, C, src, df);
    float drho = 0.f, ux = 0.f, uy = 0.f;
    if (out)
    {
        const float *sn = Cd.L.snap + t.x;
        drho = sn[0];
        ux = sn[Cd.L.plane];
        uy = sn[2 * Cd.L.plane];
    }
    float mean[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int kk = 0; kk < 4; kk++)
    {
        const bool present = __shfl_sync(0xffffffffu, has ? 1 : 0, base + kk) != 0;
#pragma unroll
        for (int q = 0; q < 9; q++)
        {
            const float v = __shfl_sync(0xffffffffu, df[q], base + kk);
            if (present) mean[q] += v;
        }
    }
    if (!out) return;
    float feq[9];
    equilibrium(drho, C.rho0 + drho, ux, uy, feq);
    const uint32_t buf = t.y & ~kCoopBuf;
    const float ratio = __uint_as_float(t.z), inv_nchild = __uint_as_float(t.w);
    float v[9];
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        v[q] = feq[q] + ratio * (mean[q] * inv_nchild - feq[q]);
        C.ibuf[(size_t)q * C.n_buf + buf] = v[q];
    }
    if (t.y & kCoopBuf) CoopSlots(Cd.L, Cd.stride, t.x, Cd.par).fill(v);
}

// fine_child for 8 rows of a warp
__device__ __forceinline__ void coop_fine(const CoopSide &F, const CoopSide &Cd, const Common &C, const float *m, bool valid)
{
    const int lane = threadIdx.x & 31, base = lane & ~3;
    const uint32_t a = __float_as_uint(m[lane]), b = __float_as_uint(m[32 + lane]);
    const uint32_t at = __float_as_uint(m[9 * 32 + lane]), buf = __float_as_uint(m[10 * 32 + lane]);
    float za[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, zb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (a != kCoopAbsent) coop_read_source(Cd.L, Cd.stride, Cd.par, C, a, za);
    if (b != kCoopAbsent) coop_read_source(Cd.L, Cd.stride, Cd.par, C, b, zb);
    float drho = 0.f, ux = 0.f, uy = 0.f;
    if (valid)
    {
        const float *sn = F.L.snap + at;
        drho = sn[0];
        ux = sn[F.L.plane];
        uy = sn[2 * F.L.plane];
    }
    float acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 6; k++)
    {
        const float w = m[(2 + k) * 32 + lane];
#pragma unroll
        for (int q = 0; q < 9; q++)
        {
            const float z = __shfl_sync(0xffffffffu, k < 4 ? za[q] : zb[q], base + (k & 3));
            acc[q] += w * z;
        }
    }
    if (!valid) return;
    float feq[9];
    equilibrium(drho, C.rho0 + drho, ux, uy, feq);
    const float rat = m[8 * 32 + lane];
#pragma unroll
    for (int q = 0; q < 9; q++)
    {
        acc[q] = feq[q] + rat * (acc[q] - feq[q]);
        C.ibuf[(size_t)q * C.n_buf + (buf & ~kCoopBuf)] = acc[q];
    }
    if (buf & kCoopBuf) CoopSlots(F.L, F.stride, at, F.par).fill(acc);
}

// First line of each of `count` ranges, whose lines start at `line`, and (in n) the
// number of warps before it; returns the line after them.  One warp, 32 ranges at a time.
template <typename Lines>
__device__ __forceinline__ int coop_place(CoopRange *rng, int count, int line, Lines lines_of)
{
    const int lane = threadIdx.x & 31;
    int all = 0;
    for (int t0 = 0; t0 < count; t0 += 32)
    {
        const int t = t0 + lane, n = t < count ? rng[t].warps() : 0, own = t < count ? n * lines_of(t) : 0;
        int sn = n, sl = own; // sums up to and with this lane
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int un = __shfl_up_sync(0xffffffffu, sn, o), ul = __shfl_up_sync(0xffffffffu, sl, o);
            if (lane >= o) sn += un, sl += ul;
        }
        if (t < count)
        {
            rng[t].line = line + sl - own;
            rng[t].n = all + sn - n;
        }
        all += __shfl_sync(0xffffffffu, sn, 31);
        line += __shfl_sync(0xffffffffu, sl, 31);
    }
    return line;
}

// The block's warps of cells (or rows) of all ranges, numbered through: warp w takes
// w, w + nw, ...; find() advances to the range of one.
struct CoopItems
{
    const CoopRange *rng;
    int count, total, t;
    __device__ __forceinline__ CoopItems(const CoopRange *r, int n)
        : rng(r), count(n), total(n ? r[n - 1].n + r[n - 1].warps() : 0), t(0)
    {
    }
    __device__ __forceinline__ void find(int i)
    {
        while (t + 1 < count && i >= rng[t + 1].n) t++;
    }
};

// Fills the block's shared memory (BACK false), or writes the stored |u| back.  A
// warp has kCoopFill warps of cells in flight, of whichever image, level and kind: a
// launch pays a few round trips to memory for it.  (List by list, one warp of cells at
// a time, a call of one step of eight 512^2 images of two levels took 345 us; now 301.)
template <bool BACK, bool RES>
__device__ __forceinline__ void coop_cells(const CoopLaunch &A, const CoopRange *rng, float *sm)
{
    constexpr int kCoopFill = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    CoopItems items(rng, A.nd * CK_KINDS);
#pragma unroll 1
    for (int i0 = warp; i0 < items.total; i0 += kCoopFill * nw)
    {
        int at[kCoopFill], xy[kCoopFill]; // range, position; -1: none
        float *m[kCoopFill];
#pragma unroll
        for (int u = 0; u < kCoopFill; u++)
        {
            const int i = i0 + u * nw;
            at[u] = xy[u] = -1;
            if (i >= items.total) continue;
            items.find(i);
            const CoopRange &r = rng[items.t];
            const CoopDesc &D = A.d[items.t / CK_KINDS];
            const int kind = items.t % CK_KINDS, k = i - r.n, c = r.lo + k * 32 + lane;
            at[u] = items.t;
            m[u] = sm + (size_t)(r.line + k * D.lines[kind]) * 32;
            if (k * 32 + lane >= r.cells) continue;
            if (kind >= CK_EDGE) xy[u] = __ldg(&D.xy[kind][c]);
            else
            {
                const SpecialRec *rec = D.C.specials + D.spec_begin + (kind == CK_LIGHT ? D.nheavy : 0) + c;
                if (BACK) xy[u] = rec->xy;
                else
                {
                    const uint4 r0 = reinterpret_cast<const uint4 *>(rec)[0], r1 = reinterpret_cast<const uint4 *>(rec)[1];
                    reinterpret_cast<uint4 *>(m[u])[lane] = r0;
                    reinterpret_cast<uint4 *>(m[u])[32 + lane] = r1;
                    xy[u] = (int)r1.z;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kCoopFill; u++)
        {
            if (at[u] < 0) continue;
            const CoopDesc &D = A.d[at[u] / CK_KINDS];
            const int kind = at[u] % CK_KINDS;
            const bool there = xy[u] >= 0;
            if (!BACK && kind >= CK_EDGE)
            {
                const uint32_t site = there ? coop_site(D.L, xy[u] & 0xFFFF, xy[u] >> 16) : kCoopNone;
                m[u][lane] = __uint_as_float(site);
                if (there) m[u][32 + lane] = D.L.omega[site & kCoopSite];
            }
            if (!there || !RES) continue;
            float *un = m[u] + (kind >= CK_EDGE ? 2 : 8) * 32 + lane;
            float *g = &D.L.unorm[site_of(D.L, xy[u] & 0xFFFF, xy[u] >> 16)];
            if (BACK) *g = *un;
            else *un = *g;
        }
    }
}

__device__ __forceinline__ int coop_place_cells(const CoopLaunch &A, CoopRange *rng)
{
    return coop_place(rng, A.nd * CK_KINDS, 0, [&](int t) { return A.d[t / CK_KINDS].lines[t % CK_KINDS]; });
}

// The places of a block's lists in shared memory, and their content.  (A call: inlined,
// it cost the stages' loops up to 0.6 % by the registers and places they got.)
template <bool RES>
__device__ __noinline__ void coop_start(const CoopLaunch &A, CoopRange *rng, CoopRange *rows, unsigned int *next, float *sm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (warp == 0)
    {
        if (lane == 0) *next = 0u;
        const int line = coop_place_cells(A, rng);
        coop_place(rows, A.np * 2, line, [](int t) { return t & 1 ? kCoopFineLines : kCoopCoarseLines; });
    }
    __syncthreads();
    coop_cells<false, RES>(A, rng, sm);
    CoopItems waves(rows, A.np * 2);
    for (int i = warp; i < waves.total; i += nw)
    {
        waves.find(i);
        const int t = waves.t, k = i - rows[t].n, r = (rows[t].lo + k) * 8 + lane / 4;
        const CoopPair &Q = A.p[t / 2];
        const LevelView &Lf = A.d[Q.df].L, &Lc = A.d[Q.dc].L;
        if (t & 1) coop_fill_fine(Q, Lf, Lc, r, lane & 3, sm + (size_t)(rows[t].line + k * kCoopFineLines) * 32);
        else coop_fill_coarse(Q, Lf, Lc, r, lane & 3, sm + (size_t)(rows[t].line + k * kCoopCoarseLines) * 32);
    }
    __syncthreads();
    for (int t = (int)threadIdx.x; t < A.nd * CK_KINDS; t += (int)blockDim.x) rng[t].n = rng[t].warps();
    for (int t = (int)threadIdx.x; t < A.np * 2; t += (int)blockDim.x) rows[t].n = rows[t].warps();
}

// The block has passed its last barrier: the last block to come here clears the
// counters for the next launch (a memset before each launch took as long as half a
// step of a small image).  Where a barrier's wait ran out (!ok), every image of the
// launch is left half stepped and noted so.
__device__ __forceinline__ void coop_leave(const CoopLaunch &A, bool ok)
{
    if (!ok)
        for (int d = (int)threadIdx.x; d < A.nd; d += (int)blockDim.x) atomicOr(A.d[d].C.err, kErrDepTimeout);
    if (threadIdx.x != 0) return;
    __threadfence(); // this block's arrivals come before its leave
    if (atomicAdd(A.bar + 1, 1u) + 1u == gridDim.x) A.bar[0] = A.bar[1] = 0u;
}

// DEF: every image has the default regularized MRT and SRBB walls (their code
// alone then passes through the instruction cache); RES: with residuals (A.every)
template <int THREADS, bool DEF, bool RES>
__global__ void __launch_bounds__(THREADS, 1) k_coop_steps(const __grid_constant__ CoopLaunch A)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ CoopRange rng[kMaxCoopDescs * CK_KINDS], rows[kMaxCoopPairs * 2]; // coarse, fine rows
    __shared__ uint2 strides[kMaxCoopDescs]; // floats per plane and per row
    __shared__ unsigned int s_next;          // next unclaimed item of a stage
    __shared__ double2 s_sums[32];           // the warps' residual terms
    // this thread's residual terms (in shared memory: registers are what limits the
    // warps of an SM), then the lines
    double2 *acc = reinterpret_cast<double2 *>(sm_raw) + threadIdx.x;
    float *sm = reinterpret_cast<float *>(sm_raw + (RES ? THREADS * sizeof(double2) : 0));
    const int b = (int)blockIdx.x, G = (int)gridDim.x;
    for (int t = (int)threadIdx.x; t < A.nd * CK_KINDS; t += (int)blockDim.x)
    {
        const int32_t *cut = A.d[t / CK_KINDS].cut[t % CK_KINDS];
        rng[t].lo = cut[b];
        rng[t].cells = cut[b + 1] - rng[t].lo;
    }
    for (int t = (int)threadIdx.x; t < A.nd; t += (int)blockDim.x)
        strides[t] = make_uint2((uint32_t)A.d[t].L.plane, (uint32_t)A.d[t].L.pitch);
    for (int t = (int)threadIdx.x; t < A.np * 2; t += (int)blockDim.x)
    {
        const CoopPair &Q = A.p[t / 2];
        const int W = ((t & 1 ? Q.nfine : Q.ncoarse) + 7) / 8;
        rows[t].lo = coop_cut(W, Q.rot, b, G);
        rows[t].cells = (coop_cut(W, Q.rot, b + 1, G) - rows[t].lo) * 32;
    }
    __syncthreads();
    coop_start<RES>(A, rng, rows, &s_next, sm);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // every step; false where a barrier's wait ran out
    auto steps = [&]() -> bool {
        unsigned int target = 0;
        int since = A.since0, prev = since == 0 ? A.every - 1 : since - 1;
#pragma unroll 1
        for (int k = 0; k < A.nsteps; k++)
        {
            const bool store = RES && since == 0; // this step's number is a multiple of A.every
            const bool diff = RES && prev == 0 && !(k == 0 && A.skip_first);
            if (RES)
            {
                prev = since;
                since = since + 1 == A.every ? 0 : since + 1;
            }
#pragma unroll 1
            for (int ph = 0; ph < A.nphase; ph++)
            {
                CoopClaim claim(&s_next);
                if (RES && diff && ph == 0) *acc = make_double2(0.0, 0.0);
#pragma unroll 1
                for (int d = 0; d < A.nd; d++)
                {
                    const CoopDesc &D = A.d[d];
                    if (ph & ((1 << D.shift) - 1)) continue;
                    const int sub = ph >> D.shift;
                    CoopStep st{};
                    st.o.parity = (D.parity0 + k * D.substeps + sub) & 1;
                    st.o.direct = k == 0 && sub == 0 && D.direct0;
                    st.o.first_sub = sub == 0;
                    st.o.snap_store = D.mb && sub == 0;
                    st.o.snap_use = D.mb && sub > 0;
                    st.diff = diff && sub == 0;
                    st.store_u = store && sub == 0;
                    st.collision = DEF ? COLL_RMRT : D.C.collision;
                    st.wall = DEF ? WALL_SRBB : D.C.wall;
                    coop_level<RES>(A, d, st, rng + d * CK_KINDS, strides + d, sm, claim, acc);
                }
                if (RES && diff && ph == 0) block_sums(acc->x, acc->y, s_sums);
                const bool end = k + 1 == A.nsteps && ph + 1 == A.nphase && A.nwave == 0;
                if (RES && diff && ph == 0)
                {
                    double *red = A.d[0].C.red + (size_t)((uint32_t)(A.slot0 + k) % (uint32_t)A.ring) * 4;
                    if (!end)
                    {
                        target += gridDim.x;
                        if (!grid_barrier(A.bar, target, A.polls, nullptr, nullptr, &s_next, s_sums, red)) return false;
                        continue;
                    }
                    __syncthreads();
                    if (warp == 1) add_block_sums(s_sums, red);
                }
                if (end) break;
                target += gridDim.x;
                if (!grid_barrier(A.bar, target, A.polls, nullptr, nullptr, &s_next)) return false;
            }
#pragma unroll 1
            for (int w = 0; w < A.nwave; w++)
            {
                CoopClaim claim(&s_next);
#pragma unroll 1
                for (int p = 0; p < A.np; p++)
                {
                    const CoopPair &Q = A.p[p];
                    const int kind = Q.l1 - 1 == w ? 0 : Q.l1 == w ? 1 : -1; // coarse rows / fine rows
                    if (kind < 0) continue;
                    const CoopRange rr = rows[p * 2 + kind];
                    const int nrows = kind == 0 ? Q.ncoarse : Q.nfine;
                    const CoopDesc &F = A.d[Q.df], &Cd = A.d[Q.dc];
                    const int pf = (F.parity0 + (k + 1) * F.substeps) & 1, pc = (Cd.parity0 + (k + 1) * Cd.substeps) & 1;
                    const CoopSide fine{F.L, strides + Q.df, pf}, coarse{Cd.L, strides + Q.dc, pc};
#pragma unroll 1
                    for (int i; (i = claim.mine - claim.base) < rr.n; claim.claim())
                    {
                        const int r = (rr.lo + i) * 8 + lane / 4;
                        const bool valid = r < nrows;
                        const float *m = sm + (size_t)(rr.line + i * (kind == 0 ? kCoopCoarseLines : kCoopFineLines)) * 32;
                        const bool slow = __any_sync(0xffffffffu, __float_as_int(m[(kind == 0 ? 2 : 11) * 32 + lane]) != 0);
                        if (kind == 0)
                        {
                            const CoarseRowDev &row = Q.coarse[valid ? r : 0];
                            if (!slow) coop_coarse(fine, coarse, F.C, m, valid);
                            else if (pf) coarse_row<1>(F.L, Cd.L, F.C, row, lane & 3, valid, pc);
                            else coarse_row<0>(F.L, Cd.L, F.C, row, lane & 3, valid, pc);
                        }
                        else
                        {
                            const FineRowDev &row = Q.fine[valid ? r : 0];
                            if (!slow) coop_fine(fine, coarse, F.C, m, valid);
                            else if (pc) fine_child<1>(F.L, Cd.L, F.C, row, lane & 3, valid, pf);
                            else fine_child<0>(F.L, Cd.L, F.C, row, lane & 3, valid, pf);
                        }
                    }
                    claim.base += rr.n;
                }
                if (k + 1 == A.nsteps && w + 1 == A.nwave) break;
                target += gridDim.x;
                if (!grid_barrier(A.bar, target, A.polls, nullptr, nullptr, &s_next)) return false;
            }
        }
        return true;
    };
    const bool ok = steps();
    coop_leave(A, ok);
    if (RES && ok)
    {
        __syncthreads(); // the last stage has no barrier: other warps' |u| are still being stored
        if (warp == 0) coop_place_cells(A, rng);
        __syncthreads();
        coop_cells<true, RES>(A, rng, sm);
    }
}

// f = f_eq(rho, u) per reference cell, written into its own slots (state then
// reads "direct") and, for interface buffers, into the interpolation buffer.
__global__ void k_set_equilibrium(AllLevels A, Common C, const int32_t *cell_level, const int32_t *cell_site, int64_t n,
                                  const double *rho, const double *ux, const double *uy)
{
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int l = cell_level[c] - 1;
    const LevelView &L = A.lv[l];
    const int s = cell_site[c];
    const double r = rho[c], vx = ux[c], vy = uy[c];
    const double usq = vx * vx + vy * vy;
    float df[9];
    for (int q = 0; q < 9; q++)
    {
        const double cu = d2q9::cx(q) * vx + d2q9::cy(q) * vy;
        // deviation from w rho0, formed in FP64 before rounding
        const double feq = d2q9::w(q) * r * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * usq);
        df[q] = (float)(feq - d2q9::w(q) * (double)C.rho0);
        L.f[(size_t)q * L.plane + s] = df[q];
    }
    if (L.rho_prev)
    {
        // the same FP32 sum as the first step's density, so an unchanged state
        // reads as no change
        float drho = 0.0f;
        for (int q = 0; q < 9; q++) drho += df[q];
        L.rho_prev[s] = C.rho0 + drho;
    }
    if (L.snap)
    {
        L.snap[s] = (float)(r - (double)C.rho0);
        L.snap[L.plane + s] = (float)vx;
        L.snap[2 * L.plane + s] = (float)vy;
    }
    if (L.omega[s] < 0.0f)
    {
        const SpecialRec rec = C.specials[L.spec[s]];
        if (((rec.m1 >> 17) & 0xFu) & SF_BUFFER)
            for (int q = 0; q < 9; q++) C.ibuf[(size_t)q * C.n_buf + rec.buf] = df[q];
    }
}
// Restart: the populations f (FP64, 9 per cell in cell order) become the state
// in the slots the first step reads directly, as after k_set_equilibrium; the
// residual side arrays take the moments of f with the FP32 arithmetic of a step.
__global__ void k_set_distributions(AllLevels A, Common C, const int32_t *cell_level, const int32_t *cell_site,
                                    int64_t n, const double *f)
{
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int l = cell_level[c] - 1;
    const LevelView &L = A.lv[l];
    const int s = cell_site[c];
    float df[9];
    for (int q = 0; q < 9; q++)
    {
        df[q] = (float)(f[c * 9 + q] - d2q9::w(q) * (double)C.rho0);
        L.f[(size_t)q * L.plane + s] = df[q];
    }
    float drho, rho, ux, uy;
    macro(df, C.rho0, L.fshift, 0.0f, drho, rho, ux, uy);
    if (L.unorm) L.unorm[s] = sqrtf(ux * ux + uy * uy);
    if (L.rho_prev)
    {
        float sum = 0.0f;
        for (int q = 0; q < 9; q++) sum += df[q];
        L.rho_prev[s] = C.rho0 + sum;
    }
    if (L.snap)
    {
        L.snap[s] = drho;
        L.snap[L.plane + s] = ux;
        L.snap[2 * L.plane + s] = uy;
    }
    if (L.omega[s] < 0.0f)
    {
        const SpecialRec rec = C.specials[L.spec[s]];
        if (((rec.m1 >> 17) & 0xFu) & SF_BUFFER)
            for (int q = 0; q < 9; q++) C.ibuf[(size_t)q * C.n_buf + rec.buf] = df[q];
    }
}
} // namespace dev
} // namespace mantiis
