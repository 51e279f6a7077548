// fe_mg_body.cuh -- multigrid-preconditioned conjugate gradient for the pressure system, as the body of a
// persistent cooperative kernel (k_mgcg, and per scene inside k_multi_cg).
//
// Same system, same FP64 outer refinement and same convergence test as the plain solver (fe_cg.cu; the
// reference system of single_phase_pressure_solver.cpp:99-164 with the reference's relative residual
// target); only the inner FP32 solve of A e = r changes: preconditioned CG whose preconditioner is one
// multigrid V-cycle.  Results agree with the plain solver and with the reference to the solve tolerance (both stop
// on the same FP64 residual test).
//
// Hierarchy: level l >= 1 halves every axis of level l-1 (rounding up) until the largest axis is <= 8.  phi, the
// fluid fraction of a coarse cell, is the mean of its children's, BOUNDRY cells left out; a coarse cell is in the system when
// phi > kMaskPhi, and one of nothing but BOUNDRY cells is a wall.
// Its operator is the 7-point matrix with spacing 2^l h, except that the coefficient toward a cell outside the system
// is h_l^-2 / d, d the distance (in h_l) from the cell's centre to the air value (0) as the fractions put it:
// half the fluid of the cell's own half on that side, all of the neighbour's, and half a level-0 cell.  A coarse cell
// centre lies up to half a coarse cell away from where the level-0 surface is, and with the plain coefficient (d = 1)
// the coarse correction is wrong there by that much: inner iterations to 1e-6 with / without d on the 64^3 and 128^3
// dam breaks 7 / 9 and 7 / 10.  A cell none of whose neighbours is air adds kInnerAir (h_x^-2 + h_y^-2 + h_z^-2)
// sqrt(1 - phi): air pockets inside it hold the pressure down, which no side's coefficient tells, and without it the coarse
// correction overshoots wherever fluid has splashed.
//
// V-cycle (symmetric, so the preconditioner is SPD): two Jacobi sweeps with the weights of the degree-2 Chebyshev
// polynomial on [kChebLow, 2] (the spectrum of D^-1 A lies in (0, 2]) down, starting from zero; residual;
// restriction = kRestrictScale x the transpose of the prolongation; the coarsest level gets kCoarseSweeps Chebyshev
// sweeps from zero in one block's shared memory; up: z = z + P z_coarse, then the same two sweeps.  P is
// cell-centred trilinear: per axis a fine cell takes 3/4 of its parent and 1/4 of the parent's neighbour on its side
// (the parent again at a wall).  One damped Jacobi sweep each way (0.9) took 15 / 17 iterations where this takes 7 / 7.
//
// What bounds an iteration at 128^3 and below is the number of grid-wide passes, each a barrier plus the latency of
// its loads; so every pass does as much as a halo of two cells in shared memory allows.  Work is dealt in tiles of
// 8^3 cells, one tile per team of threads at a time; a team loads the tile with the cells within two steps of
// it and takes both sweeps and the residual (down) or the correction and both sweeps (up) from there, so each level
// costs one barrier going down and one going up.  The restriction is summed per tile in shared memory first, so a
// tile adds at most 6^3 coarse values with global atomics instead of 8 per cell (4.1 M atomics an iteration at
// 128^3).  Only tiles that hold cells of the system are listed; teams take them round-robin over the blocks.
//
// Passes (grid barriers) per inner iteration, L levels: A: x, r update, level 0's sweeps, residual and restriction
// (carries ||r||^2); D: the same for each level 1 .. L-2; the coarsest solve; U: correction and sweeps for each level
// L-2 .. 0 (level 0 carries (r, z)); C: the search direction p = z + beta p, q = A p (carries (p, q)).  Levels from
// block_from on are processed by the first block alone.
#pragma once

#include "fe_solver_common.cuh"

namespace fe {
namespace {

// Chebyshev interval of the smoother and scale of the restriction: digits of residual reduction per inner iteration
// over dam breaks of 32^3 .. 128^3, the 64^3 pool and a 61 x 90 x 47 pool: [0.4, 2] 0.98 / 1.00 / 0.98 at scales
// 0.125 / 0.13 / 0.135, [0.5, 2] 0.94 / 0.97 / 0.95, [0.6, 1.9] 0.92 / 0.95 / 0.93.
constexpr float kChebLow = 0.4f;
constexpr float kRestrictScale = 0.13f;
// Sweep weights 1 / (theta +- delta cos(pi / 4)), theta and delta the centre and half width of [kChebLow, 2].
constexpr float kCos45 = 0.70710678f;
constexpr float kWa = 1.f / (0.5f * (2.f + kChebLow) + 0.5f * (2.f - kChebLow) * kCos45);
constexpr float kWb = 1.f / (0.5f * (2.f + kChebLow) - 0.5f * (2.f - kChebLow) * kCos45);
// Coarsest level: degree-6 Chebyshev on [0.2, 2] (the same digits per iteration as 10 damped Jacobi sweeps or 4
// symmetric Gauss-Seidel sweeps; degree 4 on [0.3, 2] loses a tenth).
constexpr int kCoarseSweeps = 6;
constexpr float kMaskPhi = 0.4f;
// Iterations (and us a solve) at 0 / 4 in 128^3 dam breaks, FLIP after 240 and 300 substeps 10 / 7 (1293 / 963) and 13 / 8 (1812
// / 1198), APIC 12 / 9 (1734 / 1347) and 18 / 9 (2160 / 1187); with a tenth of the cells emptied at random (48^3) 31 / 6;
// the same counts at 120 substeps and before, where no cell holds pockets.  Digits per iteration at 3 are 5 % fewer, at 6
// equal; in all cells instead of those without air beside them it costs the regular surfaces up to one iteration.
constexpr float kInnerAir = 4.f;

// The tile is worked on in a box of 12^3 cells, of which only the cells within two steps of the tile are used: 1376;
// the second sweep covers those within one step: 896 of a box of 10^3.  Both sets are listed in shared memory once per
// solve, so a thread finds its cells with one load instead of divisions (a tile's passes are bound by issue).
constexpr int kBoxW = 12, kBoxCells = kBoxW * kBoxW * kBoxW;
constexpr int kMidW = 10, kMidCells = kMidW * kMidW * kMidW;
constexpr int kBoxList = 512 + 6 * 2 * 64 + 12 * 8, kMidList = 512 + 6 * 64;

// Shared memory of one team.
struct MgTeam {
    float r[kBoxCells];    // right-hand side of the level (0 outside the system)
    float inv[kBoxCells];  // 1 / D (0 outside the system)
    float z[kBoxCells];    // the first sweep's values
    float t[kMidCells];    // the second sweep's values (going up, before that: the 8^3 coarse values around the tile)
    float px[384];         // the residual restricted along x: 6 x 8 x 8
    float py[288];         // ... and y: 6 x 6 x 8
};

constexpr int kTileCache = 192;  // listed tiles of the block, all levels, kept in shared memory
struct MgShared {
    double sh[kShDoubles];
    float inv_lut[128];                // level 0: 1 / D of a cell code (0: not in the system, or left to the loose tiles)
    uint2 box[kBoxList];               // box index | in the tile << 11; cell offset from the tile's first cell (level 0)
    uint2 mid[kMidList];               // box index | 10^3 index << 11; cell offset
    uint16_t boxc[kBoxList], midc[kMidList];  // x | y << 4 | z << 8 in the 12^3 box
    uint32_t ntiles[kMaxMgLevels];     // listed tiles per level
    uint32_t off[kMaxMgLevels];        // first flag / list entry of each level
    uint32_t cache[kTileCache];        // the block's first tiles of each level
    uint32_t cache_at[kMaxMgLevels + 1];
    uint32_t scan[33];
    double p_sum[2];                   // a tank full of fluid: the sum of the starting pressure and the present one's
};

template <int TEAM>
__device__ __forceinline__ void team_sync(int team)
{
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(TEAM) : "memory");
}
// Barrier of the team that returns whether any of its threads passed a non-zero value.
template <int TEAM>
__device__ __forceinline__ bool team_any(int team, bool x)
{
    unsigned out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(out)
        : "r"(x ? 1u : 0u), "r"(team + 1), "n"(TEAM)
        : "memory");
    return out != 0;
}

// ... and how many passed true.
template <int TEAM>
__device__ __forceinline__ int team_count(int team, bool x)
{
    int out;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.popc.u32 %0, %2, %3, p;\n\t}"
                 : "=r"(out)
                 : "r"(x ? 1u : 0u), "r"(team + 1), "n"(TEAM)
                 : "memory");
    return out;
}

__device__ __forceinline__ int tiles_of(int n) { return (n + 7) >> 3; }
// A listed tile: its coordinates, 10 bits each (at most 4096 / 8 tiles per axis).
__device__ __forceinline__ uint32_t pack_tile(int x, int y, int z) { return (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 20); }
struct Tile {
    int x0, y0, z0;  // first cell
};
__device__ __forceinline__ Tile unpack_tile(uint32_t t)
{
    return {(int)(t & 1023u) << 3, (int)((t >> 10) & 1023u) << 3, (int)(t >> 20) << 3};
}

// Tiles of at most kLooseCells cells that touch no fuller tile -- spray; with 0.1 % of the particles in the air they are
// more than half of a dam break's or pool's occupied tiles -- stay out of the V-cycle.  Their cells are few and coupled
// to little else, so a warp takes such a tile with one lane per cell and preconditions it by kLooseSweeps Chebyshev
// sweeps on [0.4, 1.7] over the couplings inside the tile, through shuffles.  (Left to plain Jacobi, or with the partly
// filled tiles of the bulk's surface among them, they cost 2 to 6 more iterations.)
constexpr int kLooseCells = 32;
constexpr int kLooseSweeps = 4;
constexpr uint32_t kLooseBit = 64;  // in a level-0 cell code, above the six neighbour bits
enum : uint8_t { kTileEmpty = 0, kTileFull = 1, kTileFew = 2 };

// The box cells within two steps of the tile and, among them, those within one step, x fastest: x | y << 4 | z << 8.
struct BoxTable {
    uint16_t box[kBoxList];
    uint16_t mid[kMidList];
};
constexpr int box_steps(int x) { return x < 2 ? 2 - x : (x > 9 ? x - 9 : 0); }
constexpr BoxTable make_box_table()
{
    BoxTable t{};
    int nb = 0, nm = 0;
    for (int k = 0; k < kBoxW; ++k)
        for (int j = 0; j < kBoxW; ++j)
            for (int i = 0; i < kBoxW; ++i) {
                const int d = box_steps(i) + box_steps(j) + box_steps(k);
                const uint16_t c = (uint16_t)(i | (j << 4) | (k << 8));
                if (d <= 2) t.box[nb++] = c;
                if (d <= 1) t.mid[nm++] = c;
            }
    return t;
}
__device__ const BoxTable g_box_table = make_box_table();

// The lists in shared memory, with the level-0 cell offsets (whole block; ends without a barrier).
__device__ __forceinline__ void load_box_lists(MgShared& ms, int nx, int sxy)
{
    for (int q = (int)threadIdx.x; q < kBoxList + kMidList; q += (int)blockDim.x) {
        const bool in_mid = q >= kBoxList;
        const uint16_t c = in_mid ? g_box_table.mid[q - kBoxList] : g_box_table.box[q];
        const int i = c & 15, j = (c >> 4) & 15, k = c >> 8;
        const uint32_t b = (uint32_t)(i + kBoxW * (j + kBoxW * k));
        const uint32_t off = (uint32_t)((i - 2) + nx * (j - 2) + sxy * (k - 2));
        if (in_mid) {
            ms.mid[q - kBoxList] = make_uint2(b | ((uint32_t)((i - 1) + kMidW * ((j - 1) + kMidW * (k - 1))) << 11), off);
            ms.midc[q - kBoxList] = c;
        } else {
            ms.box[q] = make_uint2(b | (box_steps(i) + box_steps(j) + box_steps(k) == 0 ? 1u << 11 : 0u), off);
            ms.boxc[q] = c;
        }
    }
}

// Sum of the six neighbours times h^-2 per axis at box index q of a box of width W.
template <int W>
__device__ __forceinline__ float neighbour_sum(const float* a, int q, float hx, float hy, float hz)
{
    return hx * (a[q - 1] + a[q + 1]) + hy * (a[q - W] + a[q + W]) + hz * (a[q - W * W] + a[q + W * W]);
}

// What a pass over a level needs to know of it.
struct LevelArgs {
    int nx, ny, nz;
    float hx, hy, hz;      // 1 / h_l^2 per axis
    const float* inv;      // level >= 1
    float* z2;             // pre-smoothed correction
    float* z;              // result
};

// The second sweep on the tile and one cell around it: s.t = s.z + w (inv (s.r + sum s.z) - s.z).
template <int TEAM>
__device__ __forceinline__ void tile_mid_sweep(MgTeam& s, const MgShared& ms, const LevelArgs& L, float w, int lt)
{
#pragma unroll
    for (int e = 0; e < (kMidList + TEAM - 1) / TEAM; ++e) {
        const int q = lt + e * TEAM;
        if (q < kMidList) {
            const uint32_t m = ms.mid[q].x;
            const int b = (int)(m & 2047u);
            const float z1 = s.z[b];
            s.t[m >> 11] = z1 + w * (s.inv[b] * (s.r[b] + neighbour_sum<kBoxW>(s.z, b, L.hx, L.hy, L.hz)) - z1);
        }
    }
}

// The tile's down pass from s.r, s.inv and s.z = kWa inv r on the box: the second sweep, the residual in the tile, and
// its restriction into the coarse right-hand side C.r.  Stores the pre-smoothed values of the tile.  The next tile may
// be loaded right after it (s.px and s.py are not part of the box).
template <int TEAM>
__device__ __forceinline__ void tile_down(MgTeam& s, const MgShared& ms, const LevelArgs& L, const MgLevel& C,
                                          const Tile& t, int team, int lt)
{
    tile_mid_sweep<TEAM>(s, ms, L, kWb, lt);
    team_sync<TEAM>(team);
#pragma unroll
    for (int it = 0; it < (512 + TEAM - 1) / TEAM; ++it) {
        const int q = lt + it * TEAM;
        if (512 % TEAM != 0 && q >= 512) break;  // whole warps
        const int i = q & 7, j = (q >> 3) & 7, k = q >> 6;
        const int m = (i + 1) + kMidW * ((j + 1) + kMidW * (k + 1));
        const int b = (i + 2) + kBoxW * ((j + 2) + kBoxW * (k + 2));
        const float inv = s.inv[b], z2 = s.t[m];
        float v = 0.f;
        if (inv != 0.f) {
            v = s.r[b] + neighbour_sum<kMidW>(s.t, m, L.hx, L.hy, L.hz) - __fdividef(z2, inv);
            L.z2[(size_t)(t.x0 + i) + (size_t)L.nx * ((size_t)(t.y0 + j) + (size_t)L.ny * (size_t)(t.z0 + k))] = z2;
        }
        // along x: coarse o (parent of fine x0 + 2 (o - 1)) takes 1/4, 3/4, 3/4, 1/4 of fine 2 o - 3 .. 2 o; a row's 8
        // lanes give its 6 sums: even lanes o = i / 2 + 1, lanes 1 and 7 the two ends
        const float l1 = __shfl_up_sync(0xffffffffu, v, 1, 8), r1 = __shfl_down_sync(0xffffffffu, v, 1, 8);
        const float r2 = __shfl_down_sync(0xffffffffu, v, 2, 8);
        float* row = s.px + 6 * (j + 8 * k);
        if ((i & 1) == 0) row[(i >> 1) + 1] = 0.75f * (v + r1) + 0.25f * ((i > 0 ? l1 : 0.f) + (i < 6 ? r2 : 0.f));
        else if (i == 1) row[0] = 0.25f * l1;
        else if (i == 7) row[5] = 0.25f * v;
    }
    team_sync<TEAM>(team);
#pragma unroll
    for (int e = 0; e < (288 + TEAM - 1) / TEAM; ++e) {
        const int o = lt + e * TEAM;
        if (o < 288) {
            const int oi = o % 6, oj = (o / 6) % 6, k = o / 36;
            const float* col = s.px + oi + 48 * k;
            const int f = 2 * oj - 3;
            float sum = 0.f;
            if (f >= 0) sum += 0.25f * col[6 * f];
            if ((unsigned)(f + 1) < 8u) sum += 0.75f * col[6 * (f + 1)];
            if ((unsigned)(f + 2) < 8u) sum += 0.75f * col[6 * (f + 2)];
            if (f + 3 < 8) sum += 0.25f * col[6 * (f + 3)];
            s.py[o] = sum;
        }
    }
    team_sync<TEAM>(team);
    if (lt < 216) {
        const int oi = lt % 6, oj = (lt / 6) % 6, ok = lt / 36;
        const float* col = s.py + oi + 6 * oj;
        const int f = 2 * ok - 3;
        float sum = 0.f;
        if (f >= 0) sum += 0.25f * col[36 * f];
        if ((unsigned)(f + 1) < 8u) sum += 0.75f * col[36 * (f + 1)];
        if ((unsigned)(f + 2) < 8u) sum += 0.75f * col[36 * (f + 2)];
        if (f + 3 < 8) sum += 0.25f * col[36 * (f + 3)];
        if (sum != 0.f) {  // beyond a wall: the parent's own (clamped)
            const int I = min(max((t.x0 >> 1) - 1 + oi, 0), C.nx - 1), J = min(max((t.y0 >> 1) - 1 + oj, 0), C.ny - 1);
            const int K = min(max((t.z0 >> 1) - 1 + ok, 0), C.nz - 1);
            atomicAdd(C.r + ((size_t)I + (size_t)C.nx * ((size_t)J + (size_t)C.ny * (size_t)K)), kRestrictScale * sum);
        }
    }
}

// The 8^3 coarse values around the tile, from two below its first parent on (clamped ones: the parent at a wall), into
// s.t.
template <int TEAM>
__device__ __forceinline__ void tile_load_correction(MgTeam& s, const MgLevel& C, const Tile& t, int lt)
{
#pragma unroll
    for (int it = 0; it < (512 + TEAM - 1) / TEAM; ++it) {
        const int q = lt + it * TEAM;
        if (512 % TEAM != 0 && q >= 512) break;
        const int I = min(max((t.x0 >> 1) - 2 + (q & 7), 0), C.nx - 1);
        const int J = min(max((t.y0 >> 1) - 2 + ((q >> 3) & 7), 0), C.ny - 1);
        const int K = min(max((t.z0 >> 1) - 2 + (q >> 6), 0), C.nz - 1);
        s.t[q] = __ldcg(C.z + ((size_t)I + (size_t)C.nx * ((size_t)J + (size_t)C.ny * (size_t)K)));
    }
}
// Adds the prolonged correction to the box's values of cells in the system (each thread its own cells).
template <int TEAM>
__device__ __forceinline__ void tile_correct(MgTeam& s, const MgShared& ms, int lt)
{
#pragma unroll
    for (int e = 0; e < (kBoxList + TEAM - 1) / TEAM; ++e) {
        const int q = lt + e * TEAM;
        if (q < kBoxList) {
            const uint32_t w = ms.boxc[q];
            const int i = (int)(w & 15u), j = (int)((w >> 4) & 15u), k = (int)(w >> 8);
            const int b = i + kBoxW * (j + kBoxW * k);
            const int pi = (i >> 1) + 1, pj = (j >> 1) + 1, pk = (k >> 1) + 1;
            const float* p = s.t + pi + 8 * (pj + 8 * pk);
            const int di = (i & 1) ? 1 : -1, dj = (j & 1) ? 8 : -8, dk = (k & 1) ? 64 : -64;
            const float y00 = 0.75f * p[0] + 0.25f * p[di], y10 = 0.75f * p[dj] + 0.25f * p[dj + di];
            const float y01 = 0.75f * p[dk] + 0.25f * p[dk + di], y11 = 0.75f * p[dk + dj] + 0.25f * p[dk + dj + di];
            const float zp = 0.75f * (0.75f * y00 + 0.25f * y10) + 0.25f * (0.75f * y01 + 0.25f * y11);
            s.z[b] = s.inv[b] != 0.f ? s.z[b] + zp : 0.f;
        }
    }
}

// The tile's up pass from s.r, s.inv and the corrected s.z on the box: both sweeps; zout(i, j, k, b, value) takes the
// tile's results.  Ends with the team's barrier.
template <int TEAM, class Out>
__device__ __forceinline__ void tile_up(MgTeam& s, const MgShared& ms, const LevelArgs& L, int team, int lt, Out zout)
{
    tile_mid_sweep<TEAM>(s, ms, L, kWa, lt);
    team_sync<TEAM>(team);
#pragma unroll
    for (int it = 0; it < (512 + TEAM - 1) / TEAM; ++it) {
        const int q = lt + it * TEAM;
        if (512 % TEAM != 0 && q >= 512) break;  // whole warps
        const int i = q & 7, j = (q >> 3) & 7, k = q >> 6;
        const int m = (i + 1) + kMidW * ((j + 1) + kMidW * (k + 1));
        const int b = (i + 2) + kBoxW * ((j + 2) + kBoxW * (k + 2));
        const float z1 = s.t[m];
        zout(i, j, k, b, z1 + kWb * (s.inv[b] * (s.r[b] + neighbour_sum<kMidW>(s.t, m, L.hx, L.hy, L.hz)) - z1));
    }
    team_sync<TEAM>(team);  // the next tile overwrites the box
}

// Cell coordinates of box cell w = x | y << 4 | z << 8 of tile t, and whether they lie in the grid.
__device__ __forceinline__ bool box_in_grid(const Tile& t, int nx, int ny, int nz, uint32_t w, int& gi, int& gj, int& gk)
{
    gi = t.x0 - 2 + (int)(w & 15u);
    gj = t.y0 - 2 + (int)((w >> 4) & 15u);
    gk = t.z0 - 2 + (int)(w >> 8);
    return (unsigned)gi < (unsigned)nx && (unsigned)gj < (unsigned)ny && (unsigned)gk < (unsigned)nz;
}
// Level 0: most tiles lie at least two cells from every wall and need no test per cell.
__device__ __forceinline__ bool tile_inside(const Tile& t, int nx, int ny, int nz)
{
    return t.x0 >= 2 && t.y0 >= 2 && t.z0 >= 2 && t.x0 + 10 <= nx && t.y0 + 10 <= ny && t.z0 + 10 <= nz;
}

// Level l >= 1: right-hand side and 1 / D on the box; WITH_Z: also the pre-smoothed values, else the first sweep from
// zero.
template <int TEAM, bool WITH_Z>
__device__ __forceinline__ void tile_load_coarse(MgTeam& s, const MgShared& ms, const LevelArgs& L, const float* r,
                                                 const Tile& t, int lt)
{
#pragma unroll
    for (int e = 0; e < (kBoxList + TEAM - 1) / TEAM; ++e) {
        const int q = lt + e * TEAM;
        if (q < kBoxList) {
            int gi, gj, gk;
            float inv = 0.f, rc = 0.f, z = 0.f;
            if (box_in_grid(t, L.nx, L.ny, L.nz, ms.boxc[q], gi, gj, gk)) {
                const int c = gi + L.nx * (gj + L.ny * gk);
                inv = __ldcg(L.inv + c);
                rc = __ldcg(r + c);
                if (WITH_Z) z = __ldcg(L.z2 + c);
                if (inv == 0.f) rc = 0.f;
                if (!WITH_Z) z = kWa * inv * rc;
            }
            const int b = (int)(ms.box[q].x & 2047u);
            s.r[b] = rc;
            s.inv[b] = inv;
            s.z[b] = z;
        }
    }
}

// Level 0 passes over the block's full tiles; tile(k) is the block's k-th of n.  `team` and `lt`: this thread's team of
// TEAM threads and its place in it; the block's teams take the tiles in turn.
struct FineArgs {
    int nx, ny, nz, sxy;
    const uint8_t* code;
    const float* r;        // pass A: the old residual; pass U: the new one
    float* rn;             // pass A: the new residual
    const float* q;
    const float* p;
    float* pn;
    float* z;
    float* z2;
    float* x;
};

// Pass A: x += alpha p, r' = r - alpha q (FRESH: neither); the sweeps from zero, the residual and its restriction.
// Returns this thread's part of ||r'||^2.
template <int TEAM, bool FRESH, class TileAt>
__device__ __forceinline__ double fine_down(MgTeam* teams, const MgShared& ms, const FineArgs& f, const LevelArgs& A,
                                            const MgLevel& C, float alpha, uint32_t n, TileAt tile)
{
    const int team = (int)threadIdx.x / TEAM, lt = (int)threadIdx.x % TEAM;
    MgTeam& s = teams[team];
    double acc = 0.0;
    for (uint32_t e = (uint32_t)team; e < n; e += blockDim.x / TEAM) {
        const Tile t = tile(e);
        const bool inside = tile_inside(t, f.nx, f.ny, f.nz);
        const int c0 = t.x0 + f.nx * t.y0 + f.sxy * t.z0;
#pragma unroll
        for (int k = 0; k < (kBoxList + TEAM - 1) / TEAM; ++k) {
            const int q = lt + k * TEAM;
            if (q < kBoxList) {
                const uint2 w = ms.box[q];
                const int c = c0 + (int)w.y;
                int gi, gj, gk;
                float inv = 0.f, rc = 0.f;
                if (inside || box_in_grid(t, f.nx, f.ny, f.nz, ms.boxc[q], gi, gj, gk)) {
                    const uint32_t m = __ldcg(f.code + c);
                    rc = __ldcg(f.r + c);
                    if (!FRESH) rc -= alpha * __ldcg(f.q + c);
                    inv = ms.inv_lut[m];
                    if (inv == 0.f) rc = 0.f;
                    else if (w.x >> 11) {
                        if (!FRESH) f.x[c] += alpha * __ldcg(f.p + c);
                        f.rn[c] = rc;
                        acc += (double)rc * (double)rc;
                    }
                }
                const int b = (int)(w.x & 2047u);
                s.r[b] = rc;
                s.inv[b] = inv;
                s.z[b] = kWa * inv * rc;
            }
        }
        team_sync<TEAM>(team);
        tile_down<TEAM>(s, ms, A, C, t, team, lt);
    }
    return acc;
}

// Pass U: the coarse correction and both sweeps.  Returns this thread's part of (r, z).
template <int TEAM, class TileAt>
__device__ __forceinline__ double fine_up(MgTeam* teams, const MgShared& ms, const FineArgs& f, const LevelArgs& A,
                                          const MgLevel& C, uint32_t n, TileAt tile)
{
    const int team = (int)threadIdx.x / TEAM, lt = (int)threadIdx.x % TEAM;
    MgTeam& s = teams[team];
    double acc = 0.0;
    for (uint32_t e = (uint32_t)team; e < n; e += blockDim.x / TEAM) {
        const Tile t = tile(e);
        const bool inside = tile_inside(t, f.nx, f.ny, f.nz);
        const int c0 = t.x0 + f.nx * t.y0 + f.sxy * t.z0;
        tile_load_correction<TEAM>(s, C, t, lt);
#pragma unroll
        for (int k = 0; k < (kBoxList + TEAM - 1) / TEAM; ++k) {
            const int q = lt + k * TEAM;
            if (q < kBoxList) {
                const uint2 w = ms.box[q];
                const int c = c0 + (int)w.y;
                int gi, gj, gk;
                float inv = 0.f, rc = 0.f, z = 0.f;
                if (inside || box_in_grid(t, f.nx, f.ny, f.nz, ms.boxc[q], gi, gj, gk)) {
                    const uint32_t m = __ldcg(f.code + c);
                    rc = __ldcg(f.r + c);
                    z = __ldcg(f.z2 + c);
                    inv = ms.inv_lut[m];
                    if (inv == 0.f) rc = 0.f;
                }
                const int b = (int)(w.x & 2047u);
                s.r[b] = rc;
                s.inv[b] = inv;
                s.z[b] = z;
            }
        }
        team_sync<TEAM>(team);
        tile_correct<TEAM>(s, ms, lt);
        team_sync<TEAM>(team);
        tile_up<TEAM>(s, ms, A, team, lt, [&](int i, int j, int k, int b, float z) {
            if (s.inv[b] != 0.f) {
                f.z[c0 + i + f.nx * j + f.sxy * k] = z;
                acc += (double)s.r[b] * (double)z;
            }
        });
    }
    return acc;
}

// Pass C: p' = z + beta p (FIRST: z), q = A p'.  Returns this thread's part of (p', q).
template <int TEAM, class TileAt>
__device__ __forceinline__ double fine_search(MgTeam* teams, const MgShared& ms, const FineArgs& f, float* qv,
                                              const LevelArgs& A, float beta, bool first, uint32_t n, TileAt tile)
{
    const int team = (int)threadIdx.x / TEAM, lt = (int)threadIdx.x % TEAM;
    MgTeam& s = teams[team];
    uint32_t* s_m = reinterpret_cast<uint32_t*>(s.inv);
    double acc = 0.0;
    for (uint32_t e = (uint32_t)team; e < n; e += blockDim.x / TEAM) {
        const Tile t = tile(e);
        const bool inside = tile_inside(t, f.nx, f.ny, f.nz);
        const int c0 = t.x0 + f.nx * t.y0 + f.sxy * t.z0;
#pragma unroll
        for (int k = 0; k < (kMidList + TEAM - 1) / TEAM; ++k) {
            const int q = lt + k * TEAM;
            if (q < kMidList) {
                const uint2 w = ms.mid[q];
                const int c = c0 + (int)w.y;
                int gi, gj, gk;
                float pv = 0.f;
                uint32_t m = 0;
                if (inside || box_in_grid(t, f.nx, f.ny, f.nz, ms.midc[q], gi, gj, gk)) {
                    m = __ldcg(f.code + c) & 63u;
                    pv = __ldcg(f.z + c);
                    if (!first) pv += beta * __ldcg(f.p + c);
                    if (m == 0u) pv = 0.f;
                }
                s.z[w.x >> 11] = pv;
                s_m[w.x >> 11] = m;
            }
        }
        team_sync<TEAM>(team);
#pragma unroll
        for (int it = 0; it < (512 + TEAM - 1) / TEAM; ++it) {
            const int q = lt + it * TEAM;
            if (512 % TEAM != 0 && q >= 512) break;
            const int i = q & 7, j = (q >> 3) & 7, k = q >> 6;
            const int mq = (i + 1) + kMidW * ((j + 1) + kMidW * (k + 1));
            const uint32_t m = s_m[mq];
            if (m) {
                const float pv = s.z[mq];
                float ax = 0.f, ay = 0.f, az = 0.f;
                if (m & kXm) ax += pv - s.z[mq - 1];
                if (m & kXp) ax += pv - s.z[mq + 1];
                if (m & kYm) ay += pv - s.z[mq - kMidW];
                if (m & kYp) ay += pv - s.z[mq + kMidW];
                if (m & kZm) az += pv - s.z[mq - kMidW * kMidW];
                if (m & kZp) az += pv - s.z[mq + kMidW * kMidW];
                const float qc = A.hx * ax + A.hy * ay + A.hz * az;
                const int c = c0 + i + f.nx * j + f.sxy * k;
                f.pn[c] = pv;
                qv[c] = qc;
                acc += (double)pv * (double)qc;
            }
        }
        team_sync<TEAM>(team);  // the next tile overwrites the box
    }
    return acc;
}

// Levels >= 1, one level down (residual restricted to the next) or up, over the block's n listed tiles.
template <int TEAM, class TileAt>
__device__ __forceinline__ void coarse_down(MgTeam* teams, const MgShared& ms, const LevelArgs& a, const float* r,
                                            const MgLevel& C, uint32_t n, TileAt tile)
{
    const int team = (int)threadIdx.x / TEAM, lt = (int)threadIdx.x % TEAM;
    MgTeam& s = teams[team];
    for (uint32_t e = (uint32_t)team; e < n; e += blockDim.x / TEAM) {
        const Tile t = tile(e);
        tile_load_coarse<TEAM, false>(s, ms, a, r, t, lt);
        team_sync<TEAM>(team);
        tile_down<TEAM>(s, ms, a, C, t, team, lt);
    }
}
template <int TEAM, class TileAt>
__device__ __forceinline__ void coarse_up(MgTeam* teams, const MgShared& ms, const LevelArgs& a, const float* r,
                                          const MgLevel& C, uint32_t n, TileAt tile)
{
    const int team = (int)threadIdx.x / TEAM, lt = (int)threadIdx.x % TEAM;
    MgTeam& s = teams[team];
    for (uint32_t e = (uint32_t)team; e < n; e += blockDim.x / TEAM) {
        const Tile t = tile(e);
        tile_load_correction<TEAM>(s, C, t, lt);
        tile_load_coarse<TEAM, true>(s, ms, a, r, t, lt);
        team_sync<TEAM>(team);
        tile_correct<TEAM>(s, ms, lt);
        team_sync<TEAM>(team);
        tile_up<TEAM>(s, ms, a, team, lt, [&](int i, int j, int k, int b, float z) {
            if (s.inv[b] != 0.f)
                a.z[(size_t)(t.x0 + i) + (size_t)a.nx * ((size_t)(t.y0 + j) + (size_t)a.ny * (size_t)(t.z0 + k))] = z;
        });
    }
}

// ---- levels [LB, L), at most kBlockCellBytes of the block's memory per cell (mg_block_from keeps to what it has): the first
// block takes the whole lower part of the V-cycle with the levels in shared memory, block barriers between the sweeps.  (One
// tile after the other through global memory took 16 us for a 16^3 level and the 8^3 below it at 128^3, spread over the grid
// 13 us with its barriers.)
constexpr int kBlockCellBytes = 17;
struct BlockLevel {
    int nx, ny, nz, n;
    float hx, hy, hz;
    float *r, *inv, *z, *t;
    uint8_t* nb;  // neighbours inside the grid
};
__device__ __forceinline__ float block_sum6(const BlockLevel& B, const float* a, int c)
{
    const uint32_t m = B.nb[c];
    const int sy = B.nx, sz = B.nx * B.ny;
    float x = 0.f, y = 0.f, z = 0.f;
    if (m & 1u) x += a[c - 1];
    if (m & 2u) x += a[c + 1];
    if (m & 4u) y += a[c - sy];
    if (m & 8u) y += a[c + sy];
    if (m & 16u) z += a[c - sz];
    if (m & 32u) z += a[c + sz];
    return B.hx * x + B.hy * y + B.hz * z;
}
// dst = src + w (inv (r + sum src) - src) at every cell
__device__ __forceinline__ void block_sweep(const BlockLevel& B, const float* src, float* dst, float w)
{
    for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x) {
        const float z = src[c];
        dst[c] = z + w * (B.inv[c] * (B.r[c] + block_sum6(B, src, c)) - z);
    }
    __syncthreads();
}
// Fine taps of coarse index I along one axis: 2 I - 1 .. 2 I + 2 with 1/4, 3/4, 3/4, 1/4; a tap beyond the first face, or
// beyond the last one of an even level, is the wall's own cell once more.
__device__ __forceinline__ int tap_index(int I, int k, int nf)
{
    const int f = 2 * I - 1 + k;
    if (f < 0) return 0;
    if (f < nf) return f;
    return f == nf && (nf & 1) == 0 ? nf - 1 : -1;
}
// Level l of the hierarchy in the block's memory, after the levels from LB on before it.
__device__ __forceinline__ BlockLevel block_level(const MgWork& mg, int LB, int l, unsigned char* mem)
{
    for (int k = LB; k < l; ++k) {
        const int n = mg.lv[k].nx * mg.lv[k].ny * mg.lv[k].nz;
        mem += (size_t)((n + 3) & ~3) * kBlockCellBytes;
    }
    const MgLevel& M = mg.lv[l];
    BlockLevel B;
    B.nx = M.nx;
    B.ny = M.ny;
    B.nz = M.nz;
    B.n = M.nx * M.ny * M.nz;
    B.hx = M.ih2[0];
    B.hy = M.ih2[1];
    B.hz = M.ih2[2];
    const int n4 = (B.n + 3) & ~3;
    B.r = reinterpret_cast<float*>(mem);
    B.inv = B.r + n4;
    B.z = B.inv + n4;
    B.t = B.z + n4;
    B.nb = reinterpret_cast<uint8_t*>(B.t + n4);
    return B;
}
__device__ __forceinline__ void block_vcycle(const MgWork& mg, int LB, int L, unsigned char* mem)
{
    for (int l = LB; l < L; ++l) {
        const BlockLevel B = block_level(mg, LB, l, mem);
        const MgLevel& M = mg.lv[l];
        for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x) {
            const int I = c % B.nx, J = (c / B.nx) % B.ny, K = c / (B.nx * B.ny);
            const float inv = __ldcg(M.inv + c);
            B.inv[c] = inv;
            B.nb[c] = (uint8_t)((I > 0 ? 1u : 0u) | (I + 1 < B.nx ? 2u : 0u) | (J > 0 ? 4u : 0u) | (J + 1 < B.ny ? 8u : 0u) |
                                (K > 0 ? 16u : 0u) | (K + 1 < B.nz ? 32u : 0u));
            if (l == LB) {
                const float r = inv != 0.f ? __ldcg(M.r + c) : 0.f;
                B.r[c] = r;
                B.z[c] = kWa * inv * r;
                M.r[c] = 0.f;  // the next cycle restricts into it
            }
        }
    }
    __syncthreads();
    for (int l = LB; l + 1 < L; ++l) {  // down; B.z holds the first sweep
        const BlockLevel B = block_level(mg, LB, l, mem), N = block_level(mg, LB, l + 1, mem);
        block_sweep(B, B.z, B.t, kWb);
        for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x) {
            const float inv = B.inv[c];
            B.z[c] = inv != 0.f ? B.r[c] + block_sum6(B, B.t, c) - __fdividef(B.t[c], inv) : 0.f;  // the residual
        }
        __syncthreads();
        for (int c = (int)threadIdx.x; c < N.n; c += (int)blockDim.x) {
            const int I = c % N.nx, J = (c / N.nx) % N.ny, K = c / (N.nx * N.ny);
            const float inv = N.inv[c];
            float r = 0.f;
            if (inv != 0.f) {
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const int fk = tap_index(K, d, B.nz);
                    if (fk < 0) continue;
                    float plane = 0.f;
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        const int fj = tap_index(J, b, B.ny);
                        if (fj < 0) continue;
                        float row = 0.f;
#pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            const int fi = tap_index(I, a, B.nx);
                            if (fi >= 0) row += (a == 0 || a == 3 ? 0.25f : 0.75f) * B.z[fi + B.nx * (fj + B.ny * fk)];
                        }
                        plane += (b == 0 || b == 3 ? 0.25f : 0.75f) * row;
                    }
                    r += (d == 0 || d == 3 ? 0.25f : 0.75f) * plane;
                }
                r *= kRestrictScale;
            }
            N.r[c] = r;
            N.z[c] = kWa * inv * r;
        }
        __syncthreads();
    }
    {  // the coarsest level: Chebyshev sweeps from zero
        const BlockLevel B = block_level(mg, LB, L - 1, mem);
        // 1 / (theta + delta cos((2 k + 1) pi / 12)) on [0.2, 2]
        constexpr float kCosine[kCoarseSweeps] = {0.96592583f, 0.70710678f, 0.25881905f, -0.25881905f, -0.70710678f, -0.96592583f};
        for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x)
            B.t[c] = (1.f / (1.1f + 0.9f * kCosine[0])) * (B.inv[c] * B.r[c]);
        __syncthreads();
        static_assert(kCoarseSweeps % 2 == 0, "the last sweep leaves the result in z");
#pragma unroll
        for (int k = 1; k < kCoarseSweeps; ++k)
            block_sweep(B, k & 1 ? B.t : B.z, k & 1 ? B.z : B.t, 1.f / (1.1f + 0.9f * kCosine[k]));
    }
    for (int l = L - 2; l >= LB; --l) {  // up; B.t holds the pre-smoothed correction
        const BlockLevel B = block_level(mg, LB, l, mem), N = block_level(mg, LB, l + 1, mem);
        for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x) {
            float z = 0.f;
            if (B.inv[c] != 0.f) {
                const int g[3] = {c % B.nx, (c / B.nx) % B.ny, c / (B.nx * B.ny)};
                const int nn[3] = {N.nx, N.ny, N.nz};
                int p[3], n[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    p[a] = g[a] >> 1;
                    n[a] = min(max((g[a] & 1) ? p[a] + 1 : p[a] - 1, 0), nn[a] - 1);
                }
                auto at = [&](int i, int j, int k) { return N.z[i + N.nx * (j + N.ny * k)]; };
                const float y00 = 0.75f * at(p[0], p[1], p[2]) + 0.25f * at(n[0], p[1], p[2]);
                const float y10 = 0.75f * at(p[0], n[1], p[2]) + 0.25f * at(n[0], n[1], p[2]);
                const float y01 = 0.75f * at(p[0], p[1], n[2]) + 0.25f * at(n[0], p[1], n[2]);
                const float y11 = 0.75f * at(p[0], n[1], n[2]) + 0.25f * at(n[0], n[1], n[2]);
                z = B.t[c] + 0.75f * (0.75f * y00 + 0.25f * y10) + 0.25f * (0.75f * y01 + 0.25f * y11);
            }
            B.z[c] = z;
        }
        __syncthreads();
        block_sweep(B, B.z, B.t, kWa);
        block_sweep(B, B.t, B.z, kWb);
    }
    const BlockLevel B = block_level(mg, LB, LB, mem);
    for (int c = (int)threadIdx.x; c < B.n; c += (int)blockDim.x) mg.lv[LB].z[c] = B.z[c];
    __syncthreads();
}

// The solver body, run by `nblk` blocks of which this is block `blk`; every barrier and reduction spans
// those blocks.  Vectors: r (ping-pong r0/r1), z (w0), q = A p (w1), p (ping-pong s0/s1), the pre-smoothed level-0
// correction (pv), x (the inner solve's correction); the cell codes and the tiles' flags lie in xcg, the tile lists in
// list.  Entries of cells outside the system are never read for their value, so nothing has to be cleared for cells
// that leave it.  Tiles with rank r in their level's list belong to block r % nblk, whose teams take them in turn: teams
// of MANY threads where there are more than two tiles per block (more tiles in flight hide more of the loads' latency:
// 11.0 against 14.0 us for pass U at 128^3), of FEW threads where not (each tile is through sooner: 3.1 against 4.4 us).
// teams: shared memory of blockDim.x / MANY teams, then 96 words per warp.
template <int FEW, int MANY>
__device__ __forceinline__ void mg_body(MgShared& ms, MgTeam* __restrict__ teams, const SceneView& v, const CgWork& w,
                                        const MgWork& mg, const CgParams& prm, const int blk, const int nblk,
                                        int* out_its = nullptr, int* out_fluid = nullptr)
{
    double* sh = ms.sh;
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const size_t sxy = (size_t)nx * ny;
    const size_t nc = sxy * nz;
    const int nteam = (int)blockDim.x / MANY;
    const int team = (int)threadIdx.x / MANY, lt = (int)threadIdx.x % MANY;
    const int wid = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31;
    const uint32_t G = (uint32_t)(nblk * nteam), gteam = (uint32_t)(team * nblk + blk);
    const uint32_t GW = (uint32_t)(nblk * (int)(blockDim.x >> 5)), gwarp = (uint32_t)(wid * nblk + blk);
    MgTeam& s = teams[team];
    uint32_t* const own_loose = reinterpret_cast<uint32_t*>(teams + nteam) + 96 * wid;  // the warp's first loose tile
    const double ih2d[3] = {v.inv_h[0] * v.inv_h[0], v.inv_h[1] * v.inv_h[1], v.inv_h[2] * v.inv_h[2]};
    const float ih2[3] = {(float)ih2d[0], (float)ih2d[1], (float)ih2d[2]};
    double* p64 = v.p;
    const double* __restrict__ b = v.b;
    float* Z = w.w0;
    float* Q = w.w1;
    float* X = w.x;
    uint8_t* code = reinterpret_cast<uint8_t*>(w.xcg);
    uint8_t* flags = code + nc;  // one byte per tile, level after level
    uint32_t* list = w.list;     // listed tiles, level after level
    const int L = mg.levels;
    const int LB = mg.block_from;  // first level of the first block's share (mg_block_from: its memory holds them)
    unsigned gen = 0;
    const bool solids = prm.gate != nullptr;  // a scene with colliders: there may be BOUNDRY cells

    if (threadIdx.x < 128) {
        const int m = (int)threadIdx.x;
        const float d = ih2[0] * (float)__popc(m & 3) + ih2[1] * (float)__popc(m & 12) + ih2[2] * (float)__popc(m & 48);
        ms.inv_lut[m] = m && !(m & kLooseBit) ? 1.f / d : 0.f;
    }
    load_box_lists(ms, nx, (int)sxy);
    if (threadIdx.x == 0) {
        uint32_t o = 0;
        for (int l = 0; l < L; ++l) {
            ms.off[l] = o;
            o += (uint32_t)(tiles_of(mg.lv[l].nx) * tiles_of(mg.lv[l].ny) * tiles_of(mg.lv[l].nz));
        }
    }
    __syncthreads();
    const int tn[3] = {tiles_of(nx), tiles_of(ny), tiles_of(nz)};
    const uint32_t nt0 = (uint32_t)(tn[0] * tn[1] * tn[2]);
    const uint32_t nflags =
        ms.off[L - 1] + (uint32_t)(tiles_of(mg.lv[L - 1].nx) * tiles_of(mg.lv[L - 1].ny) * tiles_of(mg.lv[L - 1].nz));
    uint8_t* kind0 = flags + nflags;                  // the level-0 tiles' kinds
    uint32_t* loose = list + nflags;                  // 96 words per loose tile
    uint32_t* cell_bits = loose + 96 * (size_t)nt0;   // 16 words per tile: its cells in the system
    // loose tiles pay where the blocks would otherwise take several rounds of tiles (32^3: 238 us a solve without, 299
    // with; 128^3: 980 without, 805 with); grids a cell or two thin have no room for their lists
    const bool use_loose = nt0 > 2u * (uint32_t)nblk && (size_t)nflags + 112 * (size_t)nt0 <= nc;
    // ---- setup 1: cell codes, ||b||^2 and the cells of the system; fluid fractions of levels 1 .. 3 of each tile
    // (into the levels' t arrays); cells outside the system get pressure 0
    double acc2[2] = {0.0, 0.0};
    for (uint32_t ti = gteam; ti < nt0; ti += G) {
        const int tx = (int)(ti % tn[0]), ty = (int)((ti / tn[0]) % tn[1]), tz = (int)(ti / (tn[0] * tn[1]));
        int cells = 0;
#pragma unroll
        for (int it = 0; it < 512 / MANY; ++it) {
            const int q = lt + it * MANY;
            const int i = tx * 8 + (q & 7), j = ty * 8 + ((q >> 3) & 7), k = tz * 8 + (q >> 6);
            float phi = -1.f;  // outside the grid, or no part of the system as a wall is none
            if (i < nx && j < ny && k < nz) {
                const size_t c = (size_t)i + (size_t)nx * j + sxy * k;
                const uint32_t m = solve_mask(v.marks, (int)c, i, j, k, nx, ny, nz);
                code[c] = (uint8_t)m;
                phi = m ? 1.f : (solids && v.marks[c] != FE_CELL_AIR ? -1.f : 0.f);
                if (m) {
                    acc2[0] += b[c] * b[c];
                    acc2[1] += 1.0;
                } else {
                    p64[c] = 0.0;
                }
            }
            s.r[q] = phi;
            const unsigned bits = __ballot_sync(0xffffffffu, phi > 0.f);
            if (lane == 0 && use_loose) cell_bits[16 * (size_t)ti + (q >> 5)] = bits;
            cells += team_count<MANY>(team, phi > 0.f);
        }
        if (lt == 0) flags[ti] = cells == 0 ? kTileEmpty : (cells <= kLooseCells && use_loose ? kTileFew : kTileFull);
        // means over the children inside the grid, level after level
        const float* src = s.r;
        float* dst = s.z;
        for (int l = 1, e = 4; l <= 3 && l < L; ++l, e >>= 1) {
            if (lt < e * e * e) {
                const int i = lt % e, j = (lt / e) % e, k = lt / (e * e);
                float sum = 0.f, cnt = 0.f;
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                    const float x = src[(2 * i + (d & 1)) + 2 * e * ((2 * j + ((d >> 1) & 1)) + 2 * e * (2 * k + (d >> 2)))];
                    if (x >= 0.f) {
                        sum += x;
                        cnt += 1.f;
                    }
                }
                const float phi = cnt > 0.f ? sum / cnt : -1.f;
                dst[lt] = phi;
                const MgLevel& C = mg.lv[l];
                const int I = tx * e + i, J = ty * e + j, K = tz * e + k;
                if (I < C.nx && J < C.ny && K < C.nz) C.t[(size_t)I + (size_t)C.nx * ((size_t)J + (size_t)C.ny * K)] = phi;
            }
            src = dst;
            dst += 64;
            team_sync<MANY>(team);
        }
    }
    if (!grid_reduce<2>(acc2, sh, w, gen, nblk, blk)) return;
    const double bnorm = sqrt(acc2[0]);
    const int F = (int)acc2[1];

    // ---- setup 2: 1 / D of a coarse level from its fractions and its children's, and its tiles' flags
    auto level_inv = [&](int l, uint32_t g0, uint32_t stride) {
        const MgLevel& C = mg.lv[l];
        const MgLevel& Fl = mg.lv[l - 1];
        const int cn[3] = {C.nx, C.ny, C.nz};
        const int ct[3] = {tiles_of(C.nx), tiles_of(C.ny), tiles_of(C.nz)};
        const float half_h0 = 0.5f / (float)(1 << l);
        const size_t st[3] = {1, (size_t)C.nx, (size_t)C.nx * C.ny};
        for (uint32_t ti = g0; ti < (uint32_t)(ct[0] * ct[1] * ct[2]); ti += stride) {
            const int t0[3] = {8 * (int)(ti % ct[0]), 8 * (int)((ti / ct[0]) % ct[1]), 8 * (int)(ti / (ct[0] * ct[1]))};
            bool any = false;
#pragma unroll
            for (int it = 0; it < 512 / MANY; ++it) {
                const int q = lt + it * MANY;
                const int g[3] = {t0[0] + (q & 7), t0[1] + ((q >> 3) & 7), t0[2] + (q >> 6)};
                if (g[0] >= cn[0] || g[1] >= cn[1] || g[2] >= cn[2]) continue;
                const size_t c = g[0] * st[0] + g[1] * st[1] + g[2] * st[2];
                const float own = __ldcg(C.t + c);
                float inv = 0.f;
                if (own > kMaskPhi) {
                    any = true;
                    float child[8];
#pragma unroll
                    for (int d = 0; d < 8; ++d) {
                        const int i = 2 * g[0] + (d & 1), j = 2 * g[1] + ((d >> 1) & 1), k = 2 * g[2] + (d >> 2);
                        child[d] = -1.f;
                        if (i < Fl.nx && j < Fl.ny && k < Fl.nz) {
                            const size_t f = (size_t)i + (size_t)Fl.nx * ((size_t)j + (size_t)Fl.ny * (size_t)k);
                            child[d] = l > 1 ? __ldcg(Fl.t + f) : (__ldcg(code + f) ? 1.f : (solids && v.marks[f] != FE_CELL_AIR ? -1.f : 0.f));
                        }
                    }
                    float diag = 0.f;
                    bool inner = true;  // no neighbour is air
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            const int n = g[a] + (side ? 1 : -1);
                            if (n < 0 || n >= cn[a]) continue;  // wall: no flux
                            const float phi = __ldcg(C.t + (side ? c + st[a] : c - st[a]));
                            if (phi < 0.f) continue;  // nothing but BOUNDRY: a wall
                            float coef = 1.f;
                            if (!(phi > kMaskPhi)) {
                                inner = false;
                                float sum = 0.f, cnt = 0.f;
#pragma unroll
                                for (int d = 0; d < 8; ++d)
                                    if (((d >> a) & 1) == side && child[d] >= 0.f) {
                                        sum += child[d];
                                        cnt += 1.f;
                                    }
                                const float dist = 0.5f * (cnt > 0.f ? sum / cnt : 0.f) + phi + half_h0;
                                coef = 1.f / fminf(fmaxf(dist, 0.25f), 1.5f);
                            }
                            diag += C.ih2[a] * coef;
                        }
                    if (inner && own < 1.f) diag += kInnerAir * (C.ih2[0] + C.ih2[1] + C.ih2[2]) * sqrtf(1.f - own);
                    inv = diag > 0.f ? 1.f / diag : 0.f;
                }
                C.inv[c] = inv;
                C.r[c] = 0.f;
                if (inv == 0.f) C.z[c] = 0.f;  // read by the finer level's correction
            }
            any = team_any<MANY>(team, any);
            if (lt == 0) flags[ms.off[l] + ti] = any ? 1 : 0;
        }
    };
    // fractions of level l >= 4 from level l - 1 (first block)
    auto level_phi = [&](int l) {
        const MgLevel& C = mg.lv[l];
        const MgLevel& Fl = mg.lv[l - 1];
        const int n = C.nx * C.ny * C.nz;
        for (int t = (int)threadIdx.x; t < n; t += (int)blockDim.x) {
            const int I = t % C.nx, J = (t / C.nx) % C.ny, K = t / (C.nx * C.ny);
            float sum = 0.f, cnt = 0.f;
            for (int d = 0; d < 8; ++d) {
                const int i = 2 * I + (d & 1), j = 2 * J + ((d >> 1) & 1), k = 2 * K + (d >> 2);
                if (i >= Fl.nx || j >= Fl.ny || k >= Fl.nz) continue;
                const float x = __ldcg(Fl.t + ((size_t)i + (size_t)Fl.nx * ((size_t)j + (size_t)Fl.ny * (size_t)k)));
                if (x >= 0.f) {
                    sum += x;
                    cnt += 1.f;
                }
            }
            C.t[t] = cnt > 0.f ? sum / cnt : -1.f;
        }
        __threadfence();
        __syncthreads();
    };
    // ---- setup 2 also settles the tiles of few cells: loose, unless a cell of theirs touches one of a full tile; a
    // loose tile's cells leave the V-cycle (kLooseBit).  In a tile of few cells lane s < 16 holds the bits of cells 32 s
    // .. 32 s + 31, `before` counts the cells of earlier lanes, and lane n takes the n-th cell (-1: none).
    auto few_cells = [&](uint32_t ti, unsigned& bits, int& before) -> int {
        bits = lane < 16 ? __ldcg(cell_bits + 16 * (size_t)ti + lane) : 0u;
        before = __popc(bits);
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += x;
        }
        const int count = __shfl_sync(0xffffffffu, before, 15);
        before -= __popc(bits);
        int* cells = reinterpret_cast<int*>(own_loose);
        __syncwarp();
        int at = before;
        for (unsigned rest = bits; rest; rest &= rest - 1u) cells[at++] = 32 * lane + (__ffs((int)rest) - 1);
        __syncwarp();
        return lane < count ? cells[lane] : -1;
    };
    for (uint32_t ti = gwarp; ti < nt0; ti += GW) {
        const uint8_t f = __ldcg(flags + ti);
        uint8_t kind = f;
        if (f == kTileFew) {
            unsigned bits;
            int before;
            const int q = few_cells(ti, bits, before);
            const int tx = (int)(ti % tn[0]), ty = (int)((ti / tn[0]) % tn[1]), tz = (int)(ti / (tn[0] * tn[1]));
            bool touches = false;
            size_t c = 0;
            if (q >= 0) {
                const int i = q & 7, j = (q >> 3) & 7, k = q >> 6;
                c = (size_t)(tx * 8 + i) + (size_t)nx * (ty * 8 + j) + sxy * (tz * 8 + k);
                const uint32_t m = __ldcg(code + c);
                auto full = [&](size_t cn, uint32_t t) { return (__ldcg(code + cn) & 63u) && __ldcg(flags + t) == kTileFull; };
                if (i == 0 && (m & kXm)) touches |= full(c - 1, ti - 1);
                if (i == 7 && (m & kXp)) touches |= full(c + 1, ti + 1);
                if (j == 0 && (m & kYm)) touches |= full(c - nx, ti - tn[0]);
                if (j == 7 && (m & kYp)) touches |= full(c + nx, ti + tn[0]);
                if (k == 0 && (m & kZm)) touches |= full(c - sxy, ti - tn[0] * tn[1]);
                if (k == 7 && (m & kZp)) touches |= full(c + sxy, ti + tn[0] * tn[1]);
            }
            if (__any_sync(0xffffffffu, touches)) kind = kTileFull;
            else if (q >= 0) code[c] = (uint8_t)(__ldcg(code + c) | kLooseBit);
        }
        if (lane == 0) kind0[ti] = kind;
    }
    for (int l = 1; l < L && l <= 3; ++l) level_inv(l, gteam, G);
    if (blk == 0)
        for (int l = 4; l < L; ++l) {
            __syncthreads();
            level_phi(l);
            level_inv(l, (uint32_t)team, (uint32_t)nteam);
        }
    if (!grid_sync(w, gen, nblk, sh, blk)) return;

    // ---- tile lists.  Tiles with flag `kind` among flag[0 .. nt): every block ranks all of them and keeps those of its
    // rank r % step % nblk; entry(rank, tile) stores one.  Returns how many there are.
    auto build_list = [&](const uint8_t* flag, uint8_t kind, uint32_t nt, uint32_t step, auto entry) -> uint32_t {
        uint32_t base = 0;
        for (uint32_t c0 = 0; c0 < nt; c0 += 4 * blockDim.x) {
            const uint32_t ti = c0 + 4 * threadIdx.x;
            unsigned on = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (ti + k < nt && __ldcg(flag + ti + k) == kind) on |= 1u << k;
            uint32_t before = (uint32_t)__popc(on);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before += x;
            }
            if (lane == 31) ms.scan[wid] = before;
            before -= (uint32_t)__popc(on);
            __syncthreads();
            uint32_t total = 0;
            for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
                const uint32_t x = ms.scan[k];
                before += k < wid ? x : 0u;
                total += x;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if ((on >> k) & 1u) {
                    const uint32_t rank = base + before++;
                    if ((int)((rank % step) % (uint32_t)nblk) == blk) entry(rank, ti + k);
                }
            base += total;
            __syncthreads();
        }
        return base;
    };
    {
        uint32_t at = 0;
        for (int l = 0; l < LB; ++l) {
            const uint32_t o = ms.off[l];
            const int tnx = tiles_of(mg.lv[l].nx), tny = tiles_of(mg.lv[l].ny);
            const uint32_t n = build_list(l == 0 ? kind0 : flags + o, kTileFull, (uint32_t)(tnx * tny * tiles_of(mg.lv[l].nz)),
                                          (uint32_t)nblk, [&](uint32_t rank, uint32_t ti) {
                                              const uint32_t t = pack_tile((int)(ti % tnx), (int)((ti / tnx) % tny), (int)(ti / (tnx * tny)));
                                              const uint32_t k = at + rank / (uint32_t)nblk;
                                              list[o + rank] = t;
                                              if (k < kTileCache) ms.cache[k] = t;
                                          });
            if (threadIdx.x == 0) {
                ms.ntiles[l] = n > (uint32_t)blk ? (n - (uint32_t)blk - 1u) / (uint32_t)nblk + 1u : 0u;  // the block's
                ms.cache_at[l] = at;
                if (l == 0) ms.cache_at[kMaxMgLevels] = n;
            }
            at = min(at + (n > (uint32_t)blk ? (n - (uint32_t)blk - 1u) / (uint32_t)nblk + 1u : 0u), (uint32_t)kTileCache);
        }
    }
    // loose tiles: three words per lane: the cell (~0: none); the lanes of its six neighbours in the tile, 5 bits each;
    // which of those exist | its neighbour mask << 6
    const uint32_t nloose = build_list(kind0, kTileFew, nt0, GW, [&](uint32_t rank, uint32_t ti) { loose[96 * (size_t)rank] = ti; });
    __syncthreads();
    for (uint32_t e = gwarp; e < nloose; e += GW) {
        const uint32_t ti = loose[96 * (size_t)e];
        unsigned bits;
        int before;
        const int cell = few_cells(ti, bits, before);
        const int tx = (int)(ti % tn[0]), ty = (int)((ti / tn[0]) % tn[1]), tz = (int)(ti / (tn[0] * tn[1]));
        uint32_t lanes = 0, exist = 0, m = 0, c = ~0u;
        const int q = cell & 511;
        if (cell >= 0) {
            c = (uint32_t)((size_t)(tx * 8 + (q & 7)) + (size_t)nx * (ty * 8 + ((q >> 3) & 7)) + sxy * (tz * 8 + (q >> 6)));
            m = __ldcg(code + c) & 63u;
        }
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            const int a = d >> 1, nco = ((q >> (3 * a)) & 7) + ((d & 1) ? 1 : -1);
            const bool in = cell >= 0 && (unsigned)nco < 8u;
            const int nq = in ? q + ((d & 1) ? 1 : -1) * (1 << (3 * a)) : 0;
            const unsigned nb = __shfl_sync(0xffffffffu, bits, nq >> 5);
            const int n0 = __shfl_sync(0xffffffffu, before, nq >> 5);
            if (in && ((nb >> (nq & 31)) & 1u)) {
                lanes |= (uint32_t)(n0 + __popc(nb & ((1u << (nq & 31)) - 1u))) << (5 * d);
                exist |= 1u << d;
            }
        }
        __syncwarp();  // every lane has the tile
        loose[96 * (size_t)e + lane] = c;
        loose[96 * (size_t)e + 32 + lane] = lanes;
        loose[96 * (size_t)e + 64 + lane] = exist | (m << 6);
    }
    __syncwarp();
    if (gwarp < nloose)
        for (int k = lane; k < 96; k += 32) own_loose[k] = loose[96 * (size_t)gwarp + k];
    __syncthreads();
    auto loose_rec = [&](uint32_t e) -> const uint32_t* { return e == gwarp ? own_loose : loose + 96 * (size_t)e; };
    const uint32_t n_fine = ms.ntiles[0];                                          // this block's full tiles
    const bool many = FEW == MANY || ms.cache_at[kMaxMgLevels] > 2u * (uint32_t)nblk;
    // the block's k-th tile of level l
    auto tiles = [&](int l) {
        const uint32_t at = ms.cache_at[l], room = (uint32_t)kTileCache - at;
        const uint32_t* rest = list + ms.off[l] + blk;
        return [&ms, at, room, rest, nblk](uint32_t k) { return unpack_tile(k < room ? ms.cache[at + k] : rest[(size_t)k * nblk]); };
    };
    const auto fine_tile = tiles(0);

    // right-hand side of level l back to zero (its cells of the system: the others are never read)
    auto zero_level = [&](int l) {
        const MgLevel& C = mg.lv[l];
        const auto tile = tiles(l);
        const uint32_t n = ms.ntiles[l];
        for (uint32_t e = (uint32_t)team; e < n; e += (uint32_t)nteam) {
            const Tile t = tile(e);
#pragma unroll
            for (int it = 0; it < 512 / MANY; ++it) {
                const int q = lt + it * MANY;
                const int i = t.x0 + (q & 7), j = t.y0 + ((q >> 3) & 7), k = t.z0 + (q >> 6);
                if (i < C.nx && j < C.ny && k < C.nz)
                    C.r[(size_t)i + (size_t)C.nx * ((size_t)j + (size_t)C.ny * (size_t)k)] = 0.f;
            }
        }
    };
    // calls f(c, m) for this thread's cells of the system
    auto for_cells = [&](auto f) {
        for (uint32_t e = (uint32_t)team; e < n_fine; e += (uint32_t)nteam) {
            const Tile t = fine_tile(e);
#pragma unroll
            for (int it = 0; it < 512 / MANY; ++it) {
                const int q = lt + it * MANY;
                const int i = t.x0 + (q & 7), j = t.y0 + ((q >> 3) & 7), k = t.z0 + (q >> 6);
                if (i >= nx || j >= ny || k >= nz) continue;
                const size_t c = (size_t)i + (size_t)nx * j + sxy * k;
                const uint32_t m = __ldcg(code + c);
                if (m) f(c, m);
            }
        }
        for (uint32_t e = gwarp; e < nloose; e += GW) {
            const uint32_t* rec = loose_rec(e);
            const uint32_t c = rec[lane];
            if (c != ~0u) f((size_t)c, rec[64 + lane] >> 6);
        }
    };

    auto level_args = [&](int l) {
        const MgLevel& M = mg.lv[l];
        LevelArgs a;
        a.nx = M.nx;
        a.ny = M.ny;
        a.nz = M.nz;
        a.hx = M.ih2[0];
        a.hy = M.ih2[1];
        a.hz = M.ih2[2];
        a.inv = M.inv;
        a.z2 = l == 0 ? w.pv : M.t;
        a.z = l == 0 ? Z : M.z;
        return a;
    };
    const LevelArgs A0 = level_args(0);
    FineArgs fa;
    fa.nx = nx;
    fa.ny = ny;
    fa.nz = nz;
    fa.sxy = (int)sxy;
    fa.code = code;
    fa.q = Q;
    fa.z = Z;
    fa.z2 = w.pv;
    fa.x = X;

    const double target = prm.rel_tol * bnorm;
    if (bnorm == 0.0) for_cells([&](size_t c, uint32_t) { p64[c] = 0.0; });
    int total_it = 0, refinements = 0;
    double rnorm = 0.0, rho_old = 1.0;
    bool converged = bnorm == 0.0;
    bool first = true;
    int pc = 0;  // ping-pong index of p
    while (!converged) {
        // ---- outer residual r = b - A p in FP64, stored in FP32; the inner solve's correction starts at zero
        double racc[1] = {0.0};
        for_cells([&](size_t c, uint32_t m) {
            const double pc0 = __ldcg(p64 + c);
            double ax = 0.0, ay = 0.0, az = 0.0;
            if (m & kXm) ax += pc0 - __ldcg(p64 + c - 1);
            if (m & kXp) ax += pc0 - __ldcg(p64 + c + 1);
            if (m & kYm) ay += pc0 - __ldcg(p64 + c - nx);
            if (m & kYp) ay += pc0 - __ldcg(p64 + c + nx);
            if (m & kZm) az += pc0 - __ldcg(p64 + c - sxy);
            if (m & kZp) az += pc0 - __ldcg(p64 + c + sxy);
            const double rr = b[c] - (ih2d[0] * ax + ih2d[1] * ay + ih2d[2] * az);
            w.r0[c] = (float)rr;
            X[c] = 0.f;
            racc[0] += rr * rr;
        });
        // the last pass A of the inner solve before restricted into level 1
        if (LB > 1) zero_level(1);
        else if (blk == 0)
            for (int c = (int)threadIdx.x; c < mg.lv[1].nx * mg.lv[1].ny * mg.lv[1].nz; c += (int)blockDim.x) mg.lv[1].r[c] = 0.f;
        if (!grid_reduce<1>(racc, sh, w, gen, nblk, blk)) return;
        rnorm = sqrt(racc[0]);
        if ((size_t)F == nc) {  // the sum of p, at first and now
            racc[0] = 0.0;
            for_cells([&](size_t c, uint32_t) { racc[0] += __ldcg(p64 + c); });
            if (!grid_reduce<1>(racc, sh, w, gen, nblk, blk)) return;
            if (threadIdx.x == 0) ms.p_sum[refinements > 0] = racc[0];
        }
        if (rnorm <= target) {
            converged = true;
            break;
        }
        if (refinements >= prm.max_refine || total_it >= prm.max_it) break;
        ++refinements;

        // ---- inner MG-preconditioned CG on A e = r.  A refinement replaces the residual by the FP64 one and keeps the
        // search direction: the residual only changes by the FP32 rounding, and starting over would cost an iteration.
        const double want = fmax(prm.inner_tol, 0.25 * target / rnorm);
        double stop = 0.0;
        float alpha = 0.f;
        int cur = 0;  // ping-pong index of r
        bool fresh = true;
        while (true) {
            // pass A: x += alpha p, r' = r - alpha q; level 0's sweeps from zero, residual and restriction
            {
                fa.r = cur ? w.r1 : w.r0;
                fa.rn = cur ? w.r0 : w.r1;
                fa.p = pc ? w.s1 : w.s0;
                double acc[1] = {0.0};
                for (uint32_t e = gwarp; e < nloose; e += GW) {
                    const uint32_t c = loose_rec(e)[lane];
                    if (c == ~0u) continue;
                    float rc = __ldcg(fa.r + c);
                    if (!fresh) {
                        rc -= alpha * __ldcg(Q + c);
                        X[c] += alpha * __ldcg(fa.p + c);
                    }
                    fa.rn[c] = rc;
                    acc[0] += (double)rc * (double)rc;
                }
                if (fresh) acc[0] += fine_down<MANY, true>(teams, ms, fa, A0, mg.lv[1], alpha, n_fine, fine_tile);
                else if (many) acc[0] += fine_down<MANY, false>(teams, ms, fa, A0, mg.lv[1], alpha, n_fine, fine_tile);
                else acc[0] += fine_down<FEW, false>(teams, ms, fa, A0, mg.lv[1], alpha, n_fine, fine_tile);
                if (!grid_reduce<1>(acc, sh, w, gen, nblk, blk)) return;
                cur ^= 1;
                if (fresh) stop = want * want * acc[0];
                else ++total_it;
                fresh = false;
                if (acc[0] <= stop || !(acc[0] == acc[0]) || total_it >= prm.max_it) break;
            }
            for (int l = 1; l < LB; ++l) {
                const LevelArgs a = level_args(l);
                coarse_down<FEW>(teams, ms, a, mg.lv[l].r, mg.lv[l + 1], ms.ntiles[l], tiles(l));
                if (!grid_sync(w, gen, nblk, sh, blk)) return;
            }
            if (blk == 0) block_vcycle(mg, LB, L, reinterpret_cast<unsigned char*>(teams));
            if (!grid_sync(w, gen, nblk, sh, blk)) return;
            for (int l = LB - 1; l >= 1; --l) {
                const LevelArgs a = level_args(l);
                if (l + 1 < LB) zero_level(l + 1);
                coarse_up<FEW>(teams, ms, a, mg.lv[l].r, mg.lv[l + 1], ms.ntiles[l], tiles(l));
                if (!grid_sync(w, gen, nblk, sh, blk)) return;
            }
            // level 0: correction and sweeps, (r, z)
            double rho;
            {
                fa.r = cur ? w.r1 : w.r0;
                double acc[1] = {0.0};
                for (uint32_t e = gwarp; e < nloose; e += GW) {
                    const uint32_t* rec = loose_rec(e);
                    const uint32_t c = rec[lane], lanes = rec[32 + lane], em = rec[64 + lane];
                    const float rc = c != ~0u ? __ldcg(fa.r + c) : 0.f;
                    const uint32_t m = em >> 6;
                    const float d = ih2[0] * (float)__popc(m & 3u) + ih2[1] * (float)__popc(m & 12u) + ih2[2] * (float)__popc(m & 48u);
                    const float inv = m ? __fdividef(1.f, d) : 0.f;
                    float z = 0.f;
#pragma unroll
                    for (int sw = 0; sw < kLooseSweeps; ++sw) {
                        constexpr float kCosine[kLooseSweeps] = {0.92387953f, 0.38268343f, -0.38268343f, -0.92387953f};
                        const float omega = 1.f / (1.05f + 0.65f * kCosine[sw]);
                        float sum = rc;
                        if (sw > 0) {
#pragma unroll
                            for (int k = 0; k < 6; ++k) {
                                const float zn = __shfl_sync(0xffffffffu, z, (int)((lanes >> (5 * k)) & 31u));
                                if ((em >> k) & 1u) sum += ih2[k >> 1] * zn;
                            }
                        }
                        z += omega * (inv * sum - z);
                    }
                    if (c != ~0u) {
                        Z[c] = z;
                        acc[0] += (double)rc * (double)z;
                    }
                }
                if (LB > 1) zero_level(1);
                if (many) acc[0] += fine_up<MANY>(teams, ms, fa, A0, mg.lv[1], n_fine, fine_tile);
                else acc[0] += fine_up<FEW>(teams, ms, fa, A0, mg.lv[1], n_fine, fine_tile);
                if (!grid_reduce<1>(acc, sh, w, gen, nblk, blk)) return;
                rho = acc[0];
            }
            // pass C, search direction: p' = z + beta p, q = A p', (p', q)
            const double beta = first ? 0.0 : rho / rho_old;
            rho_old = rho;
            {
                const float bf = (float)beta;
                fa.p = pc ? w.s1 : w.s0;
                fa.pn = pc ? w.s0 : w.s1;
                double acc[1] = {0.0};
                for (uint32_t e = gwarp; e < nloose; e += GW) {
                    const uint32_t* rec = loose_rec(e);
                    const uint32_t c = rec[lane];
                    if (c == ~0u) continue;
                    const uint32_t m = rec[64 + lane] >> 6;
                    // a neighbour in the grid, in the system or not: its code decides whether its value counts
                    const int step[6] = {-1, 1, -nx, nx, -(int)sxy, (int)sxy};
                    float zn[6], pn_[6];
                    uint32_t cn[6];
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        const int q = ((m >> k) & 1u) ? (int)c + step[k] : (int)c;
                        cn[k] = __ldcg(code + q);
                        zn[k] = __ldcg(Z + q);
                        pn_[k] = first ? 0.f : __ldcg(fa.p + q);
                    }
                    float pv = __ldcg(Z + c);
                    if (!first) pv += bf * __ldcg(fa.p + c);
                    float qc = 0.f;
#pragma unroll
                    for (int k = 0; k < 6; ++k)
                        if ((m >> k) & 1u) {
                            float o = 0.f;
                            if (cn[k] & 63u) o = first ? zn[k] : zn[k] + bf * pn_[k];
                            qc += ih2[k >> 1] * (pv - o);
                        }
                    fa.pn[c] = pv;
                    Q[c] = qc;
                    acc[0] += (double)pv * (double)qc;
                }
                if (many) acc[0] += fine_search<MANY>(teams, ms, fa, Q, A0, bf, first, n_fine, fine_tile);
                else acc[0] += fine_search<FEW>(teams, ms, fa, Q, A0, bf, first, n_fine, fine_tile);
                if (!grid_reduce<1>(acc, sh, w, gen, nblk, blk)) return;
                first = false;
                pc ^= 1;
                const double a = rho / acc[0];
                if (!(a > 0.0) || !isfinite(a)) {  // FP32 breakdown: leave it to the outer loop, which starts afresh
                    first = true;
                    break;
                }
                alpha = (float)a;
            }
        }
        // ---- p += e (FP64); the next residual pass reads neighbours' p, hence the barrier
        for_cells([&](size_t c, uint32_t) { p64[c] = __ldcg(p64 + c) + (double)X[c]; });
        if (!grid_sync(w, gen, nblk, sh, blk)) return;
    }
    // A tank full of fluid (no air, so no cell has a fixed pressure) determines p up to a constant.  The plain CG keeps the mean
    // that p starts with; the preconditioner moves it, so it is put back.
    if ((size_t)F == nc && refinements > 0) {
        __syncthreads();
        const double shift = (ms.p_sum[1] - ms.p_sum[0]) / (double)F;
        for (size_t c = (size_t)blk * blockDim.x + threadIdx.x; c < nc; c += (size_t)nblk * blockDim.x) p64[c] = __ldcg(p64 + c) - shift;
    }
    if (blk == 0 && threadIdx.x == 0 && out_its) {
        *out_its = total_it;
        *out_fluid = F;
    }
    if (blk == 0 && threadIdx.x == 0 && prm.stats_ring) {
        const unsigned slot = atomicAdd(prm.stats_counter, 1u) % prm.stats_cap;
        fe_step_stats st;
        st.cg_iterations = total_it;
        st.refinements = refinements;
        st.converged = converged ? 1 : 0;
        st.fluid_cells = F;
        st.rel_residual = bnorm > 0.0 ? rnorm / bnorm : rnorm;
        st.b_norm = bnorm;
        prm.stats_ring[slot] = st;
    }
}

// Dynamic shared memory of the body with `threads` threads per block.
inline size_t mg_dynamic_smem(int threads)
{
    return (size_t)(threads / 256) * sizeof(MgTeam) + (size_t)(threads / 32) * 96 * sizeof(uint32_t);
}

}  // namespace
}  // namespace fe
