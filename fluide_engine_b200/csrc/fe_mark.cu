// fe_mark.cu -- FLUID / AIR cell marking (K_mark), bit-exact with the reference.
//
// Reference: PICSimulator::BuildSignedDistanceField (pic_simulator.cpp:452-475) builds, at every
// cell-centred node c, sdf(c) = min(2r, min |p - c| over the particles its hash searcher visits) - r
// with r = 1.2 max(h) / sqrt(2); HashGridParticleSearcher::ForEachNearbyPoint
// (particle_systems/hash_grid_particle_searcher.cpp:97-126,154-204) visits the particles of 8 buckets of
// edge 2r (the node's bucket and, per axis, the neighbour on the side of the node's half) whose squared
// distance is <= (2r)^2.  SinglePhasePressureSolver::BuildMarkers (fluid_solvers/
// single_phase_pressure_solver.cpp:30-48) then marks a cell FLUID iff the trilinear sample of sdf at
// the cell centre is < 0.
//
// When the cell-centre sample lands exactly on node c (every power-of-two grid on an origin-0 domain,
// checked per axis on the host), the mark is FLUID iff some visited particle has |p - c| < r, because
// a - r < 0 <=> a < r in IEEE arithmetic.  K_mark therefore scatters from particles: each particle tests
// the few nodes within r of it with the reference's exact FP64 expressions (no fused multiply-add,
// correctly rounded sqrt, the same bucket membership) and stores FLUID.  On axes where the sample is off
// the node by a rounding error, the sign of the sample equals the sign of the node value unless the
// node value is within ~1e-15 r of zero; such "critical" cells are listed and re-evaluated with the full
// band SDF and the reference's trilinear sample by k_mark_fixup.  The result is byte-identical to the
// reference in every case.
#include <cmath>

#include "fe_internal.cuh"

namespace fe {
namespace {

__device__ __forceinline__ double dist2_ref(double px, double py, double pz, double cx, double cy, double cz)
{
    // (p - c).GetLengthSquared() = x*x + y*y + z*z, left to right, each operation rounded
    double dx = __dsub_rn(px, cx), dy = __dsub_rn(py, cy), dz = __dsub_rn(pz, cz);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ int bucket_of(double x, double spacing)
{
    return (int)floor(__ddiv_rn(x, spacing));
}

// floor(x / spacing) exactly as the reference computes it; the multiply by the reciprocal decides it
// unless the quotient is within 1e-9 of an integer, where the correctly rounded division is used.
__device__ __forceinline__ int bucket_fast(double x, double spacing, double inv_spacing)
{
    const double q = x * inv_spacing;
    const double fq = floor(q);
    const double fr = q - fq;
    if (fr > 1e-9 && fr < 1.0 - 1e-9) return (int)fq;
    return bucket_of(x, spacing);
}

__device__ __forceinline__ bool visited(const SceneView& v, int pbx, int pby, int pbz, int i, int j, int k)
{
    return (pbx == v.q_b0[0][i] || pbx == v.q_b1[0][i]) && (pby == v.q_b0[1][j] || pby == v.q_b1[1][j]) &&
           (pbz == v.q_b0[2][k] || pbz == v.q_b1[2][k]);
}

// One thread per particle: the nodes within r of it (2 per axis for cubic cells, where 2r = 1.7 h;
// more along an axis whose spacing is finer than max(h)) get the reference's exact FP64 test.
// A node the particle is within band of: FLUID when within r; on grids with inexact cell-centre samples, a node
// whose distance is within crit_eps of r is listed for the full trilinear sample.
__device__ __forceinline__ void mark_node(const SceneView& v, const MarkConst& mc, double d2, int i, int j, int k)
{
    if (!(d2 <= mc.R2)) return;
    const size_t c = idx3(i, j, k, v.g.nx, v.g.ny);
    // sqrt(d2) < r exactly when d2 <= rin2 (correctly rounded sqrt is monotonic): no square root
    if (d2 <= mc.rin2) v.marks[c] = FE_CELL_FLUID;
    if (v.any_inexact && !(v.q_exact[0][i] && v.q_exact[1][j] && v.q_exact[2][k]) &&
        fabs(__dsqrt_rn(d2) - v.radius) <= mc.crit_eps) {
        unsigned* word = (unsigned*)(v.crit_flag + (c & ~(size_t)3));
        unsigned bit = 1u << (8 * (c & 3));
        if (!(atomicOr(word, bit) & bit)) {
            uint32_t slot = atomicAdd(v.crit_count, 1u);
            v.crit_list[slot] = (uint32_t)c;
        }
    }
}

// The common case, every axis' node window holding at most two nodes (cubic cells: 2r = 1.7 h): the 2 x 2 x 2
// candidates are tested without loops, every table load issued first and each node's test predicated, so the
// lanes of a warp stay converged.  Same nodes, same FP64 expressions and bucket tests as mark_body's loops.
__device__ __forceinline__ void mark_particle2(const SceneView& v, const MarkConst& mc, uint64_t p)
{
    const double X[3] = {(double)v.px[p], (double)v.py[p], (double)v.pz[p]};
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    int node[3][2];
    bool ok[3][2];
    double q[3][2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double t = (X[a] - v.sdf_origin[a]) * v.inv_h[a];
        const double rr = v.radius * v.inv_h[a] + 1e-6;
        const int lo = max((int)floor(t - rr) + 1, 0);
        const int hi = min((int)floor(t + rr), n[a] - 1);
        const int pb = bucket_fast(X[a], v.bucket, mc.inv_bucket);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int idx = min(lo + s, n[a] - 1);  // clamped for the loads; out-of-window nodes are not ok
            node[a][s] = idx;
            ok[a][s] = lo + s <= hi && (pb == v.q_b0[a][idx] || pb == v.q_b1[a][idx]);
            q[a][s] = v.q_pos[a][idx];
        }
    }
#pragma unroll
    for (int sk = 0; sk < 2; ++sk)
#pragma unroll
        for (int sj = 0; sj < 2; ++sj)
#pragma unroll
            for (int si = 0; si < 2; ++si)
                if (ok[2][sk] && ok[1][sj] && ok[0][si])
                    mark_node(v, mc, dist2_ref(X[0], X[1], X[2], q[0][si], q[1][sj], q[2][sk]), node[0][si],
                              node[1][sj], node[2][sk]);
}

// The same candidates in FP32: nodes base + (0|1, 0|1, 0|1) with squared distances d2[0][.] + d2[1][.] + d2[2][.].  A node
// further inside r than the FP32 distance can be wrong is marked, one further outside is not; a particle with a node in
// between (about one in 10^4), or too far from the grid, takes the exact test, which also lists the critical cells.  The
// buckets need no test for a node inside r by that much: its search visits all of them.  near: bit a + 3 b + 9 c of the
// nodes that are marked.  Returns false when the particle needs the exact test.
__device__ __forceinline__ bool near_nodes(const SceneView& v, const MarkConst& mc, const float X[3], int base[3],
                                           uint32_t& near)
{
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    float d2[3][2];
    bool in[3][2];
    bool fine = mc.fp32 != 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float t = (X[a] - v.originf[a]) * v.inv_hf[a] - 0.5f;  // in cells from the first node
        const float fl = floorf(t);
        fine = fine && fabsf(t) < 1e6f;
        base[a] = (int)fl;
        const float lo = (t - fl) * v.hf[a], hi = (1.f - (t - fl)) * v.hf[a];
        d2[a][0] = lo * lo;
        d2[a][1] = hi * hi;
        in[a][0] = (unsigned)base[a] < (unsigned)n[a];
        in[a][1] = (unsigned)(base[a] + 1) < (unsigned)n[a];
    }
    near = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int a = t & 1, b = (t >> 1) & 1, c = t >> 2;
        const float d = d2[0][a] + d2[1][b] + d2[2][c];
        const bool inside = in[0][a] && in[1][b] && in[2][c];
        if (inside && d < mc.near2) near |= 1u << (a + 3 * b + 9 * c);
        fine = fine && !(inside && d >= mc.near2 && d <= mc.far2);
    }
    return fine;
}

// One thread per particle (any order of the particles): 75 us at 128^3, bound by the byte stores; 100.7 with FP64 tests
// of all 8 nodes.
__device__ __forceinline__ void mark_particle(const SceneView& v, const MarkConst& mc, uint64_t p)
{
    const float X[3] = {v.px[p], v.py[p], v.pz[p]};
    int base[3];
    uint32_t near;
    if (!near_nodes(v, mc, X, base, near)) {
        mark_particle2(v, mc, p);
        return;
    }
    const int64_t c0 = (int64_t)base[0] + (int64_t)v.g.nx * ((int64_t)base[1] + (int64_t)v.g.ny * (int64_t)base[2]);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int a = t & 1, b = (t >> 1) & 1, c = t >> 2;
        if ((near >> (a + 3 * b + 9 * c)) & 1u)
            v.marks[c0 + a + (int64_t)v.g.nx * ((int64_t)b + (int64_t)v.g.ny * (int64_t)c)] = FE_CELL_FLUID;
    }
}
__device__ __forceinline__ void mark_body2(const SceneView& v, const MarkConst& mc, uint32_t blk)
{
    const uint64_t p = blk * (uint64_t)blockDim.x + threadIdx.x;
    if (p < v.np) mark_particle(v, mc, p);
}

// Many particles, sorted by their cells, in two passes, because nearly every cell that holds particles is marked by its
// own: a particle is in reach of its cell's centre unless it sits in a corner, and stores of marks are what the pass
// above is bound by.
//   own    a thread per particle tests its own cell's node alone
//   near   a block per 8^3-cell tile: the cells with an unmarked node among the 27 around them test all their particles
//          against all their nodes, 8 lanes a cell, a cell of more than kNearLanesCap the whole block; the others are done
//          without reading a particle
// A node that is marked needs no further test: one particle in reach decides it, and on grids with inexact cell-centre
// samples a mark set from within crit_eps of r is listed when it is set, while one set from further inside makes the
// sample negative whatever else is near.
__device__ __forceinline__ void mark_own_body(const SceneView& v, const MarkConst& mc, uint32_t blk)
{
    const uint64_t p = blk * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= v.np) return;
    const float X[3] = {v.px[p], v.py[p], v.pz[p]};
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    int c[3];
    float d2 = 0.f;
    bool in = mc.fp32 != 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float t = (X[a] - v.originf[a]) * v.inv_hf[a];
        const float fl = floorf(t);
        c[a] = (int)fl;
        in = in && t >= 0.f && t < (float)n[a];
        const float d = (t - fl - 0.5f) * v.hf[a];
        d2 += d * d;
    }
    // the FP32 fraction is within near2's margin of the exact one whichever cell the rounding puts the particle in
    if (in && d2 < mc.near2) v.marks[idx3(c[0], c[1], c[2], n[0], n[1])] = FE_CELL_FLUID;
}
struct MarkShared {
    uint8_t open[10 * 10 * 10];       // 1 where a node in the grid is not marked: the tile and one cell around it
    uint16_t list[FE_TILE_CELLS];     // cells to test: from the front 8 lanes each, from the back the whole block
    int count, crowded;
};
// Particles that 8 lanes test for one cell.  Fluid that has splashed piles up along the walls: with 8 lanes a cell whatever it
// holds, a 128^3 FLIP dam break after 480 substeps, 1600 to 2000 particles in its fullest cell, took 172 us here (one pass over the
// particles 112), now 46.
constexpr uint32_t kNearLanesCap = 64;
constexpr int kNearThreads = 256;
__device__ __forceinline__ void mark_near_body(const SceneView& v, const MarkConst& mc, int tile, MarkShared& sh)
{
    const uint32_t first = (uint32_t)tile * FE_TILE_CELLS;
    if (v.cell_start[first] == v.cell_start[first + FE_TILE_CELLS]) return;
    const int x0 = tile % v.g.tnx * FE_TILE, y0 = (tile / v.g.tnx) % v.g.tny * FE_TILE, z0 = tile / (v.g.tnx * v.g.tny) * FE_TILE;
    if (threadIdx.x == 0) sh.count = sh.crowded = 0;
    for (int q = (int)threadIdx.x; q < 1000; q += (int)blockDim.x) {
        const int i = x0 - 1 + q % 10, j = y0 - 1 + (q / 10) % 10, k = z0 - 1 + q / 100;
        const bool in = (unsigned)i < (unsigned)v.g.nx && (unsigned)j < (unsigned)v.g.ny && (unsigned)k < (unsigned)v.g.nz;
        sh.open[q] = in && v.marks[idx3(i, j, k, v.g.nx, v.g.ny)] != FE_CELL_FLUID ? 1 : 0;
    }
    __syncthreads();
    for (int t = (int)threadIdx.x; t < FE_TILE_CELLS; t += (int)blockDim.x) {
        const uint32_t held = v.cell_start[first + t + 1] - v.cell_start[first + t];
        if (held == 0) continue;
        const uint8_t* o = sh.open + (t & 7) + 10 * ((t >> 3) & 7) + 100 * (t >> 6);
        unsigned any = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) any |= o[10 * j + 100 * k] | o[10 * j + 100 * k + 1] | o[10 * j + 100 * k + 2];
        if (any) {
            if (held <= kNearLanesCap) sh.list[atomicAdd(&sh.count, 1)] = (uint16_t)t;
            else sh.list[FE_TILE_CELLS - 1 - atomicAdd(&sh.crowded, 1)] = (uint16_t)t;
        }
    }
    __syncthreads();
    // one loop for both kinds of cell (with two calls of mark_particle 6 us more at 128^3)
#pragma unroll 1
    for (int lg = 3; lg <= 8; lg += 5) {  // 8 lanes, then the block's 256
        const int n = lg == 3 ? sh.count : sh.crowded;
        for (int e = (int)threadIdx.x >> lg; e < n; e += kNearThreads >> lg) {
            const uint32_t key = first + sh.list[lg == 3 ? e : FE_TILE_CELLS - 1 - e];
            const uint32_t step = 1u << lg;
            for (uint32_t p = v.cell_start[key] + (threadIdx.x & (step - 1u)), pe = v.cell_start[key + 1]; p < pe; p += step)
                mark_particle(v, mc, p);
        }
    }
}

__device__ __forceinline__ void mark_body(const SceneView& v, const MarkConst& mc, uint32_t blk)
{
    uint64_t p = blk * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= v.np) return;
    const double X[3] = {(double)v.px[p], (double)v.py[p], (double)v.pz[p]};
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    const double inv_bucket = mc.inv_bucket;
    int lo[3], hi[3], pb[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // nodes i with |q_i - x| < r, widened by 1e-6 h (the exact test below decides)
        const double t = (X[a] - v.sdf_origin[a]) * v.inv_h[a];
        const double rr = v.radius * v.inv_h[a] + 1e-6;
        lo[a] = max((int)floor(t - rr) + 1, 0);
        hi[a] = min((int)floor(t + rr), n[a] - 1);
        pb[a] = bucket_fast(X[a], v.bucket, inv_bucket);
    }
    for (int k = lo[2]; k <= hi[2]; ++k) {
        if (pb[2] != v.q_b0[2][k] && pb[2] != v.q_b1[2][k]) continue;
        for (int j = lo[1]; j <= hi[1]; ++j) {
            if (pb[1] != v.q_b0[1][j] && pb[1] != v.q_b1[1][j]) continue;
            for (int i = lo[0]; i <= hi[0]; ++i) {
                if (pb[0] != v.q_b0[0][i] && pb[0] != v.q_b1[0][i]) continue;
                mark_node(v, mc, dist2_ref(X[0], X[1], X[2], v.q_pos[0][i], v.q_pos[1][j], v.q_pos[2][k]), i, j, k);
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_mark(SceneView v, MarkConst mc)
{
    if (mc.two) mark_body2(v, mc, blockIdx.x);
    else mark_body(v, mc, blockIdx.x);
}

// Band-limited SDF value of node (i, j, k) exactly as BuildSignedDistanceField computes it.
__device__ double node_sdf(const SceneView& v, int i, int j, int k, double R2)
{
    const double q[3] = {v.q_pos[0][i], v.q_pos[1][j], v.q_pos[2][k]};
    double minDistance = v.band;
    const int c0[3] = {i, j, k};
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    int lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // particles within the band 2r of the node lie in cells within ceil(2r/h + 0.5) of it
        const int reach = (int)ceil(v.band * v.inv_h[a] + 0.5) + 1;
        lo[a] = max(c0[a] - reach, 0);
        hi[a] = min(c0[a] + reach, n[a] - 1);
    }
    for (int cz = lo[2]; cz <= hi[2]; ++cz)
        for (int cy = lo[1]; cy <= hi[1]; ++cy)
            for (int cx = lo[0]; cx <= hi[0]; ++cx) {
                const uint32_t key = fe_cell_key(cx, cy, cz, n[0], n[1]);
                for (uint32_t p = v.cell_start[key]; p < v.cell_start[key + 1]; ++p) {
                    const double X = v.px[p], Y = v.py[p], Z = v.pz[p];
                    if (!visited(v, bucket_of(X, v.bucket), bucket_of(Y, v.bucket), bucket_of(Z, v.bucket), i, j, k))
                        continue;
                    const double d2 = dist2_ref(X, Y, Z, q[0], q[1], q[2]);
                    if (!(d2 <= R2)) continue;
                    const double dist = __dsqrt_rn(d2);
                    if (dist < minDistance) minDistance = dist;
                }
            }
    return __dsub_rn(minDistance, v.radius);
}

__device__ __forceinline__ double lerp_ref(double a, double b, double f)
{
    return __dadd_rn(__dmul_rn(__dsub_rn(1.0, f), a), __dmul_rn(f, b));
}

// ScalarGrid3D::Sample at the cell centre (3d/scalar_grid3d.cpp:33-65) with exact band SDF values.
__device__ double sample_cell_sdf(const SceneView& v, int i, int j, int k, double R2)
{
    const int i0 = v.q_i0[0][i], j0 = v.q_i0[1][j], k0 = v.q_i0[2][k];
    const double fx = v.q_f[0][i], fy = v.q_f[1][j], fz = v.q_f[2][k];
    const int ip = min(i0 + 1, v.g.nx - 1), jp = min(j0 + 1, v.g.ny - 1), kp = min(k0 + 1, v.g.nz - 1);
    const double c000 = node_sdf(v, i0, j0, k0, R2), c100 = node_sdf(v, ip, j0, k0, R2);
    const double c010 = node_sdf(v, i0, jp, k0, R2), c110 = node_sdf(v, ip, jp, k0, R2);
    const double c001 = node_sdf(v, i0, j0, kp, R2), c101 = node_sdf(v, ip, j0, kp, R2);
    const double c011 = node_sdf(v, i0, jp, kp, R2), c111 = node_sdf(v, ip, jp, kp, R2);
    const double b0 = lerp_ref(lerp_ref(c000, c100, fx), lerp_ref(c010, c110, fx), fy);
    const double b1 = lerp_ref(lerp_ref(c001, c101, fx), lerp_ref(c011, c111, fx), fy);
    return lerp_ref(b0, b1, fz);
}

__device__ __forceinline__ void mark_fixup_body(const SceneView& v, double R2, uint32_t cap, uint32_t blk, uint32_t nblk)
{
    const uint32_t count = min(*v.crit_count, cap);
    for (uint32_t t = blk * blockDim.x + threadIdx.x; t < count; t += nblk * blockDim.x) {
        const uint32_t c = v.crit_list[t];
        const int i = c % v.g.nx, j = (c / v.g.nx) % v.g.ny, k = c / (v.g.nx * v.g.ny);
        v.marks[c] = sample_cell_sdf(v, i, j, k, R2) < 0.0 ? FE_CELL_FLUID : FE_CELL_AIR;
    }
}

__global__ void k_mark_fixup(SceneView v, double R2, uint32_t cap) { mark_fixup_body(v, R2, cap, blockIdx.x, gridDim.x); }

__global__ void __launch_bounds__(256) k_mark_own(SceneView v, MarkConst mc) { mark_own_body(v, mc, blockIdx.x); }
__global__ void __launch_bounds__(kNearThreads) k_mark_near(SceneView v, MarkConst mc)
{
    __shared__ MarkShared sh;
    mark_near_body(v, mc, (int)blockIdx.x, sh);
}

// ---- flat multi-scene forms (BatchPlan, fe_internal.cuh); marks, crit flags and counts are cleared by
// launch_multi_clear
__global__ void __launch_bounds__(256) k_multi_mark(const BatchPlan* __restrict__ plan)
{
    uint32_t b;
    const int s = batch_scene_of(plan, kBkPart, b);
    const BatchScene& e = plan->sc[s];
    if (e.mark.two) mark_body2(e.dst, e.mark, b);
    else mark_body(e.dst, e.mark, b);
}

__global__ void __launch_bounds__(128) k_multi_mark_fixup(const BatchPlan* __restrict__ plan)
{
    __shared__ SceneView v;
    uint32_t b;
    const int s = batch_scene_of(plan, kBkFixup, b);
    const BatchScene& e = plan->sc[s];
    stage_view(v, e.dst);
    mark_fixup_body(v, e.mark.R2, (uint32_t)((size_t)v.g.nx * v.g.ny * v.g.nz), b,
                    plan->start[kBkFixup][s + 1] - plan->start[kBkFixup][s]);
}

__global__ void k_fluid_sdf(SceneView v, double R2, double* out)
{
    const size_t nc = (size_t)v.g.nx * v.g.ny * v.g.nz;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const int i = c % v.g.nx, j = (c / v.g.nx) % v.g.ny, k = c / ((size_t)v.g.nx * v.g.ny);
        out[c] = v.np ? node_sdf(v, i, j, k, R2) : __dsub_rn(v.band, v.radius);
    }
}


// One thread per particle: every SDF node within the band 2r of the particle that the reference's hash search
// would visit from that node and whose squared distance is <= (2r)^2 takes the minimum of that squared distance.
// The node's reference value is min(2r, min over those particles of |p - c|) - r; correctly rounded sqrt is
// monotonic, so min |p - c| = sqrt(min |p - c|^2) exactly, and the square root is taken once per node when the
// markers are sampled.  Squared distances are non-negative doubles, whose bit patterns order like their values,
// so a 64-bit atomicMin on the bits takes the minimum.  Each squared distance is summed in the reference's order,
// (dx^2 + dy^2) + dz^2; a row whose dy^2 + dz^2 already exceeds (2r)^2 is skipped (rounding is monotonic, so the
// full sum would exceed it too), and the bucket test runs once per axis.  Particles sorted by cell hit the same
// nodes as their neighbours; a plain read of the current minimum first (it only decreases, so a stale value is
// still an upper bound) skips most atomics.  For particles whose cells are not known and bands wider than k_sdf_gather's
// reach.
__global__ void __launch_bounds__(256) k_sdf_scatter(SceneView v, unsigned long long* __restrict__ node, double R2)
{
    uint64_t p = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (p >= v.np) return;
    const double X[3] = {(double)v.px[p], (double)v.py[p], (double)v.pz[p]};
    const int n[3] = {v.g.nx, v.g.ny, v.g.nz};
    const double inv_bucket = 1.0 / v.bucket;
    int lo[3], hi[3];
    unsigned long long pass[3];  // bit u: candidate node lo + u is in a bucket the node's search visits
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        // nodes i with |q_i - x| <= 2r, widened by 1e-6 h (the exact test below decides)
        const double t = (X[a] - v.sdf_origin[a]) * v.inv_h[a];
        const double rr = v.band * v.inv_h[a] + 1e-6;
        lo[a] = max((int)floor(t - rr) + 1, 0);
        hi[a] = min(min((int)floor(t + rr), n[a] - 1), lo[a] + 63);  // 2r spans at most 64 nodes per axis
        const int pb = bucket_fast(X[a], v.bucket, inv_bucket);
        pass[a] = 0ull;
        for (int i = lo[a]; i <= hi[a]; ++i)
            if (pb == v.q_b0[a][i] || pb == v.q_b1[a][i]) pass[a] |= 1ull << (i - lo[a]);
    }
    const double* qx = v.q_pos[0];
    for (int k = lo[2]; k <= hi[2]; ++k) {
        if (!((pass[2] >> (k - lo[2])) & 1ull)) continue;
        const double dz = __dsub_rn(X[2], v.q_pos[2][k]);
        const double dz2 = __dmul_rn(dz, dz);
        if (!(dz2 <= R2)) continue;
        for (int j = lo[1]; j <= hi[1]; ++j) {
            if (!((pass[1] >> (j - lo[1])) & 1ull)) continue;
            const double dy = __dsub_rn(X[1], v.q_pos[1][j]);
            const double dy2 = __dmul_rn(dy, dy);
            if (!(__dadd_rn(dy2, dz2) <= R2)) continue;
            for (int i = lo[0]; i <= hi[0]; ++i) {
                if (!((pass[0] >> (i - lo[0])) & 1ull)) continue;
                const double dx = __dsub_rn(X[0], qx[i]);
                const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), dy2), dz2);  // dist2_ref's order
                if (!(d2 <= R2)) continue;
                const unsigned long long bits = (unsigned long long)__double_as_longlong(d2);
                unsigned long long* cell = node + idx3(i, j, k, n[0], n[1]);
                if (bits < __ldcg(cell)) atomicMin(cell, bits);
            }
        }
    }
}

// Node values of BuildSignedDistanceField (pic_simulator.cpp:452-475): min(2r, sqrt(smallest squared distance)) - r.
__device__ __forceinline__ double node_value(unsigned long long raw, double band, double radius)
{
    double m = band;
    if (raw != ~0ull) {
        const double dm = __dsqrt_rn(__longlong_as_double((long long)raw));
        if (dm < m) m = dm;
    }
    return __dsub_rn(m, radius);
}

// In place: a node's distance bits become its value.
__global__ void k_node_values(double* node, size_t nc, double band, double radius)
{
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x)
        node[c] = node_value((unsigned long long)__double_as_longlong(node[c]), band, radius);
}

// The same node values from particles that are grouped by cell, gathered per node: no atomics, and nearly every node
// inside the fluid is decided by its own cell, because a particle nearer than half a cell is nearer than any of another
// cell.  A block takes a tile's nodes.  Nodes whose own cell doesn't decide are listed, so that warps are full again, and
// walk the occupied cells up to two away (the band is at most 2.5 cells wide, see node_reach), nearer ones first; a
// cell is skipped when its nearest point is further away than the smallest distance so far.  Where a cell holds too many
// particles for one thread, a warp searches all cells.  `order` (optional) gives the particle of each slot of the cells'
// runs.
//
// Bound by the latency of the listed nodes' searches (a lone particle has some 80 nodes search for it).  Against the scatter
// over particles below, which tests 64 nodes a particle and reads 21 of them: 4 M particles at 128^3 (FLIP dam with spray,
// unsorted) 512 us against 183, and 50 for grouping them; 0.5 M sorted ones at 64^3 92 against 50.  With a warp per listed
// node 630 and 160, with one walk over the rows instead of the groups of bits 321 and 82, with the bucket test for the nearest
// particle alone and a warp's search where it fails 210 and 58; four lanes a listed node gave nothing.
//
// The 125 cells around a node come in five groups, nearer ones first: the 27 that touch the node's cell, those two away along
// x in the same rows, then the 16 rows around (6, 6 and 4 of 5 cells).  A thread collects a group's occupied cells as bits
// and visits bit after bit, so that the lanes of a warp, whose nodes lie next to other cells, all have a cell to visit.
constexpr int kNodeGroups = 5, kNodeCells = 125;
struct NodeReach {
    double near2[kNodeCells];         // squared distance from a node to the nearest point of the cell
    double group2[kNodeGroups];       // the smallest of the group
    uint32_t valid[kNodeGroups];      // cells that reach into the band
    int8_t span[25];                  // of a row, (dy + 2) + 5 (dz + 2): cells at most so far along x do (-1: none)
    double own2;                      // squared distance up to which the node's own cell decides
    double safe2;                     // ... and below which a particle is in a bucket that the node's search visits
};
__host__ __device__ constexpr int node_group_first(int w) { return w == 0 ? 0 : (w == 1 ? 27 : 45 + 30 * (w - 2)); }
// Rows around a node, (dy + 2) + 5 (dz + 2): the 9 that touch its cell's row, then the 16 around, nearer ones first.
__host__ __device__ constexpr int node_row(int r)
{
    constexpr int rows[25] = {12, 7, 11, 13, 17, 6, 8, 16, 18, 2, 10, 14, 22, 1, 3, 5, 9, 15, 19, 21, 23, 0, 4, 20, 24};
    return rows[r];
}
// Offset of the cell of bit `bit` of group `w`.
__host__ __device__ constexpr void node_cell(int w, int bit, int d[3])
{
    const int width = w == 0 ? 3 : (w == 1 ? 2 : 5);
    const int row = node_row(w < 2 ? bit / width : 9 + 6 * (w - 2) + bit / width), x = bit % width;
    d[0] = w == 0 ? x - 1 : (w == 1 ? 4 * x - 2 : x - 2);
    d[1] = row % 5 - 2;
    d[2] = row / 5 - 2;
}

// Offsets of the cells in a block's halo, group after group.
struct NodeOffsets {
    int16_t at[kNodeCells];
};

// A block takes half a tile: 256 nodes, and the cells up to two around them.
constexpr int kNodeLayers = FE_TILE / 2;
constexpr int kNodeThreads = FE_TILE * FE_TILE * kNodeLayers;
constexpr int kNodeHalo = FE_TILE + 4, kNodeHaloZ = kNodeLayers + 4;
constexpr uint32_t kNodeLaneCap = 32;  // particles a thread tests for one cell; fuller cells are spread over a warp
constexpr NodeOffsets make_node_offsets()
{
    NodeOffsets t{};
    int n = 0;
    for (int w = 0; w < kNodeGroups; ++w)
        for (int bit = 0; n < (w + 1 < kNodeGroups ? node_group_first(w + 1) : kNodeCells); ++bit) {
            int d[3] = {0, 0, 0};
            node_cell(w, bit, d);
            t.at[n++] = (int16_t)(d[0] + kNodeHalo * (d[1] + kNodeHalo * d[2]));
        }
    return t;
}
__device__ const NodeOffsets g_node_offsets = make_node_offsets();
struct NodeShared {
    uint32_t start[kNodeHalo * kNodeHalo * kNodeHaloZ], count[kNodeHalo * kNodeHalo * kNodeHaloZ];
    uint16_t row[kNodeHalo * kNodeHaloZ];  // occupied cells of a row, a bit each
    uint8_t near[FE_TILE * kNodeLayers];   // nodes of a row with an occupied cell that reaches into their band
    uint16_t list[kNodeThreads];           // nodes to search, a thread each
    uint16_t hard[kNodeThreads];           // ... the crowded cells, a warp each; `out` holds the others' smallest squared distance
    double near2[kNodeCells];
    int16_t cell[kNodeCells];              // offset in start and count
    int n, nhard;
};
template <bool ORDER>
__global__ void __launch_bounds__(kNodeThreads, 4) k_sdf_gather(SceneView v, const uint32_t* __restrict__ cell_start,
                                                                const uint32_t* __restrict__ order,
                                                                const __grid_constant__ NodeReach reach, double R2,
                                                                double* __restrict__ out)
{
    __shared__ NodeShared sh;
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    const int tile = (int)blockIdx.x >> 1;
    const int tx = tile % v.g.tnx, ty = (tile / v.g.tnx) % v.g.tny, tz = tile / (v.g.tnx * v.g.tny);
    const int x0 = tx * FE_TILE, y0 = ty * FE_TILE, z0 = tz * FE_TILE + ((int)blockIdx.x & 1) * kNodeLayers;
    const double inv_bucket = 1.0 / v.bucket;

    bool any = false;
    if (threadIdx.x < 27) {
        const int i = tx - 1 + (int)threadIdx.x % 3, j = ty - 1 + (int)threadIdx.x / 3 % 3, k = tz - 1 + (int)threadIdx.x / 9;
        if ((unsigned)i < (unsigned)v.g.tnx && (unsigned)j < (unsigned)v.g.tny && (unsigned)k < (unsigned)v.g.tnz) {
            const uint32_t first = (uint32_t)(i + v.g.tnx * (j + v.g.tny * k)) * FE_TILE_CELLS;
            any = cell_start[first] != cell_start[first + FE_TILE_CELLS];
        }
    }
    const bool occupied = __syncthreads_or(any);
    if (occupied) {
        for (int q = (int)threadIdx.x; q < kNodeHalo * kNodeHalo * kNodeHaloZ; q += kNodeThreads) {
            const int i = x0 - 2 + q % kNodeHalo, j = y0 - 2 + q / kNodeHalo % kNodeHalo, k = z0 - 2 + q / (kNodeHalo * kNodeHalo);
            uint32_t beg = 0, end = 0;
            if ((unsigned)i < (unsigned)nx && (unsigned)j < (unsigned)ny && (unsigned)k < (unsigned)nz) {
                const uint32_t key = (uint32_t)((i >> 3) + v.g.tnx * ((j >> 3) + v.g.tny * (k >> 3))) * FE_TILE_CELLS +
                                     (uint32_t)((i & 7) + 8 * (j & 7) + 64 * (k & 7));
                beg = cell_start[key];
                end = cell_start[key + 1];
            }
            sh.start[q] = beg;
            sh.count[q] = end - beg;
        }
        if (threadIdx.x < kNodeCells) {
            sh.near2[threadIdx.x] = reach.near2[threadIdx.x];
            sh.cell[threadIdx.x] = g_node_offsets.at[threadIdx.x];
        }
        if (threadIdx.x == 0) sh.n = sh.nhard = 0;
    }
    __syncthreads();
    if (occupied)
        for (int r = (int)threadIdx.x; r < kNodeHalo * kNodeHaloZ; r += kNodeThreads) {
            unsigned bits = 0;
            for (int i = 0; i < kNodeHalo; ++i) bits |= sh.count[r * kNodeHalo + i] ? 1u << i : 0u;
            sh.row[r] = (uint16_t)bits;
        }
    __syncthreads();
    if (occupied && threadIdx.x < FE_TILE * kNodeLayers) {
        const uint16_t* row = sh.row + (threadIdx.x & 7) + kNodeHalo * (threadIdx.x >> 3);
        unsigned bits = 0;
#pragma unroll
        for (int b = 0; b < 25; ++b) {
            const unsigned x = row[b % 5 + kNodeHalo * (b / 5)];  // bit i + 2: the cell of node i
            const int span = reach.span[b];
            if (span >= 0) bits |= x >> 2;
            if (span >= 1) bits |= (x >> 1) | (x >> 3);
            if (span >= 2) bits |= x | (x >> 4);
        }
        sh.near[threadIdx.x] = (uint8_t)bits;
    }
    __syncthreads();
    // occupied cells of group w around local node (lx, ly, lz) that reach into the band
    auto group = [&](int w, int lx, int ly, int lz) {
        const uint16_t* row = sh.row + ly + kNodeHalo * lz;  // of (dy, dz) = (-2, -2)
        auto at = [&](int r) { return (unsigned)row[node_row(r) % 5 + kNodeHalo * (node_row(r) / 5)] >> lx; };
        unsigned m = 0;
        if (w < 2) {
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                const unsigned x = at(r);
                m |= w == 0 ? ((x >> 1) & 7u) << (3 * r) : ((x & 1u) | ((x >> 3) & 2u)) << (2 * r);
            }
        } else if (w == 2) {
#pragma unroll
            for (int r = 0; r < 6; ++r) m |= (at(9 + r) & 31u) << (5 * r);
        } else if (w == 3) {
#pragma unroll
            for (int r = 0; r < 6; ++r) m |= (at(15 + r) & 31u) << (5 * r);
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) m |= (at(21 + r) & 31u) << (5 * r);
        }
        return m & reach.valid[w];
    };

    auto value = [&](double best) { return __dsub_rn(best > R2 ? v.band : fmin(__dsqrt_rn(best), v.band), v.radius); };
    auto bucket_ok = [&](double X, double Y, double Z, int i, int j, int k) {
        return visited(v, bucket_fast(X, v.bucket, inv_bucket), bucket_fast(Y, v.bucket, inv_bucket),
                       bucket_fast(Z, v.bucket, inv_bucket), i, j, k);
    };
    // the nearest of the particles in slots [s, s + n) by the reference's squared distance, if nearer than best; the
    // buckets decide about particles more than half a bucket away only
    auto nearest = [&](uint32_t s, uint32_t n, int i, int j, int k, double qx, double qy, double qz, double& best) {
        constexpr int B = 4;
        for (uint32_t e = 0; e < n; e += B) {
            float x[B], y[B], z[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const uint32_t at = s + min(e + b, n - 1);
                const uint32_t p = ORDER ? __ldg(order + at) : at;
                x[b] = __ldg(v.px + p);
                y[b] = __ldg(v.py + p);
                z[b] = __ldg(v.pz + p);
            }
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const double d2 = dist2_ref((double)x[b], (double)y[b], (double)z[b], qx, qy, qz);
                if (d2 < best && (d2 < reach.safe2 || bucket_ok((double)x[b], (double)y[b], (double)z[b], i, j, k))) best = d2;
            }
        }
    };
    const double beyond = __longlong_as_double(__double_as_longlong(R2) + 1);  // the next double: best <= R2 counts

    {
        const int t = (int)threadIdx.x;
        const int lx = t & 7, ly = (t >> 3) & 7, lz = t >> 6;
        const int i = x0 + lx, j = y0 + ly, k = z0 + lz;
        if (i < nx && j < ny && k < nz) {
            double best = beyond;
            bool more = false;
            if (occupied) {
                const int q = lx + 2 + kNodeHalo * (ly + 2 + kNodeHalo * (lz + 2));
                const uint32_t n = sh.count[q];
                if (n > 0 && n <= kNodeLaneCap) nearest(sh.start[q], n, i, j, k, v.q_pos[0][i], v.q_pos[1][j], v.q_pos[2][k], best);
                more = !(best <= reach.own2) && ((sh.near[t >> 3] >> lx) & 1u);
            }
            if (more) sh.list[atomicAdd(&sh.n, 1)] = (uint16_t)t;
            else out[idx3(i, j, k, nx, ny)] = value(best);
        }
    }
    if (!occupied) return;
    __syncthreads();

    if ((int)threadIdx.x < sh.n) {
        const int t = sh.list[threadIdx.x];
        const int lx = t & 7, ly = (t >> 3) & 7, lz = t >> 6;
        const int i = x0 + lx, j = y0 + ly, k = z0 + lz;
        const int q0 = lx + 2 + kNodeHalo * (ly + 2 + kNodeHalo * (lz + 2));
        const double qx = v.q_pos[0][i], qy = v.q_pos[1][j], qz = v.q_pos[2][k];
        double best = beyond;
        bool full = false;
        for (int w = 0; w < kNodeGroups; ++w) {
            if (!(reach.group2[w] < best)) continue;
            const int first = node_group_first(w);
            for (unsigned m = group(w, lx, ly, lz); m; m &= m - 1) {
                const int c = first + __ffs(m) - 1;
                if (!(sh.near2[c] < best)) continue;
                const int q = q0 + sh.cell[c];
                const uint32_t n = sh.count[q];
                if (n <= kNodeLaneCap) nearest(sh.start[q], n, i, j, k, qx, qy, qz, best);
                else full = true;
            }
        }
        if (full) sh.hard[atomicAdd(&sh.nhard, 1)] = (uint16_t)t;
        out[idx3(i, j, k, nx, ny)] = full ? best : value(best);
    }
    __syncthreads();

    // the particle of slot s against node (i, j, k) at (qx, qy, qz): the reference's squared distance and bucket tests
    auto test = [&](uint32_t s, int i, int j, int k, double qx, double qy, double qz, double& best) {
        const uint32_t p = ORDER ? __ldg(order + s) : s;
        const double X = (double)__ldg(v.px + p), Y = (double)__ldg(v.py + p), Z = (double)__ldg(v.pz + p);
        const double d2 = dist2_ref(X, Y, Z, qx, qy, qz);
        if (d2 < best && (d2 < reach.safe2 || bucket_ok(X, Y, Z, i, j, k))) best = d2;
    };
    const int lane = (int)threadIdx.x & 31;
    for (int e = (int)threadIdx.x >> 5; e < sh.nhard; e += kNodeThreads >> 5) {
        const int t = sh.hard[e];
        const int lx = t & 7, ly = (t >> 3) & 7, lz = t >> 6;
        const int i = x0 + lx, j = y0 + ly, k = z0 + lz;
        const double qx = v.q_pos[0][i], qy = v.q_pos[1][j], qz = v.q_pos[2][k];
        double best = out[idx3(i, j, k, nx, ny)];  // in the other cells
        for (int first = 0; first < kNodeCells; first += 32) {  // each lane looks at a cell
            const int c = first + lane;
            uint32_t s = 0, n = 0;
            if (c < kNodeCells && sh.near2[c] < best) {
                const int q = lx + 2 + kNodeHalo * (ly + 2 + kNodeHalo * (lz + 2)) + sh.cell[c];
                s = sh.start[q];
                n = sh.count[q];
            }
            unsigned full = __ballot_sync(0xffffffffu, n > kNodeLaneCap);
            while (full) {
                const int from = __ffs(full) - 1;
                full &= full - 1;
                if (!(sh.near2[first + from] < best)) continue;
                const uint32_t fs = __shfl_sync(0xffffffffu, s, from), fn = __shfl_sync(0xffffffffu, n, from);
                for (uint32_t m = (uint32_t)lane; m < fn; m += 32) test(fs + m, i, j, k, qx, qy, qz, best);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
            }
        }
        if (lane == 0) out[idx3(i, j, k, nx, ny)] = value(best);
    }
}

// BackwardEulerDiffusionSolver::BuildX/Y/ZMarkers (fluid_solvers/backward_euler_diffusion_solver.cpp:71-128):
// a face is FLUID iff ScalarGrid3D::Sample (3d/scalar_grid3d.cpp:33-65) of the fluid SDF at the face centre is
// < 0.  The face centres are those of the copied velocity grid (data origins include the domain origin,
// grid_systems/face_centered_grid3d.cpp:11-17,303-316); their GetBarycentric index and fraction per axis come
// from host tables computed in FP64 with the reference's expressions.
__global__ void k_face_mark(SceneView v, DiffWork d)
{
    const int nx = v.g.nx, ny = v.g.ny, nz = v.g.nz;
    FaceCoord fc;
    if (!face_coord(nx, ny, nz, fc)) return;
    const int base = fc.c * 3 * d.tab_stride;
    const int i0 = d.tab_i0[base + fc.i], j0 = d.tab_i0[base + d.tab_stride + fc.j];
    const int k0 = d.tab_i0[base + 2 * d.tab_stride + fc.k];
    const double fx = d.tab_f[base + fc.i], fy = d.tab_f[base + d.tab_stride + fc.j];
    const double fz = d.tab_f[base + 2 * d.tab_stride + fc.k];
    const int ip = min(i0 + 1, nx - 1), jp = min(j0 + 1, ny - 1), kp = min(k0 + 1, nz - 1);
    const double* __restrict__ node = d.node;
    auto val = [&](int i, int j, int k) { return __ldg(node + idx3(i, j, k, nx, ny)); };
    const double c000 = val(i0, j0, k0), c100 = val(ip, j0, k0), c010 = val(i0, jp, k0), c110 = val(ip, jp, k0);
    const double c001 = val(i0, j0, kp), c101 = val(ip, j0, kp), c011 = val(i0, jp, kp), c111 = val(ip, jp, kp);
    const double b0 = lerp_ref(lerp_ref(c000, c100, fx), lerp_ref(c010, c110, fx), fy);
    const double b1 = lerp_ref(lerp_ref(c001, c101, fx), lerp_ref(c011, c111, fx), fy);
    const size_t off = fc.c == 0 ? 0 : (fc.c == 1 ? (size_t)(nx + 1) * ny * nz
                                                   : (size_t)(nx + 1) * ny * nz + (size_t)nx * (ny + 1) * nz);
    d.mark[off + fc.f] = lerp_ref(b0, b1, fz) < 0.0 ? FE_CELL_FLUID : FE_CELL_AIR;
}
}  // namespace

// Largest double d with sqrt(d) < r (sqrt correctly rounded, as IEEE 754 requires of the host's and the device's
// square root): the marking test sqrt(d2) < r becomes d2 <= sqrt_below(r), with the same outcome for every d2.
static double sqrt_below(double r)
{
    double t = r * r;
    while (t > 0.0 && std::sqrt(t) >= r) t = std::nextafter(t, 0.0);
    while (std::sqrt(std::nextafter(t, HUGE_VAL)) < r) t = std::nextafter(t, HUGE_VAL);
    return t;
}

cudaError_t launch_multi_mark(const BatchLaunch& L, cudaStream_t st)
{
    if (L.total[kBkPart]) {
        k_multi_mark<<<L.total[kBkPart], 256, 0, st>>>(L.plan);
        count_launch();
    }
    if (L.total[kBkFixup]) {
        k_multi_mark_fixup<<<L.total[kBkFixup], 128, 0, st>>>(L.plan);
        count_launch();
    }
    return cudaGetLastError();
}

// The marking constants of launch_mark: band^2, the largest squared distance whose square root is below r, and the
// window around r in which an inexact cell-centre sample is recomputed.
MarkConst mark_constants(const SceneView& v)
{
    MarkConst mc;
    mc.R2 = v.band * v.band;
    mc.rin2 = sqrt_below(v.radius);
    mc.crit_eps = 1e-9 * v.radius;
    mc.inv_bucket = 1.0 / v.bucket;
    mc.two = 1;
    for (int a = 0; a < 3; ++a)  // window (t - rr, t + rr] with rr = r / h_a + 1e-6 holds at most ceil(2 rr) nodes
        if (!(v.radius * v.inv_h[a] + 1e-6 < 1.0 - 1e-9)) mc.two = 0;
    // FP32 distances: x - origin, its product with 1 / h and the fraction are each rounded, in all less than 2^-24 times
    // |origin| + 4 |size| per axis and a few 2^-24 of the distance; twice that and more is left to the exact test
    double reach = 0.0;
    for (int a = 0; a < 3; ++a) reach = std::max(reach, std::fabs(v.origin[a]) + 4.0 * v.size[a]);
    const double delta = 4.0 * std::sqrt(3.0) * 6e-8 * reach + 1e-5 * v.radius;
    mc.fp32 = delta < 0.1 * v.radius ? 1 : 0;
    mc.near2 = std::nextafterf((float)((v.radius - delta) * (v.radius - delta)), 0.f);
    mc.far2 = std::nextafterf((float)((v.radius + delta) * (v.radius + delta)), HUGE_VALF);
    return mc;
}

// From this many particles on the two passes take less time than the one.  The passes before the solve, one marking pass
// against two: 0.6 M particles (64^3) 105.5 us against 107, 0.8 M (72^3) 149 against 150.5, 1.1 M (80^3) 172 against 172,
// 1.5 M (88^3) 206 against 203, 2 M (96^3) 252 against 239, 4.7 M (128^3) 520 against 490; of the kernels alone 75 against 50
// at 128^3 and 1018 against 363 at 256^3 (32 M).  Grids with inexact cell-centre samples take them at half as many: there the
// one pass lists the cell of every particle at a node's radius, also where another particle marks it, and fluid on a lattice
// (80^3, 1 M) took 15.5 ms against 0.055.
constexpr uint64_t kMarkTwoPasses = 1ull << 20, kMarkTwoPassesInexact = 1ull << 19;
cudaError_t launch_mark(const SceneView& v, bool cells_current, cudaStream_t st)
{
    const size_t nc = (size_t)v.g.nx * v.g.ny * v.g.nz;
    cudaError_t e = cudaMemsetAsync(v.marks, FE_CELL_AIR, nc, st);
    if (e != cudaSuccess) return e;
    const MarkConst mc = mark_constants(v);
    if (v.any_inexact) {
        if ((e = cudaMemsetAsync(v.crit_flag, 0, (nc + 3) & ~(size_t)3, st)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(v.crit_count, 0, sizeof(uint32_t), st)) != cudaSuccess) return e;
    }
    if (v.np > 0) {
        const unsigned nb = (unsigned)((v.np + 255) / 256);
        if (mc.two && cells_current && v.np >= (v.any_inexact ? kMarkTwoPassesInexact : kMarkTwoPasses)) {
            k_mark_own<<<nb, 256, 0, st>>>(v, mc);
            k_mark_near<<<(unsigned)(v.g.tnx * v.g.tny * v.g.tnz), kNearThreads, 0, st>>>(v, mc);
            count_launch(2);
        } else {
            k_mark<<<nb, 256, 0, st>>>(v, mc);
            count_launch();
        }
        if (v.any_inexact) {
            k_mark_fixup<<<148, 128, 0, st>>>(v, mc.R2, (uint32_t)nc);
            count_launch();
        }
    }
    return cudaGetLastError();
}

cudaError_t launch_fluid_sdf(const SceneView& v, double* out, cudaStream_t st)
{
    k_fluid_sdf<<<148 * 8, 128, 0, st>>>(v, v.band * v.band, out);
    count_launch();
    return cudaGetLastError();
}

// Cells up to two away hold every particle of a node's band, by the squared distances from a node (the centre of its cell) to
// the nearest points of other cells.  A particle may be listed in the cell next to its own when it is within the FP32
// rounding of their border, and in an outer cell when it is outside the grid (then it is further away than the cell).
// False when the band is wider than that.
static bool node_reach(const SceneView& v, NodeReach& r)
{
    const double R2 = v.band * v.band;
    bool ok = true;
    double near2[3][3];
    for (int8_t& span : r.span) span = -1;
    r.own2 = HUGE_VAL;
    r.safe2 = (1.0 - 1e-6) * (0.25 * v.bucket * v.bucket);
    for (int a = 0; a < 3; ++a) {
        const double delta = 1e-6 * (std::fabs(v.origin[a]) + 4.0 * v.size[a]);
        for (int d = 0; d < 3; ++d) {
            const double near = std::max(0.0, (d - 0.5) * v.h[a] - delta);
            near2[a][d] = near * near;
        }
        r.own2 = std::min(r.own2, near2[a][1]);
        ok = ok && v.band < 2.5 * v.h[a] - delta && delta < 0.1 * v.h[a];
    }
    for (int w = 0; w < kNodeGroups; ++w) {
        r.group2[w] = HUGE_VAL;
        r.valid[w] = 0;
        const int first = node_group_first(w), end = w + 1 < kNodeGroups ? node_group_first(w + 1) : kNodeCells;
        for (int c = first; c < end; ++c) {
            int d[3];
            node_cell(w, c - first, d);
            r.near2[c] = near2[0][std::abs(d[0])] + near2[1][std::abs(d[1])] + near2[2][std::abs(d[2])];
            r.group2[w] = std::min(r.group2[w], r.near2[c]);
            if (r.near2[c] <= R2) {
                r.valid[w] |= 1u << (c - first);
                int8_t& span = r.span[(d[1] + 2) + 5 * (d[2] + 2)];
                span = std::max<int8_t>(span, (int8_t)std::abs(d[0]));
            }
        }
    }
    return ok;
}

// From this many particles on the gather from cells is taken rather than the scatter by particles: where the cells are known, and
// where the particles have to be grouped first.  The gather's searches grow with the surface and wait for one another where few
// tiles hold fluid, the scatter's work is the particles'.  us before the solve of scenes with a collider, scatter / gather, 3 and
// 300 substeps into a dam break: 0.06 M particles (32^3) 161 / 170 and 200 / 278, 0.2 M (48^3) 193 / 202 and 240 / 305, 0.34 M
// (56^3) 221 / 193 and 288 / 307, 0.5 M (64^3) 287 / 257 and 344 / 352, 1 M (80^3) 427 / 345 and 525 / 563.  Surfaces, the
// gather with its grouping: 0.06 M 153 / 198 and 171 / 223, 0.5 M 204 / 210 and 229 / 240, 0.7 M (72^3) 218 / 191 and 246 / 287,
// 1 M (80^3) 256 / 206 and 281 / 362, 1.7 M (96^3) 362 / 248 and 444 / 516, 4 M (128^3) 669 / 399 and 843 / 847.
constexpr uint64_t kGatherKnown = 1ull << 18, kGatherGrouped = 1ull << 20;
bool node_sdf_uses_cells(const SceneView& v)
{
    NodeReach r;
    return v.np >= kGatherGrouped && node_reach(v, r);
}

cudaError_t launch_node_sdf(const SceneView& v, const NodeCells& cells, double* sdf, cudaStream_t st)
{
    const size_t nc = (size_t)v.g.nx * v.g.ny * v.g.nz;
    const double R2 = v.band * v.band;
    NodeReach r;
    if (v.np >= kGatherKnown && cells.start && node_reach(v, r)) {
        const unsigned blocks = 2u * (unsigned)(v.g.tnx * v.g.tny * v.g.tnz);
        if (cells.order) k_sdf_gather<true><<<blocks, kNodeThreads, 0, st>>>(v, cells.start, cells.order, r, R2, sdf);
        else k_sdf_gather<false><<<blocks, kNodeThreads, 0, st>>>(v, cells.start, nullptr, r, R2, sdf);
        count_launch();
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(sdf, 0xff, nc * sizeof(double), st);
    if (e != cudaSuccess) return e;
    if (v.np > 0) {
        k_sdf_scatter<<<(unsigned)((v.np + 255) / 256), 256, 0, st>>>(v, reinterpret_cast<unsigned long long*>(sdf), R2);
        count_launch();
    }
    k_node_values<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(sdf, nc, v.band, v.radius);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_face_fluid_marks(const SceneView& v, const NodeCells& cells, const DiffWork& d, cudaStream_t st)
{
    cudaError_t e = launch_node_sdf(v, cells, d.node, st);
    if (e != cudaSuccess) return e;
    k_face_mark<<<face_grid(v.g.nx, v.g.ny, v.g.nz), dim3(kTileX, kTileY), 0, st>>>(v, d);
    count_launch();
    return cudaGetLastError();
}


}  // namespace fe
