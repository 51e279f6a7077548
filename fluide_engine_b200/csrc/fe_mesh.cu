// fe_mesh.cu -- scene initialisation from triangle meshes: Mesh2SDF, InitializeParticles, VolumeEmitter.
//
// Reference:
//   Mesh2SDF::Build (3d/mesh_2_sdf.cpp:14-82): every node starts at max(h) * (nx + ny + nz); each triangle's index
//     box (vertex coordinates times 1 / h_x on every axis, truncated, widened by one node below and two above,
//     clamped) takes min(distance to the triangle) (Collisions::DistanceToTriangle, 3d/collisions.cpp:21-217);
//     then every node inside the mesh (TriangleMesh::IsInside, 3d/triangle_mesh.cpp:120-163: the sum of
//     atan2(det(A, B, C), k) over triangles, i.e. half the solid angle, is at least 2 pi - 0.001 in magnitude)
//     is negated.
//   PICSimulator::InitializeParticles (pic_simulator.cpp:521-548): every velocity-grid index (i, j, k) whose
//     position (domain origin + h * index) samples the fluid SDF below 0 receives particlesPerBlock particles at
//     position + h * U[0, 1]^3.
//   VolumeEmitter::Emitt (emmiter/volume_emmiter.cpp:58-86), at the start of every substep: every node of the
//     emitter's own SDF grid with sdf <= 0 whose fluid SDF value (same index, the SDF of the previous substep) is
//     >= 0 receives particlesPerBlock particles at position + h * U[0, 1]^3 with the emitter's velocity.
//
// B200 design: the band distances are one CTA per triangle over its index box, min-combined with 64-bit
// atomicMin on the bits of the non-negative distances (the same minimum as the reference's sequential loop).  The
// signs of a closed mesh come from the grid rows: away from the surface its winding sum is 2 pi times an integer that
// changes only where a row crosses a triangle, so one pass over the triangles records the crossings and one over the
// rows adds them up; nodes whose row passes within rounding of an edge, or whose crossing lies within 1e-6 cells of a
// node, sum the winding terms of all triangles, in a pass of their own.  Of an open mesh every node does, one thread per node
// (fe_mesh_to_sdf of 1280 triangles on 96^3 nodes, copies included: 13.2 ms that way, 1.3 ms by rows).  The distance
// arithmetic follows the
// reference's expressions in FP64 with round-to-nearest intrinsics, so distances are bit-identical; the sign test
// sums CUDA's atan2, whose last bits can differ from the host library's, which decides nothing unless a node lies
// within ~1e-12 of the 2 pi - 0.001 threshold (points on the surface sum to pi, points inside to 2 pi).  Seeding
// and emission are count -> scan -> write passes; the random numbers are a counter-based splitmix64 of (seed,
// particle index, axis), deterministic where the reference's std::rand() in a parallel loop is not.
#include <cinttypes>
#include <cstring>

#include "fe_geom.cuh"

namespace fe {
namespace {

// Whether the mesh is closed: every edge, as a pair of vertex positions, is used as often in one direction as in the
// other.  Each use adds a hash of the undirected edge, with its direction as the sign, to two 64-bit sums, which are
// zero for a closed mesh (and for an open one with probability 2^-128).  Then the solid angles of its triangles sum to
// an integer times 4 pi at every point off the surface.  state: the two sums, then non-zero if a coordinate is not
// finite.  mix64 is the output function of the splitmix64 generator (Steele, Lea and Flood 2014).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ unsigned long long hash_point(const double p[3], unsigned long long seed)
{
    unsigned long long h = seed;
#pragma unroll
    for (int a = 0; a < 3; ++a) h = mix64(h ^ (unsigned long long)__double_as_longlong(p[a] + 0.0));  // -0 as 0
    return h;
}
__device__ __forceinline__ int compare_points(const double p[3], const double q[3])
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (p[a] < q[a]) return -1;
        if (p[a] > q[a]) return 1;
    }
    return 0;
}
__device__ __forceinline__ void mesh_edges(const MeshView& m, unsigned long long* state)
{
    unsigned long long s0 = 0, s1 = 0;
    bool bad = false;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < m.nt; t += (uint64_t)gridDim.x * blockDim.x) {
        double p[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k) load_vertex(m, m.T[4 * t + k], p[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int a = 0; a < 3; ++a) bad |= !isfinite(p[k][a]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double* u = p[k];
            const double* v = p[(k + 1) % 3];
            const int c = compare_points(u, v);
            if (c == 0) continue;  // no edge
            const double* lo = c < 0 ? u : v;
            const double* hi = c < 0 ? v : u;
            const unsigned long long h0 = mix64(hash_point(lo, 1) + 3 * hash_point(hi, 2));
            const unsigned long long h1 = mix64(hash_point(lo, 5) ^ (hash_point(hi, 7) << 1 | 1));
            s0 += c < 0 ? h0 : 0ull - h0;
            s1 += c < 0 ? h1 : 0ull - h1;
        }
    }
    if (s0) atomicAdd(state, s0);
    if (s1) atomicAdd(state + 1, s1);
    if (bad) atomicOr(state + 2, 1ull);
}
__device__ __forceinline__ bool mesh_closed(const unsigned long long* state)
{
    return (state[0] | state[1] | state[2]) == 0ull;
}

// One CTA per triangle (grid-stride): the nodes of its index box take the minimum distance; first the sums of the edges.
__global__ void __launch_bounds__(256) k_mesh_band(MeshView m, NodeGrid g, unsigned long long* __restrict__ bits,
                                                   unsigned long long* __restrict__ state)
{
    mesh_edges(m, state);
    const double inv = dd(1.0, g.h[0]);  // the reference scales every axis by 1 / h_x
    for (uint64_t t = blockIdx.x; t < m.nt; t += gridDim.x) {
        double p[3][3];
        load_vertex(m, m.T[4 * t], p[0]);
        load_vertex(m, m.T[4 * t + 1], p[1]);
        load_vertex(m, m.T[4 * t + 2], p[2]);
        int lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double f0 = dm(p[0][d], inv), f1 = dm(p[1][d], inv), f2 = dm(p[2][d], inv);
            lo[d] = min(max((int)fmin(f0, fmin(f1, f2)) - 1, 0), g.n[d] - 1);
            hi[d] = min(max((int)fmax(f0, fmax(f1, f2)) + 2, 0), g.n[d] - 1);
        }
        const int sx = hi[0] - lo[0] + 1, sy = hi[1] - lo[1] + 1, sz = hi[2] - lo[2] + 1;
        const int64_t cells = (int64_t)sx * sy * sz;
        for (int64_t q = threadIdx.x; q < cells; q += blockDim.x) {
            const int i = lo[0] + (int)(q % sx), j = lo[1] + (int)((q / sx) % sy), k = lo[2] + (int)(q / ((int64_t)sx * sy));
            const double pt[3] = {grid_pos(g, 0, i), grid_pos(g, 1, j), grid_pos(g, 2, k)};
            const double d = distance_to_triangle(pt, p[0], p[1], p[2]);
            const unsigned long long b = (unsigned long long)__double_as_longlong(d);
            unsigned long long* cell = bits + idx3(i, j, k, g.n[0], g.n[1]);
            if (b < __ldcg(cell)) atomicMin(cell, b);
        }
    }
}

// Crossings of the grid rows along x with the triangles of a closed mesh, a warp per triangle, a lane per row.  cross[c]:
// .x the change of the winding number (half the winding sum over pi) from node c - 1 to c of the row -- at the first
// node, from far to the left --, bit 0 of .y set where the node is to sum the winding terms itself.  Those nodes are listed: the
// k-th one in the other bits of cross[k].y (on grids that 31 bits can index), state[3] of them.  Going in +x through a
// triangle whose projection on (y, z) is positively oriented leaves the side its normal points away from: -1.
// The projected point is in the triangle when its three edge functions have one sign; `tol` bounds their rounding.
__host__ __device__ __forceinline__ bool mesh_listed(const NodeGrid& g) { return (size_t)g.n[0] * g.n[1] * g.n[2] < (1ull << 31); }
__global__ void __launch_bounds__(256) k_mesh_cross(MeshView m, NodeGrid g, unsigned long long* state, int2* cross)
{
    const bool listed = mesh_listed(g);
    if (!mesh_closed(state)) return;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t t = blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); t < m.nt; t += warps) {
        double A[3], B[3], C[3], lo[3], hi[3], big = 0.0;
        load_vertex(m, m.T[4 * t], A);
        load_vertex(m, m.T[4 * t + 1], B);
        load_vertex(m, m.T[4 * t + 2], C);
        int first[3], last[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fmin(A[a], fmin(B[a], C[a]));
            hi[a] = fmax(A[a], fmax(B[a], C[a]));
            big = fmax(big, fmax(fabs(lo[a]), fabs(hi[a])) + fabs(g.o[a]));
            // nodes at or between the ends, with a margin for the rounding of the positions
            const double f0 = (lo[a] - g.o[a]) / g.h[a], f1 = (hi[a] - g.o[a]) / g.h[a];
            first[a] = (int)fmax(fmin(ceil(f0 - 1e-6), 2e9), -2e9);
            last[a] = (int)fmax(fmin(floor(f1 + 1e-6), 2e9), -2e9);
        }
        const int j0 = max(first[1], 0), j1 = min(last[1], g.n[1] - 1), k0 = max(first[2], 0), k1 = min(last[2], g.n[2] - 1);
        if (j1 < j0 || k1 < k0) continue;
        const double span = (hi[1] - lo[1]) + (hi[2] - lo[2]);
        const double tol = 1e-12 * span * (big + (g.n[1] - 1) * g.h[1] + (g.n[2] - 1) * g.h[2]);
        const int64_t rows = (int64_t)(j1 - j0 + 1) * (k1 - k0 + 1);
        for (int64_t q = lane; q < rows; q += 32) {
            const int j = j0 + (int)(q % (j1 - j0 + 1)), k = k0 + (int)(q / (j1 - j0 + 1));
            const double y = grid_pos(g, 1, j), z = grid_pos(g, 2, k);
            auto edge = [&](const double* u, const double* v) { return (v[1] - u[1]) * (z - u[2]) - (v[2] - u[2]) * (y - u[1]); };
            const double ab = edge(A, B), bc = edge(B, C), ca = edge(C, A);
            const double emin = fmin(ab, fmin(bc, ca)), emax = fmax(ab, fmax(bc, ca));
            if (emin < -tol && emax > tol) continue;  // clearly outside
            const double area = ab + bc + ca;
            int from = 1, to = 0;  // nodes that sum for themselves
            if (emin > tol || emax < -tol) {
                const double f = ((bc * A[0] + ca * B[0] + ab * C[0]) / area - g.o[0]) / g.h[0];
                const double slack = 1e-6 + 4.0 * tol / fabs(area) * (hi[0] - lo[0]) / g.h[0];
                const double r = rint(f);
                if (slack > 0.25) {
                    from = first[0] - 2;
                    to = last[0] + 2;
                } else if (fabs(f - r) <= slack) {
                    from = (int)fmax(fmin(r, 2e9), -2e9);
                    to = from + 1;
                } else {
                    const double at = fmax(ceil(f), 0.0);  // the first node after the crossing
                    if (at <= g.n[0] - 1) atomicAdd(&cross[idx3((int)at, j, k, g.n[0], g.n[1])].x, area < 0.0 ? 1 : -1);
                }
            } else {  // within rounding of an edge
                from = first[0] - 2;
                to = last[0] + 2;
            }
            if (from <= to) {
                from = max(from, 0);
                to = min(max(to, 0), g.n[0] - 1);  // left of the grid: the row's first node
                for (int i = from; i <= to; ++i) {
                    const size_t c = idx3(i, j, k, g.n[0], g.n[1]);
                    if ((atomicOr(&cross[c].y, 1) & 1) || !listed) continue;
                    atomicOr(&cross[atomicAdd(state + 3, 1ull)].y, (int)((unsigned)c << 1));
                }
            }
        }
    }
}

// The side of a point by its winding sum: inside or not, its winding number, and whether that holds beside the point too (it
// does not on the surface).
struct Winding {
    int w;
    bool in, known;
};
__device__ __forceinline__ Winding winding(double sum)
{
    const double pi = 3.14159265358979323846;
    const double turns = sum / (2.0 * pi);
    Winding r;
    r.in = fabs(sum) >= ds(dm(2.0, pi), 0.001);
    r.w = (int)rint(turns);
    r.known = fabs(turns - rint(turns)) < 1e-4;
    return r;
}

// The listed nodes' winding sums: w << 2 | known << 1 | inside in cross[c].x, which holds no crossing that matters there.  2^k
// lanes a node: all 32 for a few nodes, one where the nodes alone fill the device (then a warp's lanes read the same triangle).
// A box of 12,288 triangles with its faces on the nodes of a 96^3 grid: 14.4 ms, 38.7 with every row's nodes summed one after the
// other by the row's warp, 119 with no rows and a thread per node of the grid; with all 2 x 2 x 1024 nodes of a grid on its
// surface 1.3, 308 and 10.7 ms.
constexpr uint64_t kWindingLanes = 148 * 1024;
__global__ void __launch_bounds__(256) k_mesh_own(MeshView m, NodeGrid g, const unsigned long long* __restrict__ state, int2* cross)
{
    if (!mesh_closed(state)) return;
    const uint64_t n = mesh_listed(g) ? state[3] : 0;
    int lanes = 32;
    while (lanes > 1 && n * (uint64_t)lanes > kWindingLanes) lanes >>= 1;
    const int lane = threadIdx.x & 31, sub = lane & (lanes - 1), per = 32 / lanes;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t e0 = (blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * per; e0 < n; e0 += warps * per) {
        const uint64_t e = e0 + lane / lanes;
        const unsigned c = e < n ? (unsigned)cross[e].y >> 1 : 0u;
        double sum = 0.0;
        if (e < n) {
            const unsigned row = c / (unsigned)g.n[0];
            const double pt[3] = {grid_pos(g, 0, (int)(c % (unsigned)g.n[0])), grid_pos(g, 1, (int)(row % (unsigned)g.n[1])),
                                  grid_pos(g, 2, (int)(row / (unsigned)g.n[1]))};
            sum = winding_sum(m, pt, (uint64_t)sub, (uint64_t)lanes);
        }
        for (int o = lanes >> 1; o > 0; o >>= 1) sum = da(sum, __shfl_xor_sync(0xffffffffu, sum, o));
        if (e < n && sub == 0) {
            const Winding r = winding(sum);
            cross[c].x = r.w * 4 + (r.known ? 2 : 0) + (r.in ? 1 : 0);
        }
    }
}

// TriangleMesh::IsInside at every node, then the signed value: -d inside, d outside.  mesh_rows: a closed mesh, a
// warp per row, from the crossings (which share memory with the result: each lane reads its node's before it writes
// it).  A node that sums for itself fixes the winding number for the nodes after it, unless it lies on the surface;
// then the next one sums too, which the row's warp does where k_mesh_own has not.  mesh_signs: an open mesh, a thread per
// node.
__device__ __forceinline__ void mesh_rows(const MeshView& m, const NodeGrid& g, const unsigned long long* bits, double* sdf)
{
    const bool listed = mesh_listed(g);
    const int2* cross = reinterpret_cast<const int2*>(sdf);
    const int lane = threadIdx.x & 31;
    const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5), rows = (size_t)g.n[1] * g.n[2];
    for (size_t row = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
        const int j = (int)(row % g.n[1]), k = (int)(row / g.n[1]);
        int w = 0;
        bool known = true;
        for (int i0 = 0; i0 < g.n[0]; i0 += 32) {
            const int i = i0 + lane, count = min(32, g.n[0] - i0);
            const size_t c = idx3(i, j, k, g.n[0], g.n[1]);
            const int2 x = lane < count ? cross[c] : make_int2(0, 0);
            const unsigned own = __ballot_sync(0xffffffffu, x.y & 1);
            bool inside = false;
            if (known && own == 0u) {
                int s = x.x;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xffffffffu, s, o);
                    if (lane >= o) s += up;
                }
                inside = w + s != 0;
                w += __shfl_sync(0xffffffffu, s, 31);
            } else {
                for (int q = 0; q < count; ++q) {
                    const int step = __shfl_sync(0xffffffffu, x.x, q);
                    bool in;
                    if (listed && ((own >> q) & 1u)) {
                        w = step >> 2;
                        known = step & 2;
                        in = step & 1;
                    } else if (!known || ((own >> q) & 1u)) {
                        const double pt[3] = {grid_pos(g, 0, i0 + q), grid_pos(g, 1, j), grid_pos(g, 2, k)};
                        double sum = winding_sum(m, pt, (uint64_t)lane, 32);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) sum = da(sum, __shfl_xor_sync(0xffffffffu, sum, o));
                        const Winding r = winding(sum);
                        w = r.w;
                        known = r.known;
                        in = r.in;
                    } else {
                        w += step;
                        in = w != 0;
                    }
                    if (lane == q) inside = in;
                }
            }
            if (lane < count) {
                const double d = __longlong_as_double((long long)bits[c]);
                sdf[c] = inside ? dm(d, -1.0) : d;
            }
        }
    }
}

__device__ __forceinline__ void mesh_signs(const MeshView& m, const NodeGrid& g, const unsigned long long* bits, double* sdf)
{
    const double two_pi_tol = ds(dm(2.0, 3.14159265358979323846), 0.001);
    const size_t nc = (size_t)g.n[0] * g.n[1] * g.n[2];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(c % g.n[0]), j = (int)((c / g.n[0]) % g.n[1]), k = (int)(c / ((size_t)g.n[0] * g.n[1]));
        const double pt[3] = {grid_pos(g, 0, i), grid_pos(g, 1, j), grid_pos(g, 2, k)};
        const double d = __longlong_as_double((long long)bits[c]);
        sdf[c] = fabs(winding_sum(m, pt)) >= two_pi_tol ? dm(d, -1.0) : d;
    }
}

// crossed: the crossings are recorded.
__global__ void __launch_bounds__(256) k_mesh_finish(MeshView m, NodeGrid g, const unsigned long long* __restrict__ state, bool crossed,
                                                     const unsigned long long* __restrict__ bits, double* sdf)
{
    if (crossed && mesh_closed(state)) mesh_rows(m, g, bits, sdf);
    else mesh_signs(m, g, bits, sdf);
}

// No distance and no crossing yet, and nothing known of the mesh.
__global__ void k_mesh_start(unsigned long long* __restrict__ bits, double* __restrict__ sdf, size_t n, unsigned long long v,
                             unsigned long long* __restrict__ state)
{
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        bits[c] = v;
        sdf[c] = 0.0;
    }
    if (blockIdx.x == 0 && threadIdx.x < kMeshStateWords) state[threadIdx.x] = 0ull;
}

__device__ __forceinline__ double uniform01(uint64_t seed, uint64_t counter)
{
    uint64_t z = seed + (counter + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// InitializeParticles' cell test: 1 where the velocity-grid position samples the fluid SDF below 0.
__global__ void k_seed_count(const double* __restrict__ fluid_sdf, NodeGrid sdf_grid, NodeGrid vel_grid, uint32_t ppb,
                             uint32_t* __restrict__ count)
{
    const size_t nc = (size_t)vel_grid.n[0] * vel_grid.n[1] * vel_grid.n[2];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(c % vel_grid.n[0]), j = (int)((c / vel_grid.n[0]) % vel_grid.n[1]);
        const int k = (int)(c / ((size_t)vel_grid.n[0] * vel_grid.n[1]));
        const double pos[3] = {grid_pos(vel_grid, 0, i), grid_pos(vel_grid, 1, j), grid_pos(vel_grid, 2, k)};
        count[c] = sample_nodes(fluid_sdf, sdf_grid, pos) < 0.0 ? ppb : 0u;
    }
}

// VolumeEmitter::Emitt's node test: emitter SDF <= 0 and the fluid SDF at the same index >= 0.
__global__ void k_emit_count(const double* __restrict__ emitter_sdf, NodeGrid eg, const double* __restrict__ fluid_sdf,
                             int fnx, int fny, uint32_t ppb, uint32_t* __restrict__ count,
                             const double* __restrict__ collider_sdf)
{
    const size_t nc = (size_t)eg.n[0] * eg.n[1] * eg.n[2];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(c % eg.n[0]), j = (int)((c / eg.n[0]) % eg.n[1]), k = (int)(c / ((size_t)eg.n[0] * eg.n[1]));
        const double fv = fluid_sdf ? fluid_sdf[idx3(i, j, k, fnx, fny)] : 0.0;
        // colliderSdf(i, j, k) > 0: with no collider every node holds 1.7976931348623157e30
        const bool free_node = collider_sdf ? collider_sdf[idx3(i, j, k, fnx, fny)] > 0.0 : true;
        count[c] = (emitter_sdf[c] <= 0.0 && fv >= 0.0 && free_node) ? ppb : 0u;
    }
}

// Writes the particles of every counted node: node position + h * U[0,1]^3 (FP32), the given velocity, C = 0.
__global__ void k_spawn(NodeGrid g, const uint32_t* __restrict__ count, const uint32_t* __restrict__ offset,
                        uint64_t seed, SceneView v, uint64_t base, float vx, float vy, float vz)
{
    const size_t nc = (size_t)g.n[0] * g.n[1] * g.n[2];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const uint32_t cnt = count[c];
        if (!cnt) continue;
        const int i = (int)(c % g.n[0]), j = (int)((c / g.n[0]) % g.n[1]), k = (int)(c / ((size_t)g.n[0] * g.n[1]));
        const double pos[3] = {grid_pos(g, 0, i), grid_pos(g, 1, j), grid_pos(g, 2, k)};
        for (uint32_t q = 0; q < cnt; ++q) {
            const uint64_t p = base + offset[c] + q;
            const uint64_t id = (uint64_t)offset[c] + q;
            const double x = da(dm(g.h[0], uniform01(seed, 3 * id)), pos[0]);
            const double y = da(dm(g.h[1], uniform01(seed, 3 * id + 1)), pos[1]);
            const double z = da(dm(g.h[2], uniform01(seed, 3 * id + 2)), pos[2]);
            v.px[p] = (float)x; v.py[p] = (float)y; v.pz[p] = (float)z;
            v.vx[p] = vx; v.vy[p] = vy; v.vz[p] = vz;
            v.pid[p] = (uint32_t)p;
            if (v.c[0])
#pragma unroll
                for (int a = 0; a < 9; ++a) v.c[a][p] = 0.f;
        }
    }
}

// VolumeField::Initialize (forces/volume_field.cpp:72-89): at every node of the field's grid, the closest point on
// the first nearest triangle (Collisions::ClosestTriangleIdx, 3d/collisions.cpp:249-265: strict < from
// 1.7976931348623157e30) minus the node position, 3 doubles per node.  One thread per node over all triangles.
__global__ void __launch_bounds__(256) k_volume_vectors(MeshView m, NodeGrid g, double* __restrict__ out)
{
    const size_t nc = (size_t)g.n[0] * g.n[1] * g.n[2];
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < nc; c += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(c % g.n[0]), j = (int)((c / g.n[0]) % g.n[1]), k = (int)(c / ((size_t)g.n[0] * g.n[1]));
        const double gp[3] = {grid_pos(g, 0, i), grid_pos(g, 1, j), grid_pos(g, 2, k)};
        double best = 1.7976931348623157e30;
        uint64_t idx = 0;
        double A[3], B[3], C[3];
        for (uint64_t t = 0; t < m.nt; ++t) {
            load_vertex(m, __ldg(m.T + 4 * t), A);
            load_vertex(m, __ldg(m.T + 4 * t + 1), B);
            load_vertex(m, __ldg(m.T + 4 * t + 2), C);
            const double d = distance_to_triangle(gp, A, B, C);
            if (d < best) {
                best = d;
                idx = t;
            }
        }
        double cp[3] = {0.0, 0.0, 0.0};
        if (m.nt) {
            load_vertex(m, m.T[4 * idx], A);
            load_vertex(m, m.T[4 * idx + 1], B);
            load_vertex(m, m.T[4 * idx + 2], C);
            closest_on_triangle(gp, A, B, C, cp);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) out[3 * c + a] = ds(cp[a], gp[a]);
    }
}

NodeGrid node_grid(const int n[3], const double o[3], const double h[3])
{
    NodeGrid g;
    for (int a = 0; a < 3; ++a) { g.n[a] = n[a]; g.o[a] = o[a]; g.h[a] = h[a]; }
    return g;
}

}  // namespace

cudaError_t launch_mesh_to_sdf(const double* V, uint64_t nv, const int64_t* T, uint64_t nt, const int n[3],
                               const double o[3], const double h[3], unsigned long long* scratch, double* sdf,
                               unsigned long long* state, cudaStream_t st)
{
    const NodeGrid g = node_grid(n, o, h);
    const size_t nc = (size_t)n[0] * n[1] * n[2];
    const double hmax = (h[0] >= h[1] && h[0] >= h[2]) ? h[0] : ((h[1] >= h[0] && h[1] >= h[2]) ? h[1] : h[2]);
    const double fill = hmax * (double)((size_t)n[0] + (size_t)n[1] + (size_t)n[2]);
    unsigned long long fill_bits;
    std::memcpy(&fill_bits, &fill, sizeof(fill_bits));
    MeshView m{V, T, nv, nv ? nt : 0};  // no vertices: no distances and no triangle to wind around (the fill stays positive)
    k_mesh_start<<<(unsigned)std::min<size_t>((nc + 255) / 256, 148 * 32), 256, 0, st>>>(scratch, sdf, nc, fill_bits, state);
    count_launch();
    if (m.nt > 0) {
        k_mesh_band<<<(unsigned)std::min<uint64_t>(nt, 148 * 64), 256, 0, st>>>(m, g, scratch, state);
        count_launch();
    }
    // a node's winding terms take 0.6 us a triangle, and all nodes' 1 us for some 10^5: sums that are through sooner than the two
    // passes that save them (some 28 us) are taken directly (a call, with / without the passes: 20 triangles on 32^3 nodes 275 /
    // 259 us, 80 on 16^3 209 / 255, 320 on 16^3 230 / 455)
    const bool crossed = m.nt >= 48 || (double)m.nt * (double)nc >= 3.0 * (1 << 20);
    if (crossed) {
        k_mesh_cross<<<(unsigned)std::min<uint64_t>((nt + 7) / 8, 148 * 8), 256, 0, st>>>(m, g, state, reinterpret_cast<int2*>(sdf));
        k_mesh_own<<<148 * 8, 256, 0, st>>>(m, g, state, reinterpret_cast<int2*>(sdf));
        count_launch(2);
    }
    const size_t blocks = std::max((nc + 255) / 256, ((size_t)n[1] * n[2] + 7) / 8);
    k_mesh_finish<<<(unsigned)std::min<size_t>(blocks, 148 * 32), 256, 0, st>>>(m, g, state, crossed, scratch, sdf);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_volume_vectors(const double* V, uint64_t nv, const int64_t* T, uint64_t nt, const int n[3],
                                  const double o[3], const double h[3], double* out, cudaStream_t st)
{
    MeshView m;
    m.V = V;
    m.T = T;
    m.nv = nv;
    m.nt = nv ? nt : 0;
    const NodeGrid g = node_grid(n, o, h);
    const size_t nc = (size_t)n[0] * n[1] * n[2];
    k_volume_vectors<<<(unsigned)std::min<size_t>((nc + 255) / 256, 148 * 32), 256, 0, st>>>(m, g, out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_seed_count(const double* fluid_sdf, const int n[3], const double sdf_o[3], const double h[3],
                              const double vel_o[3], uint32_t ppb, uint32_t* count, cudaStream_t st)
{
    const NodeGrid sg = node_grid(n, sdf_o, h), vg = node_grid(n, vel_o, h);
    const size_t nc = (size_t)n[0] * n[1] * n[2];
    k_seed_count<<<(unsigned)std::min<size_t>((nc + 255) / 256, 148 * 32), 256, 0, st>>>(fluid_sdf, sg, vg, ppb, count);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_emit_count(const double* emitter_sdf, const int en[3], const double* fluid_sdf, int fnx, int fny,
                              uint32_t ppb, uint32_t* count, cudaStream_t st, const double* collider_sdf)
{
    const double z[3] = {0, 0, 0};
    const NodeGrid eg = node_grid(en, z, z);
    const size_t nc = (size_t)en[0] * en[1] * en[2];
    k_emit_count<<<(unsigned)std::min<size_t>((nc + 255) / 256, 148 * 32), 256, 0, st>>>(emitter_sdf, eg, fluid_sdf, fnx,
                                                                                        fny, ppb, count, collider_sdf);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_spawn(const int n[3], const double o[3], const double h[3], const uint32_t* count,
                         const uint32_t* offset, uint64_t seed, const SceneView& v, uint64_t base, const float vel[3],
                         cudaStream_t st)
{
    const NodeGrid g = node_grid(n, o, h);
    const size_t nc = (size_t)n[0] * n[1] * n[2];
    k_spawn<<<(unsigned)std::min<size_t>((nc + 255) / 256, 148 * 32), 256, 0, st>>>(g, count, offset, seed, v, base, vel[0],
                                                                                   vel[1], vel[2]);
    count_launch();
    return cudaGetLastError();
}

}  // namespace fe
